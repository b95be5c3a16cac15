// Device assembly of the coupled Navier-Stokes system; see ns.cuh. Built with -fmad=false.
#include "ns.cuh"

namespace vfv {

namespace {

__device__ __forceinline__ double pow5(double x) {
    const double x2 = x * x;
    return x2 * x2 * x;
}

// skew-corrected arithmetic-mean face density (opscl_dom_div.rs:104-106, flow_helper.rs:51)
__device__ __forceinline__ double face_den(const NsDev& D, int64_t v, int32_t i) {
    const int64_t N = D.n, E = D.n_dir;
    const int32_t nb = D.ni[i];
    const double sx = D.skew[i], sy = D.skew[E + i], sz = D.skew[2 * E + i];
    return 0.5 * (D.den[v] + D.den[nb]) +
           0.5 * (sx * (D.gden[v] + D.gden[nb]) + sy * (D.gden[N + v] + D.gden[N + nb]) + sz * (D.gden[2 * N + v] + D.gden[2 * N + nb]));
}

// harmonic-mean, skew-corrected, guarded face viscosity (opvec_dom_diff.rs:76-79)
__device__ __forceinline__ double face_visc(const NsDev& D, int64_t v, int32_t i) {
    const int64_t N = D.n, E = D.n_dir;
    const int32_t nb = D.ni[i];
    const double mv = D.visc[v], mn = D.visc[nb];
    const double sx = D.skew[i], sy = D.skew[E + i], sz = D.skew[2 * E + i];
    const double vm = (mv + mn != 0.0) ? 2.0 * mv * mn / (mv + mn) : 0.0;
    const double vf = vm + 0.5 * (sx * (D.gvisc[v] + D.gvisc[nb]) + sy * (D.gvisc[N + v] + D.gvisc[N + nb]) +
                                  sz * (D.gvisc[2 * N + v] + D.gvisc[2 * N + nb]));
    return vf > 0.0 ? vf : vm;
}

// body force at the control-volume centroid (opvec_dom_src.rs:57-64)
__device__ __forceinline__ void force_centroid(const NsDev& D, int64_t v, double f[3]) {
    const int64_t N = D.n;
    const double cx = D.cskew[v], cy = D.cskew[N + v], cz = D.cskew[2 * N + v];
#pragma unroll
    for (int q = 0; q < 3; ++q)
        f[q] = D.fce[q * N + v] + D.gfce[(3 * q) * N + v] * cx + D.gfce[(3 * q + 1) * N + v] * cy + D.gfce[(3 * q + 2) * N + v] * cz;
}

// The per-vertex kernels give a vertex kRowG lanes (its ~15 faces two per lane): a warp then reads the
// faces' arrays in runs instead of one address per vertex, and twice the loads are in flight. Sums
// over faces are a lane's faces in order, then a butterfly. At 110,592 vertices, one thread per vertex
// and now: k_ns_rc 159 -> 54 us, k_ns_flux 292 -> 78, k_ns_rhs 248 -> 109, k_ns_mom 182 -> 61 (cold).
constexpr int kRowG = 8;

__device__ __forceinline__ double lanes_sum(double x, unsigned mask, int g) {
    for (int o = g / 2; o > 0; o >>= 1) x += __shfl_xor_sync(mask, x, o, g);
    return x;
}
__device__ __forceinline__ unsigned lanes_mask(int g) {
    return (g == 32 ? 0xffffffffu : (1u << g) - 1u) << ((threadIdx.x & 31) & ~(g - 1));
}

// Rhie-Chow coefficient V / a_P with a_P = sum_f D_f A(|Pe_f|) + max(F_f, 0), F_f the central
// mass flux (flow_helper::update_flow, flow_helper.rs:19-66)
__global__ void __launch_bounds__(256) k_ns_rc(NsDev D) {
    const int lane = threadIdx.x & (kRowG - 1);
    const int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kRowG;
    if (v >= D.n) return;
    const int64_t N = D.n, E = D.n_dir;
    const double* u = D.x;
    double cp = 0.0;
    for (int32_t i = D.np[v] + lane; i < D.np[v + 1]; i += kRowG) {
        const int32_t nb = D.ni[i];
        const double face = D.area[i], dist = D.dist[i];
        const double nx = D.norm[i], ny = D.norm[E + i], nz = D.norm[2 * E + i];
        const double den_f = face_den(D, v, i);
        const double cond = face_visc(D, v, i) * face / dist;
        const double fl = den_f * 0.5 * ((u[v] + u[nb]) * nx + (u[N + v] + u[N + nb]) * ny + (u[2 * N + v] + u[2 * N + nb]) * nz) * face;
        const double pe = cond != 0.0 ? fl / cond : 0.0;
        const double a = fmax(1.0 - 0.1 * fabs(pe), 0.0);
        cp += cond * pow5(a) + fmax(fl, 0.0);
    }
    cp = lanes_sum(cp, lanes_mask(kRowG), kRowG);
    if (lane == 0) D.rc[v] = cp > 0.0 ? D.cvol[v] / cp : 0.0;
}

// d (grad p - fce) per vertex with grad p = sum_m c_m p_m / V (flow_helper.rs:86-113); 16 lanes for
// the ~65 coefficients of a vertex
constexpr int kGradG = 16;
__global__ void __launch_bounds__(256) k_ns_mom(NsDev D) {
    const int lane = threadIdx.x & (kGradG - 1);
    const int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kGradG;
    if (v >= D.n) return;
    const int64_t N = D.n, G = D.n_gc;
    const double* p = D.x + 3 * N;
    const double vol = D.cvol[v];
    double px = 0.0, py = 0.0, pz = 0.0;
    for (int32_t k = D.gcp[v] + lane; k < D.gcp[v + 1]; k += kGradG) {
        const double pm = p[D.gcv[k]];
        px += D.gcc[k] * pm;
        py += D.gcc[G + k] * pm;
        pz += D.gcc[2 * G + k] * pm;
    }
    const unsigned mask = lanes_mask(kGradG);
    px = lanes_sum(px, mask, kGradG) / vol;
    py = lanes_sum(py, mask, kGradG) / vol;
    pz = lanes_sum(pz, mask, kGradG) / vol;
    if (lane != 0) return;
    double f[3];
    force_centroid(D, v, f);
    const double r = D.rc[v];
    D.mom[v] = r * (px - f[0]);
    D.mom[N + v] = r * (py - f[1]);
    D.mom[2 * N + v] = r * (pz - f[2]);
}

// face mass flux with the Rhie-Chow correction (flow_helper.rs:116-173)
__global__ void __launch_bounds__(256) k_ns_flux(NsDev D) {
    const int lane = threadIdx.x & (kRowG - 1);
    const int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kRowG;
    if (v >= D.n) return;
    const int64_t N = D.n, E = D.n_dir;
    const double* u = D.x;
    const double* p = D.x + 3 * N;
    for (int32_t i = D.np[v] + lane; i < D.np[v + 1]; i += kRowG) {
        const int32_t nb = D.ni[i];
        const double face = D.area[i], dist = D.dist[i];
        const double nx = D.norm[i], ny = D.norm[E + i], nz = D.norm[2 * E + i];
        const double sx = D.skew[i], sy = D.skew[E + i], sz = D.skew[2 * E + i];
        const double den_f = face_den(D, v, i);
        double uf[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double* g = D.gvel + 3 * q * N;
            uf[q] = 0.5 * (u[q * N + v] + u[q * N + nb]) + 0.5 * (sx * (g[v] + g[nb]) + sy * (g[N + v] + g[N + nb]) + sz * (g[2 * N + v] + g[2 * N + nb]));
        }
        const double fce_e = 0.5 * (nx * (D.fce[v] + D.fce[nb]) + ny * (D.fce[N + v] + D.fce[N + nb]) + nz * (D.fce[2 * N + v] + D.fce[2 * N + nb]));
        const double mom_e = 0.5 * (nx * (D.mom[v] + D.mom[nb]) + ny * (D.mom[N + v] + D.mom[N + nb]) + nz * (D.mom[2 * N + v] + D.mom[2 * N + nb]));
        const double vel_rc = -0.5 * (D.rc[v] + D.rc[nb]) * ((p[nb] - p[v]) / dist - fce_e) + mom_e;
        D.flux[i] = den_f * (uf[0] * nx + uf[1] * ny + uf[2] * nz + vel_rc) * face;
    }
}

// sum of the gradient weights of every vertex: what a face's gradient of v takes from v itself
__global__ void __launch_bounds__(256) k_ns_gsum(NsDev D, double* __restrict__ gsum) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= D.n) return;
    double s[3] = {0.0, 0.0, 0.0};
    for (int32_t k = D.np[v]; k < D.np[v + 1]; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a) s[a] += D.gw[a * D.n_dir + k];
#pragma unroll
    for (int a = 0; a < 3; ++a) gsum[a * D.n + v] = s[a];
}

// Momentum rows: points hold advection (opvec_dom_adv.rs:64-113) plus diffusion
// (opvec_dom_diff.rs:55-91) per neighbour, their diagonal, and the pressure gradient
// (opvec_dom_grad.rs:53-67); nodes the Dirichlet diagonal (opvec_bnd_dir.rs:56-80). The three
// velocity rows of a vertex share all but the pressure part. A group of 16 lanes per vertex, so that
// the entries are written in runs: 176 us cold at 110,592 vertices (892 us with a thread per vertex
// writing triplets).
constexpr int kMomG = 16;
__global__ void __launch_bounds__(256) k_ns_mom_rows(NsDev D) {
    const int lane = threadIdx.x & (kMomG - 1);
    const int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kMomG;
    if (v >= D.n) return;
    const int64_t N = D.n, G = D.n_gc;
    const unsigned mask = lanes_mask(kMomG);
    double* row[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) row[q] = D.val + D.rp[q * N + v];
    if (v >= D.n_pts) {
#pragma unroll
        for (int q = 0; q < 3; ++q)
            if (lane == q) row[q][0] = 1.0;
        return;
    }
    const int32_t b = D.np[v], e = D.np[v + 1], dl = D.dloc[v];
    double adv = 0.0, dif = 0.0;  // the diagonal's advection and diffusion parts
    for (int32_t i = b + lane; i < e; i += kMomG) {
        const double cond = face_visc(D, v, i) * D.area[i] / D.dist[i];
        const double fl = D.flux[i];
        const double pe = cond != 0.0 ? fl / cond : 0.0;
        const double coeff = cond * (pow5(fmax(1.0 - 0.1 * fabs(pe), 0.0)) - 1.0) + fmax(-fl, 0.0);
        const int32_t k = i - b;
        const int32_t slot = k + (k >= dl ? 1 : 0);
        const double a = coeff + cond;
#pragma unroll
        for (int q = 0; q < 3; ++q) row[q][slot] = a;
        adv += -coeff;
        dif += -cond;
    }
    adv = lanes_sum(adv, mask, kMomG) + lanes_sum(dif, mask, kMomG);
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) row[q][dl] = adv;
    }
    const int32_t gb = D.gcp[v], gn = D.gcp[v + 1] - gb, o = e - b + 1;
    for (int32_t k = lane; k < gn; k += kMomG) {
#pragma unroll
        for (int q = 0; q < 3; ++q) row[q][o + k] = -D.gcc[q * G + gb + k];
    }
}

// Pressure rows, one warp per vertex: divergence (opscl_dom_div.rs:84-148, and for nodes the
// boundary sub-faces of opscl_bnd_div.rs:163-181) and the pressure stabiliser
// (opscl_dom_pstab.rs:86-146), summed into the row in shared memory and written once.
// With c_i = 0.5 rho_f A and s_i the skew vector of face i, the divergence triplets of component c are
//   -c_i n_c at v and at n_i,  -c_i n_c (w_k . s_i) at every neighbour k of v and of n_i, and
//   the opposite of their sum at v and at n_i.
// The part over v's own neighbours is w_k . M_c with M_c = sum_i c_i n_c s_i, the sums over k are
// gsum . s_i, and the same holds for the stabiliser's grad_coeff(v) part, so only the second ring is
// visited per face: ~230 + ~1000 places per row instead of ~5,000 triplets.
// Faces are taken one after the other and the places of one face differ, so no two lanes meet.
// A row longer than the shared buffer is summed in place in global memory (STAGED: there is none).
// 110,592 vertices on one B200: 0.99 ms cold, against 1.94 ms to write the triplets and 4.25 ms to sum
// them per slot (630 M triplets through HBM twice). It is bound by the latency of L2 (one to two
// instructions per scheduler every three cycles at 24 warps per SM): loading a face ahead took it from
// 1.47 ms, 80 registers (6 blocks; 164 to 208 bytes spilled) against 96 (5) and 128 (4) 1.70, 1.75 and 1.87 ms per
// assembly.
constexpr int kPWarps = 4;
constexpr int kPFaces = 32;  // faces staged at a time
constexpr int kPU = 3;       // grad_coeff entries of a neighbour per lane in flight
constexpr int kPCap = 1152;  // doubles of a row kept in shared memory (48 KB a block with the staged faces)
struct PFace {  // one face: -c_i n, s, -c_n n (stabiliser), the neighbour's lists
    double cn[3], s[3], pn[3];
    int32_t nb0, ndeg, gc0, ngc;
};

// Face i of v for the second part of its p row; returns the face density.
__device__ __forceinline__ double p_face(const NsDev& D, int64_t v, int32_t i, PFace& f) {
    const int64_t E = D.n_dir;
    const int32_t nb = D.ni[i];
    const double face = D.area[i];
    const double den_f = face_den(D, v, i);
    const double coeff = 0.5 * den_f * face;
    const double cn = den_f * 0.5 * D.rc[nb] / D.cvol[nb] * face;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double nn = D.norm[c * E + i];
        f.cn[c] = -coeff * nn;
        f.s[c] = D.skew[c * E + i];
        f.pn[c] = -cn * nn;
    }
    f.nb0 = D.np[nb];
    f.ndeg = D.np[nb + 1] - f.nb0;
    f.gc0 = D.gcp[nb];
    f.ngc = D.gcp[nb + 1] - f.gc0;
    return den_f;
}

template <typename TM, bool STAGED>
__global__ void __launch_bounds__(32 * kPWarps, 6) k_ns_p_rows(NsDev D, int cap) {
    extern __shared__ double s_rows[];
    __shared__ PFace s_face[kPWarps][kPFaces];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t v = (int64_t)blockIdx.x * kPWarps + w;
    if (v >= D.n) return;
    const int64_t N = D.n, E = D.n_dir, B = D.n_bsub, G = D.n_gc;
    const int32_t rb = D.rp[3 * N + v], len = D.rp[3 * N + v + 1] - rb;
    if (v == D.pref_vid) {
        if (lane == 0) D.val[rb] = 1.0;
        return;
    }
    const bool staged = STAGED || len <= cap;
    double* acc = STAGED ? s_rows + w * cap : staged ? s_rows + w * cap : D.val + rb;
    const int32_t L = D.qlen[v];
    double* racc = acc + 3 * L;
    for (int t = lane; t < len; t += 32) acc[t] = 0.0;
    const int32_t b = D.np[v], e = D.np[v + 1];
    PFace* fc = s_face[w];
    __syncwarp(full);
    {
        // v's own part, and the faces' coefficients (staged for the second part when one chunk holds them)
        const TM* __restrict__ qring = (const TM*)D.qring;
        const TM* __restrict__ rring = (const TM*)D.rring;
        const TM* __restrict__ rgc = (const TM*)D.rgc;
        double M[9], m1[3], nv[3], dp = 0.0;  // M[3 c + a] = sum_i -c_i n_c s_a, sum_i -c_i n_c, sum_i c_v n, sum of c_p / d
#pragma unroll
        for (int a = 0; a < 9; ++a) M[a] = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) m1[a] = nv[a] = 0.0;
        const double rc_v = D.rc[v], vol_v = D.cvol[v];
        for (int32_t i = b + lane; i < e; i += 32) {
            PFace f;
            const double den_f = p_face(D, v, i, f);
            const int32_t nb = D.ni[i];
            const double face = D.area[i], rc_n = D.rc[nb];
            const double cv = den_f * 0.5 * rc_v / vol_v * face;
            const double cp = den_f * 0.5 * (rc_v + rc_n) * face / D.dist[i];
            const double gs = D.gsum[nb] * f.s[0] + D.gsum[N + nb] * f.s[1] + D.gsum[2 * N + nb] * f.s[2];
            const int32_t pq = qring[i];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                m1[c] += f.cn[c];
                nv[c] += cv * D.norm[c * E + i];
#pragma unroll
                for (int a = 0; a < 3; ++a) M[3 * c + a] += f.cn[c] * f.s[a];
                acc[c * L + pq] += f.cn[c] - f.cn[c] * gs;  // n_i: the mean, and minus the sum over its neighbours
            }
            racc[rring[i]] += cp;
            dp += cp;
            if (e - b <= kPFaces) fc[lane] = f;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int a = 0; a < 9; ++a) M[a] += __shfl_xor_sync(full, M[a], o);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                m1[a] += __shfl_xor_sync(full, m1[a], o);
                nv[a] += __shfl_xor_sync(full, nv[a], o);
            }
            dp += __shfl_xor_sync(full, dp, o);
        }
        __syncwarp(full);
        for (int32_t k = b + lane; k < e; k += 32) {  // divergence: v's own neighbours
            const double g0 = D.gw[k], g1 = D.gw[E + k], g2 = D.gw[2 * E + k];
            double* o = acc + qring[k];
#pragma unroll
            for (int c = 0; c < 3; ++c) o[c * L] += M[3 * c] * g0 + M[3 * c + 1] * g1 + M[3 * c + 2] * g2;
        }
        const int32_t gv0 = D.gcp[v], gv1 = D.gcp[v + 1];
        if (e > b)
            for (int32_t k = gv0 + lane; k < gv1; k += 32)  // stabiliser: grad_coeff of v
                racc[rgc[k]] += -(D.gcc[k] * nv[0] + D.gcc[G + k] * nv[1] + D.gcc[2 * G + k] * nv[2]);
        __syncwarp(full);
        if (lane < 3) {  // v itself
            const double g0 = D.gsum[v], g1 = D.gsum[N + v], g2 = D.gsum[2 * N + v];
            double t = 0.0;
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (lane == c) t = m1[c] - (M[3 * c] * g0 + M[3 * c + 1] * g1 + M[3 * c + 2] * g2);
            acc[lane * L + D.qself[v]] += t;
        }
        if (lane == 3 && e > b) racc[D.rself[v]] -= dp;
        __syncwarp(full);
    }
    if (v >= D.n_pts) {
        if (lane < 3) {  // boundary sub-faces, lane c its component
            const TM* __restrict__ qsub = (const TM*)D.qsub;
            double* o = acc + lane * L;
            for (int32_t s = D.bp[v]; s < D.bp[v + 1]; ++s) {
                const double an = D.barea[s] * D.bnorm[lane * B + s];
                o[D.qself[v]] -= D.bw[s] * D.den[v] * an;
                o[qsub[s]] -= D.bw[B + s] * D.den[D.bj[s]] * an;
                o[qsub[B + s]] -= D.bw[2 * B + s] * D.den[D.bk[s]] * an;
            }
        }
        __syncwarp(full);
    }
    const TM* __restrict__ qnb = (const TM*)D.qnb + D.qoff[v];
    const TM* __restrict__ rnb = (const TM*)D.rnb + D.roff[v];
    for (int32_t c0 = b; c0 < e; c0 += kPFaces) {
        if (e - b > kPFaces) {
            __syncwarp(full);
            PFace f;
            if (c0 + lane < e) {
                p_face(D, v, c0 + lane, f);
                fc[lane] = f;
            }
            __syncwarp(full);
        }
        const int cnt = min(kPFaces, (int)(e - c0));
        // divergence: the neighbours of n_i, half a warp per face; the two faces' sums follow one
        // another. Here and below the next faces' weights are loaded before this one's are added: with
        // ~20 warps on an SM the kernel waits for L2 otherwise.
        const int h = lane >> 4, l = lane & 15;
        {
            struct Frag {
                int32_t at, mine, most;
                double g0, g1, g2;
            };
            const TM* __restrict__ pl = qnb;
            auto load = [&](int t, Frag& r) {
                const int32_t nd0 = t < cnt ? fc[t].ndeg : 0, nd1 = t + 1 < cnt ? fc[t + 1].ndeg : 0;
                r.mine = h ? nd1 : nd0;
                r.most = max(nd0, nd1);
                r.at = 0;
                r.g0 = r.g1 = r.g2 = 0.0;
                if (l < r.mine) {
                    const double* __restrict__ gw = D.gw + fc[t + h].nb0 + l;
                    r.at = pl[(h ? nd0 : 0) + l];
                    r.g0 = __ldg(gw);
                    r.g1 = __ldg(gw + E);
                    r.g2 = __ldg(gw + 2 * E);
                }
                pl += nd0 + nd1;
            };
            auto add = [&](const PFace& f, bool has, int32_t at, double g0, double g1, double g2) {
                const double ws = g0 * f.s[0] + g1 * f.s[1] + g2 * f.s[2];
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    if (h == hh && has) {
                        double* o = acc + at;
#pragma unroll
                        for (int c = 0; c < 3; ++c) o[c * L] += f.cn[c] * ws;
                    }
                    __syncwarp(full);
                }
            };
            Frag cur, nxt;
            load(0, cur);
            for (int t = 0; t < cnt; t += 2) {
                const TM* __restrict__ here = qnb;
                qnb = pl;
                load(t + 2, nxt);
                const PFace& f = fc[t + h < cnt ? t + h : t];
                add(f, l < cur.mine, cur.at, cur.g0, cur.g1, cur.g2);
                for (int k = l + 16; k - l < cur.most; k += 16) {  // vertices with more than 16 neighbours
                    const bool has = k < cur.mine;
                    const double* __restrict__ gw = D.gw + f.nb0 + k;
                    add(f, has, has ? (int32_t)here[(h ? fc[t].ndeg : 0) + k] : 0, has ? __ldg(gw) : 0.0, has ? __ldg(gw + E) : 0.0,
                        has ? __ldg(gw + 2 * E) : 0.0);
                }
                cur = nxt;
            }
            qnb = pl;
        }
        // stabiliser: grad_coeff of n_i, kPU of a lane's coefficients at a time
        {
            struct Frag {
                int32_t at[kPU];
                double g0[kPU], g1[kPU], g2[kPU];
            };
            auto load = [&](const TM* __restrict__ pl, int t, int k0, Frag& r) {
                const int32_t ngc = t < cnt ? fc[t].ngc : 0;
                const double* __restrict__ gc = D.gcc + (t < cnt ? fc[t].gc0 : 0);
#pragma unroll
                for (int u = 0; u < kPU; ++u) {
                    const int k = k0 + lane + 32 * u;
                    r.at[u] = -1;
                    if (k < ngc) {
                        r.at[u] = pl[k];
                        r.g0[u] = __ldg(gc + k);
                        r.g1[u] = __ldg(gc + G + k);
                        r.g2[u] = __ldg(gc + 2 * G + k);
                    }
                }
            };
            auto add = [&](const PFace& f, const Frag& r) {
#pragma unroll
                for (int u = 0; u < kPU; ++u)
                    if (r.at[u] >= 0) racc[r.at[u]] += r.g0[u] * f.pn[0] + r.g1[u] * f.pn[1] + r.g2[u] * f.pn[2];
            };
            Frag cur, nxt;
            load(rnb, 0, 0, cur);
            for (int t = 0; t < cnt; ++t) {
                const PFace& f = fc[t];
                const TM* __restrict__ here = rnb;
                rnb += f.ngc;
                load(rnb, t + 1, 0, nxt);
                add(f, cur);
                for (int k0 = 32 * kPU; k0 < f.ngc; k0 += 32 * kPU) {
                    load(here, t, k0, cur);
                    add(f, cur);
                }
                __syncwarp(full);
                cur = nxt;
            }
        }
    }
    if (staged)
        for (int t = lane; t < len; t += 32) D.val[rb + t] = acc[t];
}

// Right-hand side, kRowG lanes per vertex, each row in the reference's operator order:
// momentum rows of points: transpose term (opvec_dom_dtrn.rs:57-110), dilatational term
// (opvec_dom_ddil.rs:57-109), body force (opvec_dom_src.rs:52-69); momentum rows of nodes the
// boundary velocity; pressure rows the stabiliser's body-force part; the reference row p = pref.
__global__ void __launch_bounds__(256) k_ns_rhs(NsDev D) {
    const int lane = threadIdx.x & (kRowG - 1);
    const int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kRowG;
    if (v >= D.n) return;
    const unsigned mask = lanes_mask(kRowG);
    const int64_t N = D.n, E = D.n_dir;
    const int32_t b = D.np[v], e = D.np[v + 1];
    const bool point = v < D.n_pts;
    double s1[3] = {0.0, 0.0, 0.0}, s2[3] = {0.0, 0.0, 0.0}, bp = 0.0;
    double gv[9], fv[3];
#pragma unroll
    for (int q = 0; q < 9; ++q) gv[q] = point ? D.gvel[q * N + v] : 0.0;
    force_centroid(D, v, fv);
    const double div_v = gv[0] + gv[4] + gv[8];
    const double rc_v = D.rc[v];
    for (int32_t i = b + lane; i < e; i += kRowG) {
        const int32_t nb = D.ni[i];
        const double face = D.area[i];
        const double nx = D.norm[i], ny = D.norm[E + i], nz = D.norm[2 * E + i];
        if (point) {
            const double vf = face_visc(D, v, i);
            double gn[9], gf[9];
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                gn[q] = D.gvel[q * N + nb];
                gf[q] = 0.5 * (gv[q] + gn[q]);
            }
            s1[0] += vf * (gf[0] * nx + gf[3] * ny + gf[6] * nz) * face;
            s1[1] += vf * (gf[1] * nx + gf[4] * ny + gf[7] * nz) * face;
            s1[2] += vf * (gf[2] * nx + gf[5] * ny + gf[8] * nz) * face;
            const double div_n = gn[0] + gn[4] + gn[8];
            const double c = (-2.0 / 3.0) * vf * (0.5 * (div_v + div_n)) * face;
            s2[0] += c * nx;
            s2[1] += c * ny;
            s2[2] += c * nz;
        }
        double fn[3];
        force_centroid(D, nb, fn);
        const double rc_n = D.rc[nb];
        const double den_f = face_den(D, v, i);
        double frc[3];
#pragma unroll
        for (int q = 0; q < 3; ++q)
            frc[q] = 0.5 * (rc_v + rc_n) * 0.5 * (D.fce[q * N + v] + D.fce[q * N + nb]) - 0.5 * (rc_v * fv[q] + rc_n * fn[q]);
        bp += den_f * (frc[0] * nx + frc[1] * ny + frc[2] * nz) * face;
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        s1[q] = lanes_sum(s1[q], mask, kRowG);
        s2[q] = lanes_sum(s2[q], mask, kRowG);
    }
    bp = lanes_sum(bp, mask, kRowG);
    if (lane != 0) return;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        if (point) {
            double bq = 0.0;
            bq += -s1[q];
            bq += -s2[q];
            bq += -fv[q] * D.cvol[v];
            D.b[q * N + v] = bq;
        } else {
            D.b[q * N + v] = 0.0 + D.bc_vel[q * N + v];
        }
    }
    D.b[3 * N + v] = v == D.pref_vid ? D.pref : bp;
}

// 4x4 block inverses for the block-Jacobi preconditioner
__global__ void __launch_bounds__(256) k_bj4_setup(int64_t nb, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                                   const double* __restrict__ val, double* __restrict__ binv, int* bad) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nb) return;
    double a[4][8];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int64_t row = r * nb + v;
        const int32_t s0 = rp[row], s1 = rp[row + 1];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int32_t col = (int32_t)(c * nb + v);
            int32_t lo = s0, hi = s1;  // binary search of the column in the sorted row
            while (lo < hi) {
                const int32_t mid = (lo + hi) >> 1;
                if (ci[mid] < col) lo = mid + 1;
                else hi = mid;
            }
            a[r][c] = (lo < s1 && ci[lo] == col) ? val[lo] : 0.0;
            a[r][4 + c] = r == c ? 1.0 : 0.0;
        }
    }
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int piv = k;
        double best = fabs(a[k][k]);
#pragma unroll
        for (int r = k + 1; r < 4; ++r)
            if (fabs(a[r][k]) > best) {
                best = fabs(a[r][k]);
                piv = r;
            }
        if (!(best > 0.0) || !isfinite(best)) ok = false;
#pragma unroll
        for (int c = 0; c < 8; ++c) {  // swap rows k and piv (branch-free over the unrolled rows)
#pragma unroll
            for (int r = k + 1; r < 4; ++r)
                if (r == piv) {
                    const double tmp = a[k][c];
                    a[k][c] = a[r][c];
                    a[r][c] = tmp;
                }
        }
        const double inv = ok ? 1.0 / a[k][k] : 0.0;
#pragma unroll
        for (int c = 0; c < 8; ++c) a[k][c] *= inv;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (r != k) {
                const double f = a[r][k];
#pragma unroll
                for (int c = 0; c < 8; ++c) a[r][c] -= f * a[k][c];
            }
    }
    if (!ok) atomicExch(bad, 1);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) binv[(r * 4 + c) * nb + v] = a[r][4 + c];
}

inline int blocks_for(int64_t threads) { return (int)((threads + 255) / 256); }

}  // namespace

void launch_ns_gsum(cudaStream_t s, const NsDev& D, double* gsum) { k_ns_gsum<<<blocks_for(D.n), 256, 0, s>>>(D, gsum); }

void launch_ns_assemble(cudaStream_t s, const NsDev& D) {
    k_ns_rc<<<blocks_for(D.n * kRowG), 256, 0, s>>>(D);
    k_ns_mom<<<blocks_for(D.n * kGradG), 256, 0, s>>>(D);
    k_ns_flux<<<blocks_for(D.n * kRowG), 256, 0, s>>>(D);
    k_ns_mom_rows<<<blocks_for(D.n * kMomG), 256, 0, s>>>(D);
    const int cap = D.max_len < kPCap ? (D.max_len + 1) & ~1 : kPCap;
    const unsigned blocks = (unsigned)((D.n + kPWarps - 1) / kPWarps);
    const size_t smem = (size_t)kPWarps * cap * sizeof(double);
    if (D.wide) k_ns_p_rows<uint32_t, false><<<blocks, 32 * kPWarps, smem, s>>>(D, cap);
    else if (D.max_len > cap) k_ns_p_rows<uint16_t, false><<<blocks, 32 * kPWarps, smem, s>>>(D, cap);
    else k_ns_p_rows<uint16_t, true><<<blocks, 32 * kPWarps, smem, s>>>(D, cap);
    k_ns_rhs<<<blocks_for(D.n * kRowG), 256, 0, s>>>(D);
}

void launch_bj4_setup(cudaStream_t s, int64_t nb, const int32_t* rp, const int32_t* ci, const double* val, double* binv, int* bad) {
    k_bj4_setup<<<blocks_for(nb), 256, 0, s>>>(nb, rp, ci, val, binv, bad);
}

}  // namespace vfv
