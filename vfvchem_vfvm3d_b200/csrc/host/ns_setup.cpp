// Symbolic setup of the coupled Navier-Stokes system; see ns_setup.hpp.
#include "ns_setup.hpp"

#include <algorithm>
#include <climits>
#include <cstdlib>

namespace vfv {

namespace {

struct GcEnt {
    int32_t vid;
    double c[3];
};

// Tetrahedron::update_tet step 6 (geom_tet.rs:295-347) for one vertex, in push order:
// per face the arithmetic-mean pair (v, n), then the skew terms of the LSQ gradients of v and of n
// ((m, +w) and (s, -w) per neighbour m of s), then the boundary sub-faces (v, j, k).
void gc_push_order(const Dual& d, int64_t v, std::vector<GcEnt>& e) {
    const int64_t D = d.n_dir, B = (int64_t)d.bnd_j.size();
    e.clear();
    for (int64_t i = d.nbr_ptr[v]; i < d.nbr_ptr[v + 1]; ++i) {
        const int32_t nb = d.nbr_idx[i];
        const double area = d.area[i];
        const double nx = d.norm[i], ny = d.norm[D + i], nz = d.norm[2 * D + i];
        const double sx = d.skew[i], sy = d.skew[D + i], sz = d.skew[2 * D + i];
        e.push_back({(int32_t)v, {0.5 * area * nx, 0.5 * area * ny, 0.5 * area * nz}});
        e.push_back({nb, {0.5 * area * nx, 0.5 * area * ny, 0.5 * area * nz}});
        const int64_t side[2] = {v, nb};
        for (int64_t s : side)
            for (int64_t k = d.nbr_ptr[s]; k < d.nbr_ptr[s + 1]; ++k) {
                const double w = 0.5 * (d.gw[k] * sx + d.gw[D + k] * sy + d.gw[2 * D + k] * sz) * area;
                e.push_back({d.nbr_idx[k], {w * nx, w * ny, w * nz}});
                e.push_back({(int32_t)s, {-w * nx, -w * ny, -w * nz}});
            }
    }
    for (int64_t b = d.bnd_ptr[v]; b < d.bnd_ptr[v + 1]; ++b) {
        const double area = d.bnd_area[b];
        const double nx = d.bnd_norm[b], ny = d.bnd_norm[B + b], nz = d.bnd_norm[2 * B + b];
        const double wv = d.bnd_wgt[b], wj = d.bnd_wgt[B + b], wk = d.bnd_wgt[2 * B + b];
        e.push_back({(int32_t)v, {wv * area * nx, wv * area * ny, wv * area * nz}});
        e.push_back({d.bnd_j[b], {wj * area * nx, wj * area * ny, wj * area * nz}});
        e.push_back({d.bnd_k[b], {wk * area * nx, wk * area * ny, wk * area * nz}});
    }
}

// The merge of slice::sort_by_key + dedup_by: a stable sort by vertex, then the entries of equal
// vertices summed in push order. Computed without sorting the entries: the first entry of a vertex
// keeps its place in `out` and the later ones are added to it in push order (the same sums), then
// the distinct vertices are sorted. stamp[u] == v marks vertex u as seen while merging vertex v's
// list; slot[u] is its place in `out`.
void gc_merge(const std::vector<GcEnt>& e, int32_t v, std::vector<int32_t>& stamp, std::vector<int32_t>& slot, std::vector<GcEnt>& out) {
    out.clear();
    for (const GcEnt& g : e) {
        if (stamp[g.vid] != v) {
            stamp[g.vid] = v;
            slot[g.vid] = (int32_t)out.size();
            out.push_back(g);
        } else {
            GcEnt& o = out[slot[g.vid]];
            for (int q = 0; q < 3; ++q) o.c[q] += g.c[q];
        }
    }
    std::sort(out.begin(), out.end(), [](const GcEnt& a, const GcEnt& b) { return a.vid < b.vid; });
}

int64_t deg(const Dual& d, int64_t v) { return d.nbr_ptr[v + 1] - d.nbr_ptr[v]; }

// Vertices of a set seen once each (stamp[u] == tag), in `out`.
struct VertexSet {
    std::vector<int32_t> stamp, out;
    int32_t tag = 0;
    explicit VertexSet(int64_t n) : stamp(n, 0) {}
    void start() {
        ++tag;
        out.clear();
    }
    void add(int32_t u) {
        if (stamp[u] != tag) {
            stamp[u] = tag;
            out.push_back(u);
        }
    }
};

// Q(v): the vertices of v's p row in the velocity fields (divergence and boundary sub-faces)
void collect_q(const Dual& d, const NsLayout& L, int64_t v, VertexSet& s) {
    s.start();
    s.add((int32_t)v);
    for (int64_t i = d.nbr_ptr[v]; i < d.nbr_ptr[v + 1]; ++i) {
        const int64_t nb = d.nbr_idx[i];
        s.add((int32_t)nb);
        for (int64_t k = d.nbr_ptr[nb]; k < d.nbr_ptr[nb + 1]; ++k) s.add(d.nbr_idx[k]);
    }
    if (v >= L.n_pts)
        for (int64_t b = d.bnd_ptr[v]; b < d.bnd_ptr[v + 1]; ++b) {
            s.add(d.bnd_j[b]);
            s.add(d.bnd_k[b]);
        }
}

// R(v): the vertices of v's p row in the pressure field (stabiliser)
void collect_r(const Dual& d, const NsLayout& L, int64_t v, VertexSet& s) {
    s.start();
    if (d.nbr_ptr[v] == d.nbr_ptr[v + 1]) return;
    s.add((int32_t)v);
    for (int32_t k = L.gcp[v]; k < L.gcp[v + 1]; ++k) s.add(L.gcv[k]);
    for (int64_t i = d.nbr_ptr[v]; i < d.nbr_ptr[v + 1]; ++i) {
        const int64_t nb = d.nbr_idx[i];
        s.add((int32_t)nb);
        for (int32_t k = L.gcp[nb]; k < L.gcp[nb + 1]; ++k) s.add(L.gcv[k]);
    }
}

}  // namespace

void build_grad_coeff(const Dual& d, NsLayout& L) {
    const int64_t n = d.n_tot;
    std::vector<std::vector<GcEnt>> per(n);
#pragma omp parallel
    {
        std::vector<GcEnt> e, m;
        std::vector<int32_t> stamp(n, -1), slot(n, 0);
#pragma omp for schedule(dynamic, 256)
        for (int64_t v = 0; v < n; ++v) {
            gc_push_order(d, v, e);
            gc_merge(e, (int32_t)v, stamp, slot, m);
            per[v] = m;
        }
    }
    L.gcp.assign(n + 1, 0);
    for (int64_t v = 0; v < n; ++v) L.gcp[v + 1] = L.gcp[v] + (int32_t)per[v].size();
    const int64_t ng = L.gcp[n];
    L.gcv.resize(ng);
    L.gcc.resize(3 * ng);
    for (int64_t v = 0; v < n; ++v)
        for (size_t k = 0; k < per[v].size(); ++k) {
            const int64_t t = L.gcp[v] + (int64_t)k;
            L.gcv[t] = per[v][k].vid;
            for (int q = 0; q < 3; ++q) L.gcc[q * ng + t] = per[v][k].c[q];
        }
}

std::string build_ns_layout(const Dual& d, int64_t pref_vid, NsLayout& L) {
    const int64_t n = d.n_tot, D = d.n_dir;
    if (4 * n >= (int64_t)INT_MAX) return "NS system too large for 32-bit row indices";
    if (pref_vid < 0 || pref_vid >= n) return "reference-pressure vertex out of range";
    L.n = n;
    L.n_pts = d.n_pts;
    L.pref_vid = pref_vid;
    build_grad_coeff(d, L);
    auto gcn = [&](int64_t v) -> int64_t { return L.gcp[v + 1] - L.gcp[v]; };
    const int64_t R = 4 * n, P = 3 * n;
    // pass 1: triplets, |Q|, |R| and the lengths of the place lists per vertex
    L.qlen.assign(n, 0);
    L.qself.assign(n, 0);
    L.rself.assign(n, 0);
    L.qoff.assign(n + 1, 0);
    L.roff.assign(n + 1, 0);
    std::vector<int32_t> rlen(n, 0);
    int64_t trips = 0;
#pragma omp parallel reduction(+ : trips)
    {
        VertexSet set(n);
#pragma omp for schedule(dynamic, 256)
        for (int64_t v = 0; v < n; ++v) {
            trips += 3 * (v < d.n_pts ? 4 * deg(d, v) + gcn(v) : 1);
            if (v == pref_vid) {
                trips += 1;
                continue;
            }
            if (v >= d.n_pts) trips += 9 * (d.bnd_ptr[v + 1] - d.bnd_ptr[v]);
            for (int64_t i = d.nbr_ptr[v]; i < d.nbr_ptr[v + 1]; ++i) {
                const int64_t nb = d.nbr_idx[i];
                trips += 6 + 6 * deg(d, v) + 6 * deg(d, nb) + 2 + gcn(v) + gcn(nb);
                L.qoff[v + 1] += deg(d, nb);
                L.roff[v + 1] += gcn(nb);
            }
            collect_q(d, L, v, set);
            L.qlen[v] = (int32_t)set.out.size();
            collect_r(d, L, v, set);
            rlen[v] = (int32_t)set.out.size();
        }
    }
    L.n_trip = trips;
    for (int64_t v = 0; v < n; ++v) {
        L.qoff[v + 1] += L.qoff[v];
        L.roff[v + 1] += L.roff[v];
        if (v != pref_vid) L.max_len = std::max<int64_t>(L.max_len, std::min<int64_t>(INT_MAX, 3 * (int64_t)L.qlen[v] + rlen[v]));
    }
    L.rp.assign(R + 1, 0);
    int64_t tot = 0;
    for (int64_t r = 0; r < R; ++r) {
        const int64_t v = r % n;
        if (r < P) tot += v < d.n_pts ? deg(d, v) + 1 + gcn(v) : 1;
        else tot += v == pref_vid ? 1 : 3 * (int64_t)L.qlen[v] + rlen[v];
        if (tot >= (int64_t)INT_MAX) return "NS pattern too large for 32-bit slot indices";
        L.rp[r + 1] = (int32_t)tot;
    }
    L.ci.resize(tot);  // ci and the place lists are written in full by pass 2 (but for the reference vertex)
    const char* force = getenv("VFV_NS_WIDE");  // diagnostics: 32-bit places
    const bool wide = L.max_len > 65535 || (force && force[0] == '1');
    const int64_t ng = (int64_t)L.gcv.size(), B = (int64_t)d.bnd_j.size();
    L.qring.resize(D, wide);
    L.rring.resize(D, wide);
    L.qnb.resize(L.qoff[n], wide);
    L.rgc.resize(ng, wide);
    L.rnb.resize(L.roff[n], wide);
    L.qsub.resize(2 * B, wide);
    // pass 2: columns and places
#pragma omp parallel
    {
        VertexSet set(n);
        std::vector<int32_t> pos(n, 0);
#pragma omp for schedule(dynamic, 256)
        for (int64_t v = 0; v < n; ++v) {
            for (int q = 0; q < 3; ++q) {  // momentum rows
                int32_t* c = L.ci.data() + L.rp[q * n + v];
                if (v >= d.n_pts) {
                    *c = (int32_t)(q * n + v);
                    continue;
                }
                int64_t i = d.nbr_ptr[v];
                const int64_t e = d.nbr_ptr[v + 1];
                for (; i < e && d.nbr_idx[i] < v; ++i) *c++ = (int32_t)(q * n + d.nbr_idx[i]);
                *c++ = (int32_t)(q * n + v);
                for (; i < e; ++i) *c++ = (int32_t)(q * n + d.nbr_idx[i]);
                for (int32_t k = L.gcp[v]; k < L.gcp[v + 1]; ++k) *c++ = (int32_t)(P + L.gcv[k]);
            }
            int32_t* c = L.ci.data() + L.rp[P + v];
            if (v == pref_vid) {
                *c = (int32_t)(P + v);
                continue;
            }
            collect_q(d, L, v, set);
            std::sort(set.out.begin(), set.out.end());
            for (int f = 0; f < 3; ++f)
                for (int32_t u : set.out) *c++ = (int32_t)(f * n + u);
            for (size_t t = 0; t < set.out.size(); ++t) pos[set.out[t]] = (int32_t)t;
            L.qself[v] = pos[v];
            int64_t o = L.qoff[v];
            for (int64_t i = d.nbr_ptr[v]; i < d.nbr_ptr[v + 1]; ++i) {
                const int64_t nb = d.nbr_idx[i];
                L.qring.set(i, pos[nb]);
                for (int64_t k = d.nbr_ptr[nb]; k < d.nbr_ptr[nb + 1]; ++k) L.qnb.set(o++, pos[d.nbr_idx[k]]);
            }
            if (v >= d.n_pts)
                for (int64_t b = d.bnd_ptr[v]; b < d.bnd_ptr[v + 1]; ++b) {
                    L.qsub.set(b, pos[d.bnd_j[b]]);
                    L.qsub.set(B + b, pos[d.bnd_k[b]]);
                }
            collect_r(d, L, v, set);
            std::sort(set.out.begin(), set.out.end());
            for (int32_t u : set.out) *c++ = (int32_t)(P + u);
            for (size_t t = 0; t < set.out.size(); ++t) pos[set.out[t]] = (int32_t)t;
            L.rself[v] = pos[v];
            o = L.roff[v];
            for (int32_t k = L.gcp[v]; k < L.gcp[v + 1]; ++k) L.rgc.set(k, pos[L.gcv[k]]);
            for (int64_t i = d.nbr_ptr[v]; i < d.nbr_ptr[v + 1]; ++i) {
                const int64_t nb = d.nbr_idx[i];
                L.rring.set(i, pos[nb]);
                for (int32_t k = L.gcp[nb]; k < L.gcp[nb + 1]; ++k) L.rnb.set(o++, pos[L.gcv[k]]);
            }
        }
    }
    return "";
}

}  // namespace vfv
