// Symbolic setup of the coupled Navier-Stokes system (SteadyFlow, src/steady/core/steady_flow.rs)
// on the Voronoi dual: pressure-gradient coefficients, the CSR pattern of the reference's triplets
// and, for the pressure rows, the place of every contribution in its row.
//
// Unknowns are field-major, [u | v | w | p], n entries each (OperatorBase::add_vecvec_a and
// friends, src/operator/operator_base.rs:37-94). Every operator of SteadyFlow::assemble_matrix
// (steady_flow.rs:255-303) pushes only into the rows of the vertex it visits, so the push order
// restricted to one row is the operator order followed by the face order of that vertex:
//   u/v/w rows of a point:  advection (n, v per face), pressure gradient (grad_coeff of v),
//                           diffusion (n, v per face)
//   u/v/w rows of a node:   the Dirichlet diagonal
//   p row of a point:       divergence (per face: 6 + 6 deg v + 6 deg n), pressure stabiliser
//                           (per face: 2 + |gc v| + |gc n|)
//   p row of a node:        divergence faces, then 9 per boundary sub-face, then the stabiliser
//   p row of the reference vertex: the single diagonal (OpSclDomPressureReference drops the rest)
// So a momentum row holds its own field's {v} and neighbours, then the pressures of grad_coeff(v); a
// p row holds the same vertices Q(v) (v, its neighbours and theirs) in each of the fields u, v, w and
// the vertices R(v) (v, its neighbours, grad_coeff(v) and grad_coeff of the neighbours) in the field
// p, all ascending. The device adds a contribution straight to its place in Q(v) or R(v).
#pragma once
#include <cstdint>
#include <memory>
#include <new>
#include <string>
#include <type_traits>
#include <utility>
#include <vector>

#include "mesh.hpp"

namespace vfv {

// Allocator whose value-less construct default-initialises, so resize() of the large layout
// arrays leaves their (trivial) elements unset instead of zeroing gigabytes that the setup then
// overwrites; the parallel pass that writes them touches the pages first.
template <typename T>
struct UninitAlloc : std::allocator<T> {
    template <typename U>
    struct rebind { using other = UninitAlloc<U>; };
    UninitAlloc() = default;
    template <typename U>
    UninitAlloc(const UninitAlloc<U>&) noexcept {}
    template <typename U>
    void construct(U* p) noexcept(std::is_nothrow_default_constructible<U>::value) { ::new (static_cast<void*>(p)) U; }
    template <typename U, typename... A>
    void construct(U* p, A&&... a) { ::new (static_cast<void*>(p)) U(std::forward<A>(a)...); }
};
template <typename T>
using uninit_vector = std::vector<T, UninitAlloc<T>>;

// Places within a row, 16 bits each unless some row is longer than that.
struct NsPlaces {
    int64_t n = 0;
    uninit_vector<uint16_t> p16;
    uninit_vector<uint32_t> p32;
    bool wide = false;
    void resize(int64_t count, bool wide_) {
        n = count;
        wide = wide_;
        if (wide) p32.resize(count);
        else p16.resize(count);
    }
    void set(int64_t i, int32_t v) {
        if (wide) p32[i] = (uint32_t)v;
        else p16[i] = (uint16_t)v;
    }
    const void* data() const { return wide ? (const void*)p32.data() : (const void*)p16.data(); }
    size_t bytes() const { return (size_t)n * (wide ? 4 : 2); }
};

struct NsLayout {
    int64_t n = 0, n_pts = 0, pref_vid = 0, n_trip = 0;
    // Tetrahedron::grad_coeff (geom_tet.rs:295-347) as a CSR over vertices, ascending vertex ids
    std::vector<int32_t> gcp;        // [n + 1]
    std::vector<int32_t> gcv;        // [n_gc]
    std::vector<double> gcc;         // [3][n_gc]
    // pattern
    std::vector<int32_t> rp;         // CSR of the 4n x 4n matrix: row pointer [4n + 1]
    uninit_vector<int32_t> ci;       // [nnz] columns
    // places in the p rows (unset for the reference vertex)
    int32_t max_len = 0;             // entries of the longest p row
    std::vector<int32_t> qlen;       // [n] |Q(v)|
    std::vector<int32_t> qself, rself;    // [n] place of v in Q(v), R(v)
    std::vector<int64_t> qoff, roff;      // [n + 1] start of v's lists in qnb, rnb
    NsPlaces qring, rring;           // [n_dir] neighbour i of v in Q(v), R(v)
    NsPlaces qnb;                    // per face i of v in order: the neighbours of its neighbour, in Q(v)
    NsPlaces rgc;                    // [n_gc] grad_coeff entries of v in R(v)
    NsPlaces rnb;                    // per face i of v in order: grad_coeff entries of its neighbour, in R(v)
    NsPlaces qsub;                   // [2][n_bsub] boundary sub-face vertices j, k in Q(v)
    int64_t nnz() const { return (int64_t)ci.size(); }
    int64_t ntrip() const { return n_trip; }
};

// Pressure-gradient coefficients: per vertex, the (vertex, c) pairs of the Green-Gauss gradient
// with skew-corrected face values, merged by vertex in push order (stable sort, then ordered sums).
void build_grad_coeff(const Dual& d, NsLayout& L);

// Full symbolic setup (grad_coeff included). Returns "" or an error message.
std::string build_ns_layout(const Dual& d, int64_t pref_vid, NsLayout& L);

}  // namespace vfv
