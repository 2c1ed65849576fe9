// The backward sweep of the discrete adjoint as one cooperative launch, for grids whose adjoint state
// stays in L2: the transposes of adjoint_kernels.cuh in place, half a step at a time, with the grid-wide
// barrier of stencil_resident.cuh between the halves.
//
// Per step n, downwards. Phase 1 forms lambda_H' from lambda_E, the E psi adjoints and the coefficients
// (k_adj_e's sums); lambda_E does not change in it, so the gradient's sums and every neighbour read settled
// values. Phase 2 forms lambda_E from lambda_H' and the H psi adjoints (k_adj_h's). A psi adjoint is
// advanced by its own edge one phase after its neighbours read it: E's in phase 2, H's in the phase 1 of
// the next step. So nothing ping-pongs, and a step moves 72 B per node through L2 instead of 96 through
// a march whose blocks are chains of planes (k_adj_step: 141 us a step at 161x161x97).
// The objective's source joins where its node is formed: lambda_E's of step n - 1 at the end of phase 2,
// lambda_H's of step n in phase 1. With Debye media a phase 0 comes first: the Debye ADE's transpose on
// the edge list (k_adj_debye_post of step n + 1, the source on those edges, k_adj_debye_pre of step n).
// Every sum is formed in the order of the separate launches, so the gradient equals theirs bit for bit.
#pragma once

#include "adjoint_kernels.cuh"
#include "stencil_resident.cuh"

namespace fg {

struct AdjResArgs {
    ResArgs r;                       // grid, classes, barrier, index arithmetic; e, h: lambda_E, lambda_H
    float* psi;                      // the psi adjoints
    long long n_hi;                  // steps n_hi - 1 down to n_hi - r.steps
    // the source: the window of the flux plane, its weights and the steps' phase factors
    int plane_k, i0, wi, j0, wj;
    const float* w;
    const float* dft;
    // the gradient
    const float *hist_e, *hist_s;
    double *ga, *gb;
    // Debye (r.debye_*): adjoint states, each edge's term for the step before, each edge's window node
    // (2 node + comp, or -1) and, per window node, which of Ex, Ey are Debye edges
    float *ls, *lold;
    const int* dwin;
    const uint8_t* wmask;
};

// The adjoint's factors of a row node: {inv, slot, c raw, b} of H and E.
struct __align__(16) AdjNode {
    ResHalf f[2];
};
inline size_t adj_res_smem(const Geom& g) { return size_t(res_pad(g.n0) + res_pad(g.n1) + res_pad(g.n2)) * 8 * 4; }

__device__ __forceinline__ void adj_fill_rows(AdjNode* t, int n, const AxisNode* ax) {
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
        const AxisNode v = ax[q];
        t[q].f[0] = ResHalf{v.inv_d, v.slot_h, v.ch * v.raw_inv_d, v.bh};
        t[q].f[1] = ResHalf{v.inv_dd, v.slot_e, v.ce * v.raw_inv_dd, v.be};
    }
}

// Along k: inv, c raw and b of H then E as six arrays (zero outside the layer and past the axis), then the
// groups' first slots (res_fill_k).
__device__ __forceinline__ void adj_fill_k(float* z, int n, const AxisNode* ax) {
    const int np = res_pad(n);
    int* slot = reinterpret_cast<int*>(z + 6 * np);
    for (int q = threadIdx.x; q < np; q += blockDim.x) {
        AxisNode v{0, 0, 0, 0, 0, 0, 0, 0, -1, -1};
        if (q < n) v = ax[q];
        const bool le = v.slot_e >= 0, lh = v.slot_h >= 0;
        z[q] = v.inv_d;
        z[np + q] = lh ? v.ch * v.raw_inv_d : 0.f;
        z[2 * np + q] = lh ? v.bh : 0.f;
        z[3 * np + q] = v.inv_dd;
        z[4 * np + q] = le ? v.ce * v.raw_inv_dd : 0.f;
        z[5 * np + q] = le ? v.be : 0.f;
        if (q < np / 4) {
            int first = -1;
            for (int t = 0; t < 4 && 4 * q + t < n; ++t) {
                const int e = ax[4 * q + t].slot_e, h = ax[4 * q + t].slot_h;
                if (e >= 0) first = e - t;
                else if (h >= 0) first = h - t;
            }
            slot[q] = first;
        }
    }
}

struct AdjPos {
    unsigned row, id;   // the row, and the group's first node
    int i, j, k;
};

// The psi slab offset of component c along `axis` at a position: of row slots (i, j), of the group along k.
template <int F>
__device__ __forceinline__ unsigned adj_psi_row(const Geom& g, int c, int axis, int i, int j, int k, int slot) {
    return unsigned(g.psi_off[(F ? 0 : 9) + c * 3 + axis]) + unsigned(k) +
           (axis == 0 ? unsigned(slot) * unsigned(g.n1) + unsigned(j) : unsigned(i) * unsigned(2 * g.pml) + unsigned(slot)) *
               unsigned(g.pk);
}

// What edge c's adjoint feeds its two differences at a group: gg = cb lambda_E (F = 1; 0 where the edge does
// not update), gh = -k_mu lambda_H (F = 0; 0 where a neighbour lies past the grid).
template <int c, int F, typename CID>
__device__ __forceinline__ Quad adj_drive(const AdjResArgs& A, unsigned id, int i, int j, int k, float2 z) {
    const Geom& g = A.r.g;
    const Quad v = ld4((F ? A.r.e : A.r.h) + (unsigned(c) * unsigned(g.cs) + id));
    Quad o;
    if constexpr (F) {
        const uint4 cid = res_ids(static_cast<const CID*>(A.r.node_class) + id);
        const float* t = reinterpret_cast<const float*>(A.r.classes) + (4 + c);
        const float b0 = __ldg(t + cid.x * 8);
        Quad b = q_bc(b0);
        if (cid.y != cid.x || cid.z != cid.x || cid.w != cid.x)
            b = Quad{make_float2(b0, __ldg(t + cid.y * 8)), make_float2(__ldg(t + cid.z * 8), __ldg(t + cid.w * 8))};
        o = q_mul(b, v, z);
        const bool rowok = (c == 0 || i > 0) && (c == 1 || j > 0);
        if (!rowok) o = q_zero();
        if (c != 2 && k == 0) o.a.x = 0.f;
    } else {
        o = q_mul(q_bc(-A.r.k_mu), v, z);
        const bool rowok = (c == 0 || i + 1 < g.n0) && (c == 1 || j + 1 < g.n1);
        if (!rowok) o = q_zero();
        if (c != 2) {   // nodes k + 1 inside the grid
            const int nk = g.n2 - k;
            o.a = f2::pick(nk > 1, nk > 2, o.a, make_float2(0.f, 0.f));
            o.b = f2::pick(nk > 3, nk > 4, o.b, make_float2(0.f, 0.f));
        }
    }
    return o;
}
// The same at one node (its drive's own tests along k included).
template <int c, int F, typename CID>
__device__ __forceinline__ float adj_drive_one(const AdjResArgs& A, unsigned id, int i, int j, int k) {
    const Geom& g = A.r.g;
    const float v = (F ? A.r.e : A.r.h)[unsigned(c) * unsigned(g.cs) + id];
    if constexpr (F) {
        const float b = __ldg(reinterpret_cast<const float*>(A.r.classes) + (4 + c) +
                              unsigned(static_cast<const CID*>(A.r.node_class)[id]) * 8);
        return (c == 0 || i > 0) && (c == 1 || j > 0) && (c == 2 || k > 0) ? b * v : 0.f;
    } else {
        return (c == 0 || i + 1 < g.n0) && (c == 1 || j + 1 < g.n1) && (c == 2 || k + 1 < g.n2) ? -A.r.k_mu * v : 0.f;
    }
}

// s gg inv + (c raw) (s gg + psi): the adjoint of one difference.
template <int SIGN>
__device__ __forceinline__ Quad adj_signed(const Quad& q) {
    if constexpr (SIGN > 0) return q;
    return Quad{make_float2(-q.a.x, -q.a.y), make_float2(-q.b.x, -q.b.y)};
}

// The difference along i or j (AXIS) of edge c's adjoint over its neighbour on that axis: value(q) -
// value(q + 1) for F = 1, value(q - 1) - value(q) for F = 0.
template <int c, int AXIS, int SIGN, int F, typename CID>
__device__ __forceinline__ Quad adj_row_term(const AdjResArgs& A, const AdjNode* T, const AdjPos& p, float2 z) {
    const Geom& g = A.r.g;
    const int at = AXIS == 0 ? p.i : p.j, n = AXIS == 0 ? g.n0 : g.n1;
    const unsigned st = AXIS == 0 ? unsigned(g.n1) * unsigned(g.p2) : unsigned(g.p2);
    auto value = [&](int d) {
        const int i = p.i + (AXIS == 0 ? d : 0), j = p.j + (AXIS == 1 ? d : 0);
        const unsigned id = d > 0 ? p.id + st : (d < 0 ? p.id - st : p.id);
        const ResHalf f = T[at + d].f[F];
        const Quad gg = adj_signed<SIGN>(adj_drive<c, F, CID>(A, id, i, j, p.k, z));
        Quad v = q_mul(gg, q_bc(f.inv), z);
        if (f.slot >= 0)
            v = v + q_mul(q_bc(f.raw), gg + ld4(A.psi + adj_psi_row<F>(g, c, AXIS, i, j, p.k, f.slot)), z);
        return v;
    };
    const Quad own = value(0);
    if constexpr (F) return at + 1 < n ? own - value(1) : own - q_zero();
    else return at > 0 ? value(-1) - own : q_zero() - own;
}

// The same along k.
template <int c, int SIGN, int F, typename CID>
__device__ __forceinline__ Quad adj_k_term(const AdjResArgs& A, const float* Z, int np, const AdjPos& p, float2 z) {
    const Geom& g = A.r.g;
    const float* zf = Z + (F ? 3 : 0) * np;
    const int* slots = reinterpret_cast<const int*>(Z + 6 * np);
    const unsigned off = unsigned(g.psi_off[(F ? 0 : 9) + c * 3 + 2]) + p.row * unsigned(g.pw);
    const Quad gg = adj_signed<SIGN>(adj_drive<c, F, CID>(A, p.id, p.i, p.j, p.k, z));
    Quad v = q_mul(gg, ld4(zf + p.k), z);
    const int sl = slots[p.k >> 2];
    if (sl >= 0) v = v + q_mul(ld4(zf + np + p.k), gg + ld4(A.psi + (off + unsigned(sl))), z);
    const int k1 = F ? p.k + 4 : p.k - 1;   // the node past the group that the difference reads
    float e = 0.f;
    if (k1 >= 0 && k1 < g.n2) {
        const float g1 = SIGN * adj_drive_one<c, F, CID>(A, F ? p.id + 4 : p.id - 1, p.i, p.j, k1);
        e = g1 * zf[k1];
        const int s1 = slots[k1 >> 2];
        if (s1 >= 0) e += zf[np + k1] * (g1 + A.psi[off + unsigned(s1 + (k1 & 3))]);
    }
    return F ? v - q_up(v, e) : q_down(v, e) - v;
}

// Component C's two terms, in the order of k_adj_e and k_adj_h.
template <int C, int F, typename CID>
__device__ __forceinline__ Quad adj_terms2(const AdjResArgs& A, const AdjNode* X, const AdjNode* Y, const float* Z, int np,
                                           const AdjPos& p, float2 z) {
    if constexpr (C == 0) return adj_k_term<1, 1, F, CID>(A, Z, np, p, z) + adj_row_term<2, 1, -1, F, CID>(A, Y, p, z);
    else if constexpr (C == 1) return adj_row_term<2, 0, 1, F, CID>(A, X, p, z) + adj_k_term<0, -1, F, CID>(A, Z, np, p, z);
    else return adj_row_term<0, 1, 1, F, CID>(A, Y, p, z) + adj_row_term<1, 0, -1, F, CID>(A, X, p, z);
}

// b (s gg + psi) into the two psi adjoints of edge C at the group (its axes C + 1 with +, C + 2 with -).
template <int C, int F>
__device__ __forceinline__ void adj_advance(const AdjResArgs& A, const AdjNode* X, const AdjNode* Y, const float* Z, int np,
                                            const AdjPos& p, const Quad& gg, float2 z) {
    const Geom& g = A.r.g;
    auto one = [&](auto axis, auto sign) {
        constexpr int AX = decltype(axis)::value, SG = decltype(sign)::value;
        if constexpr (AX == 2) {
            const int sl = reinterpret_cast<const int*>(Z + 6 * np)[p.k >> 2];
            if (sl >= 0) {
                float* q = A.psi + (unsigned(g.psi_off[(F ? 0 : 9) + C * 3 + 2]) + p.row * unsigned(g.pw) + unsigned(sl));
                st4(q, q_mul(ld4(Z + (F ? 5 : 2) * np + p.k), adj_signed<SG>(gg) + ld4(q), z));
            }
        } else {
            const ResHalf f = (AX == 0 ? X[p.i] : Y[p.j]).f[F];
            if (f.slot >= 0) {
                float* q = A.psi + adj_psi_row<F>(g, C, AX, p.i, p.j, p.k, f.slot);
                st4(q, q_mul(q_bc(f.b), adj_signed<SG>(gg) + ld4(q), z));
            }
        }
    };
    one(std::integral_constant<int, (C + 1) % 3>{}, std::integral_constant<int, 1>{});
    one(std::integral_constant<int, (C + 2) % 3>{}, std::integral_constant<int, -1>{});
}

// The source of step n on component c (0, 1) of E (F = 1) or H (F = 0) at window node t (adj_inject).
template <int F>
__device__ __forceinline__ float adj_source(const AdjResArgs& A, long long n, int c, int t) {
    const float4 d = __ldg(reinterpret_cast<const float4*>(A.dft) + n);
    const float* w = A.w + (long long)t * 8 + (F ? 0 : 4) + 2 * c;
    return F ? 2.0f * (w[0] * d.x - w[1] * d.y) : 2.0f * (w[0] * d.z + w[1] * d.w);
}

// Adds the source to the group's node on the flux plane, if it has one. `skip`: not on Debye edges.
template <int C, int F>
__device__ __forceinline__ void adj_join(const AdjResArgs& A, const AdjPos& p, long long n, Quad& v, bool skip) {
    if constexpr (C == 2) return;
    if (p.k >> 2 != A.plane_k >> 2 || unsigned(p.i - A.i0) >= unsigned(A.wi) || unsigned(p.j - A.j0) >= unsigned(A.wj)) return;
    const int t = (p.i - A.i0) * A.wj + (p.j - A.j0);
    if (skip && (A.wmask[t] >> C & 1)) return;
    const float s = adj_source<F>(A, n, C, t);
    const int l = A.plane_k & 3;
    if (l == 0) v.a.x += s;
    else if (l == 1) v.a.y += s;
    else if (l == 2) v.b.x += s;
    else v.b.y += s;
}

// A warp's share of a phase: component C of the groups from `first` on (res_half's walk).
template <int C, int F, typename CID>
__device__ __forceinline__ void adj_half(const AdjResArgs& A, const AdjNode* X, const AdjNode* Y, const float* Z, int np,
                                         unsigned first, long long n) {
    const ResArgs& a = A.r;
    const float2 z = make_float2(a.neg0, a.neg0);
    ResWalk<F == 0> at(a, first);   // the second phase walks backwards (res_half)
    while (at.inside(a)) {
        const AdjPos p{unsigned(at.row), unsigned(at.row) * unsigned(a.g.p2) + unsigned(at.col) * 4u, at.i, at.j, at.col * 4};
        const unsigned ido = unsigned(C) * unsigned(a.g.cs) + p.id;
        const int nk = a.g.n2 - p.k;
        if constexpr (F) {
            // lambda_H'; the psi adjoints of H first take their step from the lambda_H it replaces
            const Quad t = adj_terms2<C, 1, CID>(A, X, Y, Z, np, p, z);
            adj_advance<C, 0>(A, X, Y, Z, np, p, adj_drive<C, 0, CID>(A, p.id, p.i, p.j, p.k, z), z);
            Quad v = ld4(a.h + ido);
            adj_join<C, 0>(A, p, n, v, false);
            v = v + t;
            v.a = f2::pick(true, nk > 1, v.a, make_float2(0.f, 0.f));   // the padding past the row stays 0
            v.b = f2::pick(nk > 2, nk > 3, v.b, make_float2(0.f, 0.f));
            st4(a.h + ido, v);
        } else {
            // lambda_E; the psi adjoints of E take their step from the lambda_E it replaces
            const Quad t = adj_terms2<C, 0, CID>(A, X, Y, Z, np, p, z);
            const Quad l = ld4(a.e + ido);
            const uint4 cid = res_ids(static_cast<const CID*>(a.node_class) + p.id);
            const float* f = reinterpret_cast<const float*>(a.classes) + C;
            const unsigned id4[4] = {cid.x, cid.y, cid.z, cid.w};
            const bool rowok = (C == 0 || p.i > 0) && (C == 1 || p.j > 0);
            float ca[4], cb[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float b = __ldg(f + id4[q] * 8 + 4);
                const bool m = rowok && b != 0.f && (C == 2 || p.k + q > 0);
                ca[q] = m ? __ldg(f + id4[q] * 8) : 1.f;
                cb[q] = m ? b : 0.f;
            }
            Quad v = q_mul(Quad{make_float2(ca[0], ca[1]), make_float2(ca[2], ca[3])}, l, z) + t;
            adj_advance<C, 1>(A, X, Y, Z, np, p, q_mul(Quad{make_float2(cb[0], cb[1]), make_float2(cb[2], cb[3])}, l, z), z);
            if (n > 0) adj_join<C, 1>(A, p, n - 1, v, a.n_debye > 0);
            v.a = f2::pick(true, nk > 1, v.a, make_float2(0.f, 0.f));
            v.b = f2::pick(nk > 2, nk > 3, v.b, make_float2(0.f, 0.f));
            st4(a.e + ido, v);
        }
        at.next(a);
    }
}

template <int F, typename CID>
__device__ __forceinline__ void adj_field(const AdjResArgs& A, int comp, const AdjNode* X, const AdjNode* Y, const float* Z, int np,
                                          unsigned first, long long n) {
    if (comp == 0) adj_half<0, F, CID>(A, X, Y, Z, np, first, n);
    else if (comp == 1) adj_half<1, F, CID>(A, X, Y, Z, np, first, n);
    else adj_half<2, F, CID>(A, X, Y, Z, np, first, n);
}

template <typename CID, bool CLUSTER>
__global__ void __launch_bounds__(RES_THREADS, 1) k_adj_resident(const __grid_constant__ AdjResArgs A) {
    extern __shared__ __align__(16) float adj_res_sm[];
    const ResArgs& a = A.r;
    const Geom& g = a.g;
    const int np = res_pad(g.n2);
    AdjNode *X = reinterpret_cast<AdjNode*>(adj_res_sm), *Y = X + res_pad(g.n0);
    float* Z = reinterpret_cast<float*>(Y + res_pad(g.n1));
    adj_fill_rows(X, g.n0, g.ax[0]);
    adj_fill_rows(Y, g.n1, g.ax[1]);
    adj_fill_k(Z, g.n2, g.ax[2]);
    __syncthreads();
    const int w = threadIdx.x >> 5, comp = w % 3;
    const unsigned groups = blockDim.x / 3u, G = gridDim.x, b = blockIdx.x;
    const unsigned first = b * groups + unsigned(w / 3) * 32u + (threadIdx.x & 31u);
    auto t = [] { return int(((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32u + (threadIdx.x & 31u)); };   // k_resident's
    auto nt = [] { return int(gridDim.x * blockDim.x); };
    unsigned target = a.late;
    for (long long n = A.n_hi - 1; n >= A.n_hi - a.steps; --n) {
        if (a.n_debye) {
            for (int q = t(); q < a.n_debye; q += nt()) {
                const long long fi = a.debye_f[q];
                float l = a.e[fi] + A.lold[q];
                const int dw = A.dwin[q];
                if (dw >= 0) l += adj_source<1>(A, n, dw & 1, dw >> 1);
                const float wd = a.debye_dd[q], cb = a.debye_cb[q];
                const int poles = int(a.debye_table[0]);
                float d = 0.0f;
                for (int k = 0; k < poles; ++k) d += wd * a.debye_table[2 + 2 * k] * A.ls[(long long)k * a.n_debye + q];
                const float le = l + d;
                a.e[fi] = le;
                for (int k = 0; k < poles; ++k) {
                    const long long p = (long long)k * a.n_debye + q;
                    A.ls[p] = a.debye_table[1 + 2 * k] * A.ls[p] - cb * (0.5f * (1.0f + a.debye_table[1 + 2 * k])) * le;
                }
                A.lold[q] = -d;
            }
            if (!res_barrier<CLUSTER>(a, target += G)) return;
        }
        const long long slot = n * a.n_design;
        for (int q = t(); q < a.n_design; q += nt()) {   // adj_grad; no design edge is a Debye edge
            const int4 d = a.design[q];
            const double l = a.e[d.x * g.cs + ((long long)d.y * g.n1 + d.z) * g.p2 + d.w];
            A.ga[q] += l * double(A.hist_e[slot + q]);
            A.gb[q] += l * double(A.hist_s[slot + q]);
        }
        adj_field<1, CID>(A, comp, X, Y, Z, np, first, n);
        if (!res_barrier<CLUSTER>(a, target += G)) return;
        adj_field<0, CID>(A, comp, X, Y, Z, np, first, n);
        if (!res_barrier<CLUSTER>(a, target += G)) return;
    }
}

// Which Debye edges are window nodes of the flux plane: per edge its window node (2 node + comp, or -1),
// per window node bit c where E_c is a Debye edge (wmask as 32-bit words, zeroed).
__global__ void k_adj_debye_window(const long long* __restrict__ f, int count, Geom g, int plane_k, int i0, int wi, int j0, int wj,
                                   int* __restrict__ dwin, unsigned* __restrict__ wmask) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= count) return;
    const int c = int(f[q] / g.cs);
    const long long id = f[q] - c * g.cs, row = id / g.p2;
    const int k = int(id - row * g.p2), i = int(row / g.n1), j = int(row - (long long)i * g.n1);
    int out = -1;
    if (c < 2 && k == plane_k && i >= i0 && i < i0 + wi && j >= j0 && j < j0 + wj) {
        const int t = (i - i0) * wj + (j - j0);
        out = 2 * t + c;
        atomicOr(wmask + (t >> 2), 1u << (8 * (t & 3) + c));
    }
    dwin[q] = out;
}

// The source of the sweep's first step on lambda_E (Debye edges take theirs in their phase).
__global__ void k_adj_source_e(const __grid_constant__ AdjResArgs A) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= A.wi * A.wj) return;
    const Geom& g = A.r.g;
    const long long id = ((long long)(A.i0 + t / A.wj) * g.n1 + (A.j0 + t % A.wj)) * g.p2 + A.plane_k;
    for (int c = 0; c < 2; ++c)
        if (!(A.r.n_debye > 0 && (A.wmask[t] >> c & 1))) A.r.e[c * g.cs + id] += adj_source<1>(A, A.n_hi - 1, c, t);
}

}  // namespace fg
