// Many time steps in one launch: a cooperative kernel with the whole grid's blocks resident steps E and H
// in place, half a step at a time, with a grid-wide barrier between the halves (two per step; a third where
// a design history follows the E half). For grids of up to 23 M nodes by the fused step, and every separate
// run whose axes' factors fit shared memory (engine.cu, RES_MAX_FUSED and RES_MAX_AXES).
//
// The march kernels move each field once per step through HBM, but a march is a chain of planes: a
// small grid leaves most SMs idle behind it (65^3: 42 blocks, 33 us a step). In place, a half step
// has no order inside it, so every 4-node group of the grid is one thread's own work; a step costs its
// traffic (72 B per node) and two barriers instead of three to six kernel launches. The fields (24 B per
// node) and psi of up to about 4 M nodes stay in the 126 MB L2 from step to step, but that is not what
// bounds it: 121^3 takes 15.1 ps a node, 201^3 15.6, 261^3 14.9, where the march takes 10.7 at 513^3. A
// half step's chain does: class ids, L2 loads, the arithmetic, the barrier.
//
// Phase A of step n: new H from E (psi of H included); the records that read E after step n - 1
// (port voltages, running DFTs of E, the NTFF box's M); each design edge's E^n.
// Phase B: new E from H with the Debye ADE, the source and the inductors on the edges of the block's own nodes; the
// records that read H^n+1/2 (port currents, DFTs of H, the box's J). E does not change in phase A nor
// H in phase B, so each record reads a settled field without a barrier of its own.
// Phase C (only with a design history): the design edges' curl terms.
//
// The Debye ADE needs an edge's E before and after its update, both in the hands of the thread that
// updates it, so it runs there, on weights and pole states laid out by 4-node groups (dense in the groups
// that hold a Debye edge, 0 on their other edges, which leaves those as they are). As a pass of its own
// over the edge list it cost a save of E, a third barrier and 41 bytes an edge: 41^3 9.0 us a step
// against 6.3 now, 89^3 18.6 against 16.8, 121^3 31.2 against 28.5 (each a fifth of its spheres Debye;
// 5.8, 14.4 and 26.7 without them).
//
// The arithmetic and its order are those of the other pipelines (cpu.rs:48-167, :239-265, :291-415),
// so the fields equal theirs bit for bit. A launch of an odd number of steps writes its first step
// to the other buffer set, so that the latest set stays the one the parity of the step count names.
#pragma once

#include <type_traits>
#include <vector>

#include "kernels.cuh"
#include "stencil_tma.cuh"

namespace fg {

// n / d for n < 2^31 by one 64-bit product.
struct FastDiv {
    unsigned d = 1, s = 0;
    unsigned long long m = 1;
    __host__ __device__ FastDiv() {}
    __host__ explicit FastDiv(unsigned div) : d(div) {
        while ((1ull << s) < div) ++s;
        m = ((1ull << (32 + s)) + div - 1) / div;
    }
    __host__ __device__ __forceinline__ unsigned operator()(unsigned n) const {
        return unsigned(((unsigned long long)n * m) >> (32 + s));
    }
};

struct ResArgs {
    Geom g;
    const void* node_class;
    const DevCoef* classes;
    const float *e_src, *h_src, *psi_h_src;   // what the first step reads
    float *e, *h, *psi_h, *psi_e;             // what every step writes, and all but the first read
    float k_mu;
    float neg0;                               // -0.0f (f2::mul's addend)
    int steps;
    unsigned* counter;                        // the steps done before the launch
    unsigned* bar;                            // the grid barrier's arrivals, 0 at launch
    int* error;
    unsigned long long wait_ns;
    unsigned late;                            // test knob, 0 in normal runs: arrivals every barrier waits for in vain
    FastDiv quads, rows;                      // 4-node groups per row; rows per plane
    unsigned last_row;                        // the grid's last row
    unsigned dq, drow, dj, di;                // a pass of the launch over its groups, as rows and groups; its rows as planes and rows
    // Debye edges: the list (the adjoint's) and the layout by groups
    const long long* debye_f;
    const float *debye_dd, *debye_cb, *debye_table;
    int n_debye;
    const int* rd_index;                      // per group: its place among the groups with Debye edges, or -1
    const float* rd_dd;                       // weights: [place][component][node]
    float* rd_state;                          // pole states: [pole][place][component][node]
    unsigned rd_pole;                         // floats of a pole
    // source, inductors, ports
    const DevSource* src;
    DevInductor* ind;
    const DevProbe* probes;
    const DevPortEdge* pe;
    const DevLoop* lp;
    float* series;
    int ns, ni, n_ports;
    StepConst sc;
    // records
    int plane_k;
    float* plane;                             // null: none
    const unsigned* patch;
    float* ntff;
    int n_patches;
    // the design history
    const int4* design;
    int n_design;
    const long long* hist_base;
    int hist_cap;
    float *hist_e, *hist_s;
};

constexpr int RES_GROUPS = 320;             // 4-node groups a block takes at a time, at most
constexpr int RES_THREADS = 3 * RES_GROUPS;   // a thread per group and component
constexpr int RES_CLUSTER = 16;             // blocks of a launch on the smallest grids: one cluster
constexpr int RES_MAX_AXES = 1536;   // nodes of the three axes together (their factors sit in shared memory)

__host__ __device__ inline int res_pad(int n) { return (n + 3) & ~3; }

// The axes' factors in shared memory, 12 words per node: along i and j as ResNode records (a row's
// factors in two 16-byte loads), along k as 12 arrays (length padded to 4 with zeros; a group's four in
// one load): inv_d, inv_dd, raw_d, raw_dd, be, ce, bh, ch, then per group the first slot of a group that
// reaches the layer, or -1 (its nodes' slots follow one another, see res_k_slots). The CPML's b and c are
// zero outside the layer.
struct __align__(16) ResHalf {   // of the H or the E update
    float inv;
    int slot;
    float raw, b;
};
struct __align__(16) ResNode {
    ResHalf f[2];                // H, E
    float c[2];
    float pad[2];
};

// Numbers the layer's slots along k so that the nodes of a 4-node group (k a multiple of 4) that lie in
// the layer have consecutive slots from a multiple of 4 on: the low layer's slots are its nodes, the
// high layer's start past them at its first group. pw becomes the slots' row pitch. False, and nothing
// changed, where one group would hold nodes of both layers or the pitch would outgrow the march's
// staged boxes.
inline bool res_k_slots(std::vector<AxisNode>& ax, size_t pml, int& pw) {
    const int n = int(ax.size()), p = int(pml);
    if (p == 0 || n <= 2 * p + 2) return true;   // no layer: no slots
    const int low = res_pad(p), high = (n - 1 - p) & ~3, w = low + res_pad(n) - high;
    if (high < low || (w > 32 && pw <= 32)) return false;
    for (int k = 0; k < n; ++k)
        for (int* s : {&ax[size_t(k)].slot_e, &ax[size_t(k)].slot_h})
            if (*s >= 0) *s = k < p ? k : low + (k - high);
    pw = w;
    return true;
}
inline size_t res_smem(const Geom& g) { return size_t(res_pad(g.n0) + res_pad(g.n1) + res_pad(g.n2)) * 12 * 4; }

__device__ __forceinline__ void res_fill_rows(ResNode* t, int n, const AxisNode* ax) {
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
        const AxisNode v = ax[q];
        ResNode r;
        r.f[0] = ResHalf{v.inv_d, v.slot_h, v.raw_inv_d, v.bh};
        r.f[1] = ResHalf{v.inv_dd, v.slot_e, v.raw_inv_dd, v.be};
        r.c[0] = v.ch;
        r.c[1] = v.ce;
        r.pad[0] = r.pad[1] = 0.f;
        t[q] = r;
    }
}

// E's factors at node 0 are cleared: no edge there updates along k, and its psi stays 0.
__device__ __forceinline__ void res_fill_k(float* z, int n, const AxisNode* ax) {
    const int np = res_pad(n);
    int* slot = reinterpret_cast<int*>(z + 8 * np);
    for (int q = threadIdx.x; q < np; q += blockDim.x) {
        AxisNode v{0, 0, 0, 0, 0, 0, 0, 0, -1, -1};
        if (q < n) v = ax[q];
        const bool le = v.slot_e >= 0 && q > 0, lh = v.slot_h >= 0;
        const float f[8] = {v.inv_d, v.inv_dd, v.raw_inv_d, v.raw_inv_dd, le ? v.be : 0.f, le ? v.ce : 0.f,
                            lh ? v.bh : 0.f, lh ? v.ch : 0.f};
#pragma unroll
        for (int t = 0; t < 8; ++t) z[t * np + q] = f[t];
        if (q < np / 4) {
            int first = -1;   // any live node's slot less its place in the group
            for (int t = 0; t < 4 && 4 * q + t < n; ++t) {
                const int e = ax[4 * q + t].slot_e, h = ax[4 * q + t].slot_h;
                if (e >= 0) first = e - t;
                else if (h >= 0) first = h - t;
            }
            slot[q] = first;
        }
    }
}

// Every block of the launch arrives and waits for all: of a launch that is one cluster by the cluster's
// hardware barrier, else through a counter in global memory; false when the wait ran out (the error word
// is set, and every block leaves at this barrier or the next). The block's writes before it are
// visible to all after it.
template <bool CLUSTER>
__device__ __forceinline__ bool res_barrier(const ResArgs& a, unsigned target) {
    if constexpr (CLUSTER) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
    __syncthreads();
    int bad = 0;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        unsigned v;
        unsigned long long t0 = 0;
        for (unsigned spin = 0;; ++spin) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
            if (v >= target) break;
            if ((spin & 255u) == 255u) {
                unsigned long long t;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                if (t0 == 0) t0 = t;
                else if (t - t0 > a.wait_ns) {
                    *static_cast<volatile int*>(a.error) = 3;
                    bad = 1;
                    break;
                }
            }
        }
    }
    return !__syncthreads_or(bad);
}

// Four nodes along k as two packed pairs (f2's operations round each lane as the scalar ones do).
struct Quad {
    float2 a, b;
};
__device__ __forceinline__ Quad ld4(const float* p) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    return Quad{make_float2(f.x, f.y), make_float2(f.z, f.w)};
}
__device__ __forceinline__ void st4(float* p, const Quad& q) {
    *reinterpret_cast<float4*>(p) = make_float4(q.a.x, q.a.y, q.b.x, q.b.y);
}
__device__ __forceinline__ Quad q_zero() { return Quad{make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
__device__ __forceinline__ Quad q_bc(float v) { return Quad{make_float2(v, v), make_float2(v, v)}; }
__device__ __forceinline__ Quad operator+(const Quad& x, const Quad& y) { return Quad{f2::add(x.a, y.a), f2::add(x.b, y.b)}; }
__device__ __forceinline__ Quad operator-(const Quad& x, const Quad& y) { return Quad{f2::sub(x.a, y.a), f2::sub(x.b, y.b)}; }
__device__ __forceinline__ Quad q_mul(const Quad& x, const Quad& y, float2 z) { return Quad{f2::mul(x.a, y.a, z), f2::mul(x.b, y.b, z)}; }
// the values one node up (the fourth from `next`) or one node down (the first from `prev`)
__device__ __forceinline__ Quad q_up(const Quad& x, float next) { return Quad{make_float2(x.a.y, x.b.x), make_float2(x.b.y, next)}; }
__device__ __forceinline__ Quad q_down(const Quad& x, float prev) { return Quad{make_float2(prev, x.a.x), make_float2(x.a.y, x.b.x)}; }
// one CPML term, psi' = b psi + (c d) raw (cpu.rs:73-99): psi becomes psi', t gains it
__device__ __forceinline__ void q_psi(Quad& t, Quad& psi, const Quad& d, const Quad& b, const Quad& c, const Quad& raw, float2 z) {
    psi = q_mul(b, psi, z) + q_mul(q_mul(c, d, z), raw, z);
    t = t + psi;
}

// The class ids of 4 nodes, as loaded and one by one.
template <typename CID>
using IdWords = std::conditional_t<sizeof(CID) == 1, unsigned, std::conditional_t<sizeof(CID) == 2, uint2, uint4>>;
template <typename CID>
__device__ __forceinline__ IdWords<CID> res_load_ids(const CID* p) { return __ldg(reinterpret_cast<const IdWords<CID>*>(p)); }
__device__ __forceinline__ uint4 res_each(unsigned v) { return make_uint4(v & 255u, v >> 8 & 255u, v >> 16 & 255u, v >> 24); }
__device__ __forceinline__ uint4 res_each(uint2 v) { return make_uint4(v.x & 65535u, v.x >> 16, v.y & 65535u, v.y >> 16); }
__device__ __forceinline__ uint4 res_each(uint4 v) { return v; }
template <typename CID>
__device__ __forceinline__ uint4 res_ids(const CID* p) { return res_each(res_load_ids(p)); }

// One component C of the field (F = 1: E from H, F = 0: H from E) on the 4 nodes from (i, j, k)
// (cpu.rs:48-167): its two curl terms R - S, R the difference along i or j that its row decides (x: j,
// y and z: i), S the other (along k for the x and y components, along j for z), with the sign of the y
// component's pair turned (R - S = -(S - R) exactly).
//
// A node whose update does not run keeps its value by a select; its psi is advanced all the same where
// the layer covers it: such a psi is read by no update (its edge never runs), and it stays 0 where the
// reference's does by the cleared factors. Every field load comes before the first store.
template <int C, int F, typename CID, bool DEBYE>
__device__ __forceinline__ void res_update(const ResArgs& a, const ResNode* X, const ResNode* Y, const float* Z, int np2, unsigned row,
                                           int i, int j, int k, IdWords<CID> words, int dg, const float* src, const float* own,
                                           float* out, const float* psi_in, float* psi_out) {
    const Geom& g = a.g;
    const unsigned id = row * unsigned(g.p2) + unsigned(k), cs = unsigned(g.cs);
    const float2 z = make_float2(a.neg0, a.neg0);
    constexpr bool ALONG_I = C != 0, S_J = C == 2;    // R's axis; S along j (else along k)
    const unsigned sj = unsigned(g.p2), si = unsigned(g.n1) * sj, sr = ALONG_I ? si : sj;
    const bool has_i = F ? i > 0 : i + 1 < g.n0, has_j = F ? j > 0 : j + 1 < g.n1;
    const unsigned ido = unsigned(C) * cs + id;
    const Quad f = ld4(own + ido);
    if (!(ALONG_I ? has_i : has_j) || (S_J && !has_j)) {   // no neighbour along R or S: nothing to update
        if (out != own) st4(out + ido, f);
        return;
    }
    const unsigned idr = (C == 2 ? cs : 2 * cs) + id, ids = (C == 0 ? cs : 0u) + id;
    const Quad r0 = ld4(src + idr), r1 = ld4(src + (F ? idr - sr : idr + sr));
    const Quad s0 = ld4(src + ids);
    const int nk = g.n2 - k;
    Quad s1;
    if constexpr (S_J) s1 = ld4(src + (F ? ids - sj : ids + sj));
    else if constexpr (F) s1 = q_down(s0, k > 0 ? src[ids - 1] : 0.f);
    else s1 = q_up(s0, nk > 4 ? src[ids + 4] : 0.f);
    // the psi of both differences with the fields: nearly every warp has lanes in the layer along k, and
    // a load behind the differences would cost it another round of latency
    const ResNode* tr = ALONG_I ? X + i : Y + j;
    const ResHalf fr = tr->f[F];
    const int sls = S_J ? Y[j].f[F].slot : reinterpret_cast<const int*>(Z + 8 * np2)[k >> 2];
    const unsigned orr = unsigned(g.psi_off[(F ? 0 : 9) + C * 3 + (ALONG_I ? 0 : 1)]) + unsigned(k) +
                         (ALONG_I ? unsigned(fr.slot) * unsigned(g.n1) + unsigned(j)
                                  : unsigned(i) * unsigned(2 * g.pml) + unsigned(fr.slot)) * unsigned(g.pk);
    const unsigned os = S_J ? unsigned(g.psi_off[(F ? 0 : 9) + C * 3 + 1]) + unsigned(k) +
                                  (unsigned(i) * unsigned(2 * g.pml) + unsigned(sls)) * unsigned(g.pk)
                            : unsigned(g.psi_off[(F ? 0 : 9) + C * 3 + 2]) + row * unsigned(g.pw) + unsigned(sls);
    Quad pr = q_zero(), ps = q_zero();
    if (fr.slot >= 0) pr = ld4(psi_in + orr);
    if (sls >= 0) ps = ld4(psi_in + os);
    float2 ca0, ca1, cb0, cb1;
    if constexpr (F) {
        const uint4 cid = res_each(words);
        const float* t = reinterpret_cast<const float*>(a.classes) + C;
        const float fa = __ldg(t + cid.x * 8), fb = __ldg(t + cid.x * 8 + 4);   // most groups hold one class
        ca0 = ca1 = make_float2(fa, fa);
        cb0 = cb1 = make_float2(fb, fb);
        if (cid.y != cid.x || cid.z != cid.x || cid.w != cid.x) {
            ca0.y = __ldg(t + cid.y * 8); cb0.y = __ldg(t + cid.y * 8 + 4);
            ca1 = make_float2(__ldg(t + cid.z * 8), __ldg(t + cid.w * 8));
            cb1 = make_float2(__ldg(t + cid.z * 8 + 4), __ldg(t + cid.w * 8 + 4));
        }
    }
    const Quad dr = F ? r0 - r1 : r1 - r0, ds = F ? s0 - s1 : s1 - s0;
    Quad R = q_mul(dr, q_bc(fr.inv), z), S;
    if (fr.slot >= 0) {
        q_psi(R, pr, dr, q_bc(fr.b), q_bc(tr->c[F]), q_bc(fr.raw), z);
        st4(psi_out + orr, pr);
    }
    if constexpr (S_J) {
        const ResHalf fs = Y[j].f[F];
        S = q_mul(ds, q_bc(fs.inv), z);
        if (sls >= 0) q_psi(S, ps, ds, q_bc(fs.b), q_bc(Y[j].c[F]), q_bc(fs.raw), z);
    } else {
        S = q_mul(ds, ld4(Z + (F ? 1 : 0) * np2 + k), z);
        if (sls >= 0) {
            // the group's nodes outside the layer (b = 0) keep psi = 0 past f32's range too, where c d is NaN
            const Quad b = ld4(Z + (F ? 4 : 6) * np2 + k);
            const float2 o = make_float2(0.f, 0.f);
            const Quad d{f2::pick(b.a.x != 0.f, b.a.y != 0.f, ds.a, o), f2::pick(b.b.x != 0.f, b.b.y != 0.f, ds.b, o)};
            q_psi(S, ps, d, b, ld4(Z + (F ? 5 : 7) * np2 + k), ld4(Z + (F ? 3 : 2) * np2 + k), z);
        }
    }
    if (sls >= 0) st4(psi_out + os, ps);
    const Quad t = C == 1 ? S - R : R - S;
    Quad n;
    if constexpr (F) {
        n = q_mul(Quad{ca0, ca1}, f, z) + q_mul(Quad{cb0, cb1}, t, z);
        n.a = f2::pick(cb0.x != 0.f && (S_J || k > 0), cb0.y != 0.f, n.a, f.a);
        n.b = f2::pick(cb1.x != 0.f, cb1.y != 0.f, n.b, f.b);
        if (DEBYE && dg >= 0) {   // k_debye_post_cb's arithmetic on the group
            const unsigned o = unsigned(dg) * 12u + 4u * C;
            const int poles = int(__ldg(a.debye_table));
            Quad s0 = q_zero();
            for (int m = 0; m < poles; ++m)
                s0 = s0 + q_mul(q_bc(0.5f * (1.0f + __ldg(a.debye_table + 1 + 2 * m))), ld4(a.rd_state + (m * a.rd_pole + o)), z);
            n = n - q_mul(Quad{cb0, cb1}, s0, z);
            const Quad de = n - f, w = ld4(a.rd_dd + o);
            for (int m = 0; m < poles; ++m) {
                float* p = a.rd_state + (m * a.rd_pole + o);
                const Quad b = q_bc(__ldg(a.debye_table + 1 + 2 * m)), c = q_bc(__ldg(a.debye_table + 2 + 2 * m));
                st4(p, q_mul(b, ld4(p), z) + q_mul(q_mul(w, c, z), de, z));
            }
        }
    } else {
        n = f - q_mul(q_bc(a.k_mu), t, z);
        if (!S_J) {   // the row's last node has no k + 1 neighbour (the padding past it is 0 and stays 0)
            n.a = f2::pick(nk > 1, nk > 2, n.a, f.a);
            n.b = f2::pick(nk > 3, nk > 4, n.b, f.b);
        }
    }
    st4(out + ido, n);
}

// A lane's way over the grid: the group `first`, then one a launch's pass further at a time, as rows and
// groups of a row; BACK: counted and walked from the grid's end.
template <bool BACK>
struct ResWalk {
    int row, col, i, j;
    __device__ __forceinline__ ResWalk(const ResArgs& a, unsigned first) {
        const unsigned r = a.quads(first), p = a.rows(r);
        row = int(r);
        col = int(first - r * a.quads.d);
        i = int(p);
        j = int(r - p * a.rows.d);
        if (BACK) {
            row = int(a.last_row) - row;
            col = int(a.quads.d) - 1 - col;
            i = a.g.n0 - 1 - i;
            j = a.g.n1 - 1 - j;
        }
    }
    __device__ __forceinline__ bool inside(const ResArgs& a) const { return BACK ? i >= 0 : i < a.g.n0; }
    __device__ __forceinline__ void next(const ResArgs& a) {
        const int Q = int(a.quads.d), R = int(a.rows.d);
        if (BACK) {
            col -= int(a.dq);
            row -= int(a.drow);
            j -= int(a.dj);
            i -= int(a.di);
            if (col < 0) { col += Q; --row; --j; }
            if (j < 0) { j += R; --i; }
        } else {
            col += int(a.dq);
            row += int(a.drow);
            j += int(a.dj);
            i += int(a.di);
            if (col >= Q) { col -= Q; ++row; ++j; }
            if (j >= R) { j -= R; ++i; }
        }
    }
};

// A warp's share of a half step: component C of the groups from `first` on. The E half (F = 1) walks the
// grid backwards: it starts on the planes the H half has just left in the L2, and the next H half on
// those it leaves (of a grid whose state is more than the L2 keeps, a walk in one direction finds every
// plane evicted: the adjoint sweep at 161x161x97 moved 218 MB a step through HBM; 93 -> 76 us a step).
template <int C, int F, typename CID, bool DEBYE>
__device__ __forceinline__ void res_half(const ResArgs& a, const ResNode* X, const ResNode* Y, const float* Z, int np2, unsigned first,
                                         const float* src, const float* own, float* out, const float* psi_in, float* psi_out) {
    ResWalk<F != 0> at(a, first);
    // the E half's class ids a group ahead: its coefficients' addresses stand when its other loads start
    const CID* cls = static_cast<const CID*>(a.node_class);
    auto ids = [&](const ResWalk<F != 0>& w) { return res_load_ids(cls + (unsigned(w.row) * unsigned(a.g.p2) + unsigned(w.col) * 4u)); };
    auto place = [&](const ResWalk<F != 0>& w) { return __ldg(a.rd_index + (w.row * int(a.quads.d) + w.col)); };
    IdWords<CID> words{};
    int dg = -1;
    if (F && at.inside(a)) {
        words = ids(at);
        if (DEBYE) dg = place(at);
    }
    while (at.inside(a)) {
        ResWalk<F != 0> nx = at;
        nx.next(a);
        IdWords<CID> ahead{};
        int dn = -1;
        if (F && nx.inside(a)) {
            ahead = ids(nx);
            if (DEBYE) dn = place(nx);
        }
        res_update<C, F, CID, DEBYE>(a, X, Y, Z, np2, unsigned(at.row), at.i, at.j, at.col * 4, words, dg, src, own, out, psi_in, psi_out);
        at = nx;
        words = ahead;
        dg = dn;
    }
}

template <int F, typename CID, bool DEBYE>
__device__ __forceinline__ void res_field(const ResArgs& a, int comp, const ResNode* X, const ResNode* Y, const float* Z, int np2,
                                          unsigned first, const float* src, const float* own, float* out, const float* psi_in,
                                          float* psi_out) {
    if (comp == 0) res_half<0, F, CID, DEBYE>(a, X, Y, Z, np2, first, src, own, out, psi_in, psi_out);
    else if (comp == 1) res_half<1, F, CID, DEBYE>(a, X, Y, Z, np2, first, src, own, out, psi_in, psi_out);
    else res_half<2, F, CID, DEBYE>(a, X, Y, Z, np2, first, src, own, out, psi_in, psi_out);
}

// A port's voltage (F = 0, E settled after step n) or current (F = 1, H of step n) into its series
// entry: one warp, the f64 sums of probe_block (the same order for up to 32 edges).
template <int F>
__device__ __forceinline__ void res_probe(const ResArgs& a, int port, unsigned n) {
    const DevProbe d = a.probes[port];
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    if (F == 0) {
        for (int q = lane; q < d.count; q += 32) {
            const DevPortEdge x = a.pe[d.first + q];
            s -= double(a.e[(long long)d.comp * a.g.cs + x.id] * x.w);
        }
    } else {
        for (int q = lane; q < d.loop_count; q += 32) {
            const DevLoop x = a.lp[d.loop_first + q];
            s += double(a.h[x.f] * x.w);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0 && n < a.sc.cap) a.series[((long long)n * a.sc.ports + port) * 2 + F] = float(s);
}

// The step's plane-DFT phase factors of frequency k: E's (re, im), H's (re, im), times dt (cpu.rs:344-353).
__device__ __forceinline__ float4 res_phase(const StepConst& sc, unsigned n, int k) {
    if (n < sc.cap) return __ldg(reinterpret_cast<const float4*>(sc.dft) + ((long long)n * sc.nf + k));
    const float w = sc.omega[k], te = (float(n) + 1.0f) * sc.dt, th = (float(n) + 0.5f) * sc.dt;
    return make_float4(cosf(w * te) * sc.dt, -sinf(w * te) * sc.dt, cosf(w * th) * sc.dt, -sinf(w * th) * sc.dt);
}

// k_field_dft's sums over E (F = 0) or H (F = 1) of step n.
template <int F>
__device__ __forceinline__ void res_plane(const ResArgs& a, unsigned n, unsigned t, unsigned nt) {
    const Geom& g = a.g;
    const unsigned pts = unsigned(g.n0) * unsigned(g.n1);
    constexpr int NC = F ? 2 : 3, C0 = F ? 3 : 0;
    const float* src = F ? a.h : a.e;
    for (unsigned q = t; q < pts; q += nt) {
        const long long id = (long long)q * g.p2 + a.plane_k;
        float f[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) f[c] = src[c * g.cs + id];
        for (int k = 0; k < a.sc.nf; ++k) {
            const float4 ph = res_phase(a.sc, n, k);
            const float p0 = F ? ph.z : ph.x, p1 = F ? ph.w : ph.y;
            float* out = a.plane + ((long long)k * 10 + 2 * C0) * pts + q;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                out[(2 * c) * (long long)pts] += f[c] * p0;
                out[(2 * c + 1) * (long long)pts] += f[c] * p1;
            }
        }
    }
}

// k_ntff's sums: M from E (F = 0) or J from H (F = 1) of step n.
template <int F, int A>
__device__ __forceinline__ void res_ntff_patch(const ResArgs& a, unsigned n, unsigned p, float side) {
    const int P = a.n_patches;
    auto word = [&](int m) { return __ldg(a.patch + (long long)m * P + p); };
    NtffM x;
    if constexpr (F) x = ntff_j<A>(word, a.g.cs, a.h, side);
    else x = ntff_m<A>(word, a.g.cs, a.e, side);
    for (int k = 0; k < a.sc.nf; ++k) {
        const float4 ph = ntff_phase(a.sc, n, k);
        ntff_add<A>(a.ntff + ((long long)k * 12 + (F ? 0 : 6)) * P + p, P, x, F ? ph.z : ph.x, F ? ph.w : ph.y);
    }
}
template <int F>
__device__ __forceinline__ void res_ntff(const ResArgs& a, unsigned n, unsigned t, unsigned nt) {
    for (unsigned p = t; p < unsigned(a.n_patches); p += nt) {
        const unsigned meta = __ldg(a.patch + p);
        const float side = (meta & 4) ? 1.0f : -1.0f;
        if ((meta & 3) == 0) res_ntff_patch<F, 0>(a, n, p, side);
        else if ((meta & 3) == 1) res_ntff_patch<F, 1>(a, n, p, side);
        else res_ntff_patch<F, 2>(a, n, p, side);
    }
}

// The block that updates E at the node of field index f.
__device__ __forceinline__ unsigned res_block_of(const ResArgs& a, long long f, unsigned blocks, unsigned groups) {
    const long long id = f % a.g.cs;
    const unsigned q = (a.last_row - unsigned(id / a.g.p2)) * a.quads.d + (a.quads.d - 1u - unsigned(id % a.g.p2) / 4u);
    return (q / groups) % blocks;   // counted as the E half walks
}

// At most one block per SM, every block resident: a cooperative launch. The blocks take the grid's
// 4-node groups, in row order, a third of its threads' number at a time in turn, three warps (one per
// component) to 32 groups: a block's groups are whole rows (its j neighbours and the three components' shared loads are
// mostly in its L1), and the layer's heavier groups fall on all blocks alike.
template <typename CID, bool CLUSTER, bool DEBYE>
__global__ void __launch_bounds__(RES_THREADS, 1) k_resident(const __grid_constant__ ResArgs a) {
    extern __shared__ __align__(16) float res_sm[];
    const Geom& g = a.g;
    const int np2 = res_pad(g.n2);
    ResNode *X = reinterpret_cast<ResNode*>(res_sm), *Y = X + res_pad(g.n0);
    float* Z = reinterpret_cast<float*>(Y + res_pad(g.n1));
    res_fill_rows(X, g.n0, g.ax[0]);
    res_fill_rows(Y, g.n1, g.ax[1]);
    res_fill_k(Z, g.n2, g.ax[2]);
    const int w = threadIdx.x >> 5, comp = w % 3;                                      // the warp's component
    const unsigned groups = blockDim.x / 3u;
    const unsigned first = blockIdx.x * groups + unsigned(w / 3) * 32u + (threadIdx.x & 31u);   // the lane's first group
    const unsigned G = gridDim.x, b = blockIdx.x;
    // the lists are shared out 32 entries at a time, one warp of every block before a block's next (formed
    // where used, as the history's place is: the walks between need every register)
    auto t = [] { return ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32u + (threadIdx.x & 31u); };
    auto nt = [] { return gridDim.x * blockDim.x; };
    auto place = [&](unsigned n) -> long long {   // step n's place in the design history, or -1
        const long long v = (long long)n - *a.hist_base;
        return v >= a.hist_cap ? -1 : v;
    };
    const unsigned n0 = *(volatile const unsigned*)a.counter;
    int own = 0;   // a source or inductor edge among the block's nodes
    for (int q = threadIdx.x; q < a.ns; q += blockDim.x) own |= res_block_of(a, a.src[q].f, G, groups) == b;
    for (int q = threadIdx.x; q < a.ni; q += blockDim.x) own |= res_block_of(a, a.ind[q].f, G, groups) == b;
    own = __syncthreads_or(own);
    unsigned target = a.late;
    for (int s = 0; s <= a.steps; ++s) {
        const unsigned n = n0 + unsigned(s);
        // ---- phase A: what reads E^n (E after step n - 1) ...
        if (s > 0) {
            if (threadIdx.x < 32)
                for (int p = int(G - 1 - b); p < a.n_ports; p += int(G)) res_probe<0>(a, p, n - 1);
            if (a.plane) res_plane<0>(a, n - 1, t(), nt());
            if (a.ntff) res_ntff<0>(a, n - 1, t(), nt());
        }
        if (s == a.steps) break;
        const float* e_in = s ? a.e : a.e_src;
        if (a.n_design) {
            const long long slot = place(n);
            if (slot >= 0)
                for (int q = int(t()); q < a.n_design; q += int(nt())) {
                    const int4 d = a.design[q];
                    a.hist_e[slot * a.n_design + q] = e_in[d.x * g.cs + ((long long)d.y * g.n1 + d.z) * g.p2 + d.w];
                }
        }
        // ... and the new H
        const float *h_in = s ? a.h : a.h_src, *p_in = s ? a.psi_h : a.psi_h_src;
        res_field<0, CID, false>(a, comp, X, Y, Z, np2, first, e_in, h_in, a.h, p_in, a.psi_h);
        if (!res_barrier<CLUSTER>(a, target += G)) return;
        // ---- phase B: what reads the new H, and the new E
        if (threadIdx.x < 32)
            for (int p = int(G - 1 - b); p < a.n_ports; p += int(G)) res_probe<1>(a, p, n);
        if (a.plane) res_plane<1>(a, n, t(), nt());
        if (a.ntff) res_ntff<1>(a, n, t(), nt());
        res_field<1, CID, DEBYE>(a, comp, X, Y, Z, np2, first, a.h, e_in, a.e, a.psi_e, a.psi_e);
        if (own) {   // the source, then the inductors (lumped_block), on the block's own edges
            __syncthreads();
            const float p = n < a.sc.cap ? a.sc.pulse[n] : pulse_at(a.sc, (float(n) + 0.5f) * a.sc.dt);
            for (int q = threadIdx.x; q < a.ns; q += blockDim.x) {
                const DevSource x = a.src[q];
                if (res_block_of(a, x.f, G, groups) == b) a.e[x.f] -= x.src * p;
            }
            __syncthreads();
            for (int q = threadIdx.x; q < a.ni; q += blockDim.x) {
                const DevInductor d = a.ind[q];
                if (res_block_of(a, d.f, G, groups) == b) {
                    const float x = a.e[d.f] - d.ke * d.cur;
                    a.e[d.f] = x;
                    a.ind[q].cur = d.cur + d.ki * x;
                }
            }
        }
        if (!res_barrier<CLUSTER>(a, target += G)) return;
        if (a.n_design) {
            // ---- phase C: the design edges' curl terms (k_design_record)
            const long long slot = place(n);
            if (slot >= 0)
                for (int q = int(t()); q < a.n_design; q += int(nt()))
                    a.hist_s[slot * a.n_design + q] = design_curl(g, a.design[q], a.h, a.psi_e);
            if (!res_barrier<CLUSTER>(a, target += G)) return;
        }
    }
    if (t() == 0) *a.counter = n0 + unsigned(a.steps);
}

// ---- the Debye layout by groups, from the edge list

struct RdMap {
    Geom g;
    unsigned quads;          // groups per row
    const long long* f;      // the list
    int count;
    int* index;
};
__device__ __forceinline__ unsigned rd_group(const RdMap& m, int q, unsigned& at) {
    const long long f = m.f[q];
    const int c = int(f / m.g.cs);
    const long long id = f - c * m.g.cs, row = id / m.g.p2;
    const unsigned k = unsigned(id - row * m.g.p2);
    at = 4u * unsigned(c) + (k & 3u);
    return unsigned(row) * m.quads + k / 4u;
}
__global__ void k_rd_mark(RdMap m) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m.count; q += gridDim.x * blockDim.x) {
        unsigned at;
        m.index[rd_group(m, q, at)] = 1;
    }
}
// flags and their running sums to places
__global__ void k_rd_places(int* index, const int* sums, unsigned n) {
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) index[q] = index[q] ? sums[q] : -1;
}
__global__ void k_rd_weights(RdMap m, const float* __restrict__ dd, float* __restrict__ out) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m.count; q += gridDim.x * blockDim.x) {
        unsigned at;
        const unsigned g = rd_group(m, q, at);
        out[unsigned(m.index[g]) * 12u + at] = dd[q];
    }
}
// The pole states between the list and the groups (TO: to the groups).
template <bool TO>
__global__ void k_rd_move(RdMap m, int poles, unsigned pole, float* list, float* dense) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m.count; q += gridDim.x * blockDim.x) {
        unsigned at;
        const unsigned g = rd_group(m, q, at), o = unsigned(m.index[g]) * 12u + at;
        for (int k = 0; k < poles; ++k) {
            float &l = list[(long long)k * m.count + q], &d = dense[(size_t)k * pole + o];
            if (TO) d = l;
            else l = d;
        }
    }
}

}  // namespace fg
