// Mesh -> grid rasterisation on the device: the ray-parity fill of crates/sims-field/src/raster.rs
// (fill :24-104, solid_edges :145-160, solid_cells :162-173, sheet_edges :186-264) and the closed-mesh
// check (:127-143) on the host.
//
// A fill casts one ray per sample column of each axis and pairs its crossings. All rays of an axis are
// parallel and lie on a grid, so the triangles look for their columns instead of the rays for their
// triangles (the reference's hierarchy, bvh.rs): a warp takes a triangle, tests the few columns under its
// bounding box with the reference's own hit test, and counts, then stores, each crossing in its column's
// list; a thread per column sorts its list and walks it as repeated nearest-crossing queries would. Work
// goes with the crossings, no hierarchy is built on the host (it was half of a fill; only a mesh whose
// hits it could prune needs its boxes, see Boxes), and no thread
// chases a tree through memory once per crossing: 12,288 triangles onto 160x128x96 cells take 6.9 ms a
// fill with its copies, 15.4 before.
// sheet_edges runs one block per triangle over the nodes near it. Every mark is a byte store of 1, so
// the order in which threads mark does not change the masks. The arithmetic is the reference's f64
// arithmetic in its operation order (the build has no a*b+c contraction).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/fieldgrid.h"
#include "engine.hpp"

#include <cub/cub.cuh>

namespace fg {
namespace raster {

constexpr int MAX_CROSSINGS = 1 << 20;     // per column

// The boxes that Bvh::build (bvh.rs:62-93: median splits along the longest axis, leaves of at most 4
// triangles) gives each triangle's leaf. The hit test takes a ray up to a 1e-9 part of the triangle outside
// of it, and the rays pass a 1e-6 part of a cell from the grid's lines: past the edge of a face more than
// some 1200 cells wide a ray can hit, and whether it counts is for the leaf's box to say (a triangle's own
// box never tells more than its leaf's, which holds it).
struct Boxes {
    const double* tri;
    std::vector<int> order;
    std::vector<double> out;   // per triangle: low, high

    Boxes(const double* t, size_t n) : tri(t), order(n), out(n * 6) {
        for (size_t q = 0; q < n; ++q) order[q] = int(q);
        split(0, int(n));
    }
    double centre(int i, int axis) const {
        const double* t = tri + size_t(i) * 9;
        return (t[axis] + t[3 + axis] + t[6 + axis]) / 3.0;
    }
    void split(int start, int end) {
        double b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
        for (int q = start; q < end; ++q)
            for (int c = 0; c < 9; ++c) {
                const double v = tri[size_t(order[size_t(q)]) * 9 + size_t(c)];
                b[c % 3] = std::fmin(b[c % 3], v);
                b[3 + c % 3] = std::fmax(b[3 + c % 3], v);
            }
        if (end - start <= 4) {
            for (int q = start; q < end; ++q) std::copy(b, b + 6, &out[size_t(order[size_t(q)]) * 6]);
            return;
        }
        const double ex[3] = {b[3] - b[0], b[4] - b[1], b[5] - b[2]};
        const int axis = (ex[0] >= ex[1] && ex[0] >= ex[2]) ? 0 : (ex[1] >= ex[2] ? 1 : 2);
        const int middle = (start + end) / 2;
        std::nth_element(order.begin() + start, order.begin() + middle, order.begin() + end,
                         [&](int x, int y) { return centre(x, axis) < centre(y, axis); });
        split(start, middle);
        split(middle, end);
    }
};

__device__ __forceinline__ void dsub(const double* a, const double* b, double* o) {
    o[0] = a[0] - b[0]; o[1] = a[1] - b[1]; o[2] = a[2] - b[2];
}
__device__ __forceinline__ double ddot(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
__device__ __forceinline__ void dcross(const double* a, const double* b, double* o) {
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

// hit (bvh.rs:156-177): the ray parameter of a triangle crossing, or NaN for none.
__device__ double hit(const double* t, const double* origin, const double* dir) {
    double e1[3], e2[3], p[3], s[3], q[3];
    dsub(t + 3, t, e1);
    dsub(t + 6, t, e2);
    dcross(dir, e2, p);
    const double det = ddot(e1, p);
    if (fabs(det) < 1.0e-18) return NAN;
    const double inv = 1.0 / det;
    dsub(origin, t, s);
    const double u = ddot(s, p) * inv;
    if (!(u >= -1.0e-9 && u <= 1.0 + 1.0e-9)) return NAN;
    dcross(s, e1, q);
    const double v = ddot(dir, q) * inv;
    if (v < -1.0e-9 || u + v > 1.0 + 1.0e-9) return NAN;
    return ddot(e2, q) * inv;
}

// slice::partition_point over a sorted line: the first index whose sample fails `below`.
__device__ __forceinline__ int count_below(const double* line, int n, double v, bool or_equal) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const bool in = or_equal ? line[mid] <= v : line[mid] < v;
        if (in) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// grid::nearest (grid.rs:48-55)
__device__ int nearest(const double* line, int n, double v) {
    const int i = count_below(line, n, v, false);
    if (i >= 1 && i < n) {
        if (fabs(v - line[i - 1]) <= fabs(line[i] - v)) return i - 1;
    } else if (i >= 1) {
        return i - 1;
    }
    return min(i, max(n - 1, 0));
}

struct FillAxis {
    const double* line[3];     // the sample lines of the three axes
    int n[3];
    int axis, u, v;
    int us, wide, vs, tall;    // the columns' sample spans along u and v
    double step[3];
    double start;
    double reach0, reach1;
    int order;                 // 0: (i m1 + j) m2 + k, 1: i + (j + k m1) m0
    long long m[3];            // the dimensions of the index space
};

__device__ __forceinline__ size_t index_of(const FillAxis& f, const int* c) {
    if (f.order == 0) return (size_t(c[0]) * f.m[1] + c[1]) * f.m[2] + c[2];
    return size_t(c[0]) + (size_t(c[1]) + size_t(c[2]) * f.m[1]) * f.m[0];
}

// The ray of column `col` (raster.rs:52-66): the samples' lines shifted by a small part of a cell, so that
// no ray meets an edge or a face of a mesh drawn on the grid.
__device__ __forceinline__ void column_ray(const FillAxis& f, long long col, int* cell, double* from) {
    cell[f.axis] = 0;
    cell[f.u] = f.us + int(col % f.wide);
    cell[f.v] = f.vs + int(col / f.wide);
    from[f.u] = f.line[f.u][cell[f.u]] + f.step[f.u] * 1.234567e-6;
    from[f.v] = f.line[f.v][cell[f.v]] + f.step[f.v] * 2.345678e-6;
    from[f.axis] = f.start;
}

// The samples [a, b) of a line that may lie under [lo, hi] once shifted, within a margin far above the hit
// test's own (1e-9 of the triangle).
__device__ __forceinline__ void span_under(const double* line, int n, double shift, double step, double lo, double hi, int& a,
                                           int& b) {
    const double m = 1e-6 * step + 1e-8 * (hi - lo);
    a = count_below(line, n, lo - m - shift, false);
    b = count_below(line, n, hi + m - shift, true);
}

// The crossings of one axis's columns: a warp per triangle (and part of its columns, blockIdx.y). STORE
// false: counted per column; true: stored in the columns [c0, c1)' lists, at offset[col] - base on. A hit
// beside its triangle's box counts if the ray passes through its leaf's (`leaf`; null: *stray says there is one).
template <bool STORE>
__global__ void k_crossings(FillAxis f, const double* tri, long long ntri, unsigned long long* count,
                            const unsigned long long* offset, double* hits, unsigned long long base, long long c0, long long c1,
                            const double* leaf, int* stray) {
    const long long ti = blockIdx.x * (long long)(blockDim.x / 32) + (threadIdx.x >> 5);
    if (ti >= ntri) return;
    const double* t = tri + ti * 9;
    int a[2], b[2];
    double lo[2], hi[2];
    for (int x = 0; x < 2; ++x) {
        const int ax = x ? f.v : f.u;
        lo[x] = fmin(fmin(t[ax], t[3 + ax]), t[6 + ax]);
        hi[x] = fmax(fmax(t[ax], t[3 + ax]), t[6 + ax]);
        span_under(f.line[ax], f.n[ax], f.step[ax] * (x ? 2.345678e-6 : 1.234567e-6), f.step[ax], lo[x], hi[x], a[x], b[x]);
    }
    a[0] = max(a[0] - f.us, 0);
    b[0] = min(b[0] - f.us, f.wide);
    a[1] = max(a[1] - f.vs, 0);
    b[1] = min(b[1] - f.vs, f.tall);
    if (a[0] >= b[0] || a[1] >= b[1]) return;
    const long long w = b[0] - a[0], total = w * (b[1] - a[1]);
    double dir[3] = {0.0, 0.0, 0.0};
    dir[f.axis] = 1.0;
    for (long long q = (long long)blockIdx.y * 32 + (threadIdx.x & 31); q < total; q += (long long)gridDim.y * 32) {
        const long long col = (a[1] + q / w) * f.wide + (a[0] + q % w);
        if (STORE && (col < c0 || col >= c1)) continue;
        int cell[3];
        double from[3];
        column_ray(f, col, cell, from);
        const double x = hit(t, from, dir);
        if (!(x > 0.0) || !(x < INFINITY)) continue;   // NaN: no crossing
        const double o0 = from[f.u], o1 = from[f.v];
        if (!(lo[0] < o0 && o0 < hi[0] && lo[1] < o1 && o1 < hi[1])) {
            if (leaf) {   // the slab test of bvh.rs:95-110 across the ray (a side the ray runs along is outside, a flat box in)
                const double* b6 = leaf + ti * 6;
                auto in = [&](int ax, double o) { return (b6[ax] < o && o < b6[3 + ax]) || (b6[ax] == o && o == b6[3 + ax]); };
                if (!in(f.u, o0) || !in(f.v, o1)) continue;
            } else {
                *stray = 1;
            }
        }
        const unsigned long long at = atomicAdd(count + col, 1ull);
        if (STORE) hits[offset[col] - base + at] = x;
    }
}

// Ascending order of a column's list: by insertion, or a heap where it is long.
__device__ void sort_list(double* a, long long n) {
    if (n <= 32) {
        for (long long i = 1; i < n; ++i) {
            const double v = a[i];
            long long j = i;
            for (; j > 0 && a[j - 1] > v; --j) a[j] = a[j - 1];
            a[j] = v;
        }
        return;
    }
    auto sift = [&](long long r, long long e) {
        const double v = a[r];
        for (long long c; (c = 2 * r + 1) < e; r = c) {
            if (c + 1 < e && a[c + 1] > a[c]) ++c;
            if (!(a[c] > v)) break;
            a[r] = a[c];
        }
        a[r] = v;
    };
    for (long long r = n / 2; r-- > 0;) sift(r, n);
    for (long long e = n - 1; e > 0; --e) {
        const double v = a[0];
        a[0] = a[e];
        a[e] = v;
        sift(0, e);
    }
}

// fill's column loop (raster.rs:52-99), one thread per column of [c0, c1): the crossings in order, each at
// least a 1e-9 part of a step past the one before, in pairs.
__global__ void k_fill_axis(FillAxis f, const unsigned long long* count, const unsigned long long* offset, double* hits,
                            unsigned long long base, long long c0, long long c1, uint8_t* inside, uint8_t* thin, int* error) {
    const long long col = c0 + blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (col >= c1) return;
    const long long crossings = (long long)count[col];
    if (crossings == 0) return;
    double* list = hits + (offset[col] - base);
    sort_list(list, crossings);
    int cell[3];
    double from[3];
    column_ray(f, col, cell, from);
    const double* line = f.line[f.axis];
    const int n = f.n[f.axis];
    double last = 0.0, a = 0.0;
    bool open = false;      // a crossing waits for its pair
    auto pair = [&](double pa, double pb) {
        const int first = count_below(line, n, pa, false);
        const int last_n = count_below(line, n, pb, true);   // partition_point(s <= b); last = that - 1
        if (last_n >= 1 && first <= last_n - 1) {
            if (f.axis == 0)
                for (int k = first; k <= last_n - 1; ++k) {
                    int c[3] = {cell[0], cell[1], cell[2]};
                    c[f.axis] = k;
                    inside[index_of(f, c)] = 1;
                }
        } else if (isfinite(pb)) {
            const double middle = 0.5 * (pa + pb);
            if (middle >= f.reach0 && middle < f.reach1) {
                int c[3] = {cell[0], cell[1], cell[2]};
                c[f.axis] = nearest(line, n, middle);
                thin[index_of(f, c)] = 1;
            }
        }
    };
    int taken = 0;
    for (long long q = 0; q < crossings; ++q) {
        const double t = list[q];
        if (!(t > last + f.step[f.axis] * 1.0e-9)) continue;
        const double x = f.start + t;
        if (open) pair(a, x);
        else a = x;
        open = !open;
        last = t;
        if (++taken == MAX_CROSSINGS) { atomicExch(error, 2); return; }
    }
    if (open) pair(a, INFINITY);
}

// thin keeps the samples that are not inside (raster.rs:100-103).
__global__ void k_thin_only(const uint8_t* inside, uint8_t* thin, size_t n) {
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
        if (inside[q]) thin[q] = 0;
}

struct SheetArgs {
    const double* line[3];
    int n[3];
};

__device__ int cell_of(const double* line, int n, double v) {   // grid::cell_of (grid.rs:57-59)
    const int i = max(count_below(line, n, v, true) - 1, 0);
    return min(i, max(n - 2, 0));
}

__device__ double local_size(const double* line, int n, int i, bool centre) {   // raster.rs:175-184
    if (centre) return line[min(i + 1, n - 1)] - line[min(i, n - 2)];
    const double before = i > 0 ? line[i] - line[i - 1] : line[1] - line[0];
    const double after = i + 1 < n ? line[i + 1] - line[i] : line[n - 1] - line[n - 2];
    return 0.5 * (before + after);
}

// sheet_edges (raster.rs:186-264): one block per triangle, its threads over the nodes near it.
__global__ void k_sheet_edges(SheetArgs g, const double* tris, long long ntri, uint8_t* mask) {
    for (long long ti = blockIdx.x; ti < ntri; ti += gridDim.x) {
        const double* t = tris + ti * 9;
        double e0[3], e1[3], normal[3];
        dsub(t + 3, t, e0);
        dsub(t + 6, t, e1);
        dcross(e0, e1, normal);
        const double area2 = sqrt(ddot(normal, normal));
        if (area2 <= 1e-30) continue;
        const double nrm[3] = {normal[0] / area2, normal[1] / area2, normal[2] / area2};
        double lo[3], hi[3];
        const double inf = INFINITY;
        for (int a = 0; a < 3; ++a) {
            lo[a] = fmin(fmin(fmin(inf, t[a]), t[3 + a]), t[6 + a]);
            hi[a] = fmax(fmax(fmax(-inf, t[a]), t[3 + a]), t[6 + a]);
        }
        const double d00 = ddot(e0, e0), d01 = ddot(e0, e1), d11 = ddot(e1, e1);
        const double det = d00 * d11 - d01 * d01;
        const size_t nn = size_t(g.n[0]) * g.n[1] * g.n[2];
        for (int c = 0; c < 3; ++c) {
            if (fabs(nrm[c]) >= 0.75) continue;
            int first[3], count[3];
            for (int a = 0; a < 3; ++a) {
                const double* line = g.line[a];
                const int n = g.n[a];
                const int il = cell_of(line, n, lo[a]), ih = cell_of(line, n, hi[a]);
                const double reach = fmax(line[il + 1] - line[il], line[ih + 1] - line[ih]);
                const int f0 = count_below(line, n, lo[a] - reach, false);
                int l0 = count_below(line, n, hi[a] + reach, true);
                if (a == c) l0 = min(l0, n - 1);
                first[a] = f0;
                count[a] = max(l0 - f0, 0);
            }
            const long long total = (long long)count[0] * count[1] * count[2];
            for (long long q = threadIdx.x; q < total; q += blockDim.x) {
                const int p[3] = {first[0] + int(q / ((long long)count[1] * count[2])),
                                  first[1] + int((q / count[2]) % count[1]), first[2] + int(q % count[2])};
                if (p[c] + 1 >= g.n[c]) continue;
                double mid[3], h[3];
                for (int a = 0; a < 3; ++a) {
                    const double* l = g.line[a];
                    mid[a] = a == c ? 0.5 * (l[p[a]] + l[p[a] + 1]) : l[p[a]];
                    h[a] = local_size(l, g.n[a], p[a], a == c);
                }
                double sum = 0.0;
                for (int a = 0; a < 3; ++a) sum = sum + fabs(nrm[a]) * h[a];
                const double tol = 0.5 * sum;
                double r[3];
                dsub(mid, t, r);
                const double d = ddot(r, nrm);
                const double eps = 1e-9 * tol;
                if (d <= eps - tol || d > tol + eps) continue;
                const double nd[3] = {nrm[0] * d, nrm[1] * d, nrm[2] * d};
                double m1[3], qv[3];
                dsub(mid, nd, m1);
                dsub(m1, t, qv);
                const double q0 = ddot(qv, e0), q1 = ddot(qv, e1);
                const double v = (d11 * q0 - d01 * q1) / det;
                const double w = (d00 * q1 - d01 * q0) / det;
                const double slack = 1e-9;
                if (v >= -slack && w >= -slack && v + w <= 1.0 + slack)
                    mask[size_t(c) * nn + (size_t(p[0]) * g.n[1] + p[1]) * g.n[2] + p[2]] = 1;
            }
        }
    }
}

// spacing (raster.rs:13-15): the smallest positive gap of a line (INFINITY when none).
double spacing(const std::vector<double>& line) {
    double s = INFINITY;
    for (size_t i = 0; i + 1 < line.size(); ++i) {
        const double d = line[i + 1] - line[i];
        if (d > 0.0) s = std::fmin(s, d);
    }
    return s;
}

size_t partition(const std::vector<double>& line, double v, bool or_equal) {
    return size_t(std::partition_point(line.begin(), line.end(),
                                       [&](double x) { return or_equal ? x <= v : x < v; }) - line.begin());
}

}  // namespace raster

#define RS_CUDA(call)                                                                              \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            err = std::string(#call) + ": " + cudaGetErrorString(e_);                              \
            return FG_ERR_CUDA;                                                                    \
        }                                                                                          \
    } while (0)

static int fill_masks(Gpu* gpu, const double* tris, uint64_t ntri, const std::vector<double>* samples, const size_t* dims,
                int order, uint8_t* inside, uint8_t* thin, std::string& err) {
    using namespace raster;
    const size_t total = dims[0] * dims[1] * dims[2];
    auto nothing = [&] {
        std::memset(inside, 0, total);
        std::memset(thin, 0, total);
        return FG_OK;
    };
    if (ntri == 0 || total == 0) return nothing();
    if (ntri >= (uint64_t(1) << 31)) { err = "too many triangles"; return FG_ERR_INVALID; }
    RS_CUDA(cudaSetDevice(gpu->device));
    double low[3], high[3];   // the mesh's box
    for (int a = 0; a < 3; ++a) { low[a] = INFINITY; high[a] = -INFINITY; }
    for (uint64_t q = 0; q < ntri * 3; ++q)
        for (int a = 0; a < 3; ++a) {
            low[a] = std::fmin(low[a], tris[q * 3 + a]);
            high[a] = std::fmax(high[a], tris[q * 3 + a]);
        }
    double step[3];
    for (int a = 0; a < 3; ++a) {
        const double s = spacing(samples[a]);
        step[a] = std::isfinite(s) ? s : std::fmax(std::fmax(high[0] - low[0], high[1] - low[1]), 1.0);
    }
    int sp0[3], sp1[3];
    for (int a = 0; a < 3; ++a) {   // span (raster.rs:17-22)
        const std::vector<double>& line = samples[a];
        if (line.empty()) return nothing();
        const size_t last_sample = line.size() - 1;
        size_t first = partition(line, low[a], true);
        first = first >= 1 ? first - 1 : 0;
        first = first >= 2 ? first - 2 : 0;
        const size_t last = std::min(partition(line, high[a], false) + 2, last_sample);
        if (first > last) return nothing();
        sp0[a] = int(first);
        sp1[a] = int(last);
    }
    const size_t lens[3] = {samples[0].size(), samples[1].size(), samples[2].size()};
    FillAxis f[3];
    long long cols[3], col0[4] = {0, 0, 0, 0};   // the three axes' columns side by side
    for (int axis = 0; axis < 3; ++axis) {
        FillAxis& x = f[axis];
        x = FillAxis{};
        for (int a = 0; a < 3; ++a) { x.n[a] = int(lens[a]); x.step[a] = step[a]; x.m[a] = (long long)dims[a]; }
        x.axis = axis;
        x.u = (axis + 1) % 3;
        x.v = (axis + 2) % 3;
        x.us = sp0[x.u];
        x.wide = sp1[x.u] - sp0[x.u] + 1;
        x.vs = sp0[x.v];
        x.tall = sp1[x.v] - sp0[x.v] + 1;
        const std::vector<double>& line = samples[axis];
        x.start = std::fmin(line[0], low[axis]) - 2.0 * step[axis];
        x.reach0 = line[0] - step[axis] * 0.5;
        x.reach1 = line[line.size() - 1] + step[axis] * 0.5;
        x.order = order;
        cols[axis] = (long long)x.wide * x.tall;
        col0[axis + 1] = col0[axis] + cols[axis];
    }
    cudaStream_t st;
    RS_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    struct Bufs {
        void* p[3] = {};
        cudaStream_t st;
        ~Bufs() {
            cudaStreamSynchronize(st);
            for (void* q : p) if (q) cudaFree(q);
            cudaStreamDestroy(st);
        }
    } m;
    m.st = st;
    // one allocation: the mesh, the lines, the masks, the columns' counts and offsets, the scan's room and
    // room for the lists of an ordinary mesh (8 crossings a column)
    const size_t nc = size_t(col0[3]);
    size_t scan = 0;
    RS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan, (const unsigned long long*)nullptr, (unsigned long long*)nullptr, (long long)(nc + 1), st));
    auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t room = 8 * nc;
    const size_t sizes[8] = {al(size_t(ntri) * 72), al((lens[0] + lens[1] + lens[2]) * 8), al(total), al(total), 256,
                             al((nc + 1) * 8), al((nc + 1) * 8), al(scan)};
    size_t bytes = al(room * 8);
    for (size_t b : sizes) bytes += b;
    RS_CUDA(cudaMalloc(&m.p[0], bytes));
    char* cur = static_cast<char*>(m.p[0]);
    char* part[9];
    for (int q = 0; q < 8; ++q) { part[q] = cur; cur += sizes[q]; }
    part[8] = cur;
    double* tri = reinterpret_cast<double*>(part[0]);
    double* dl = reinterpret_cast<double*>(part[1]);
    uint8_t *d_in = reinterpret_cast<uint8_t*>(part[2]), *d_thin = reinterpret_cast<uint8_t*>(part[3]);
    int* d_err = reinterpret_cast<int*>(part[4]);
    unsigned long long *count = reinterpret_cast<unsigned long long*>(part[5]), *offset = reinterpret_cast<unsigned long long*>(part[6]);
    double* hits = reinterpret_cast<double*>(part[8]);
    RS_CUDA(cudaMemcpyAsync(tri, tris, size_t(ntri) * 72, cudaMemcpyHostToDevice, st));
    for (int a = 0, at = 0; a < 3; at += int(lens[a]), ++a) {
        RS_CUDA(cudaMemcpyAsync(dl + at, samples[a].data(), lens[a] * 8, cudaMemcpyHostToDevice, st));
        for (int axis = 0; axis < 3; ++axis) f[axis].line[a] = dl + at;
    }
    RS_CUDA(cudaMemsetAsync(d_in, 0, sizes[2] + sizes[3] + sizes[4] + sizes[5], st));
    const dim3 grid(unsigned((ntri + 3) / 4), unsigned(std::min<uint64_t>(64, std::max<uint64_t>(1, 148 * 16 / ((ntri + 3) / 4)))));
    unsigned long long crossings = 0;
    const double* leaf = nullptr;
    auto count_all = [&]() -> int {   // each column's crossings, where its list starts, and whether a hit was a stray
        for (int a = 0; a < 3; ++a)
            k_crossings<false><<<grid, 128, 0, st>>>(f[a], tri, (long long)ntri, count + col0[a], nullptr, nullptr, 0, 0, cols[a], leaf,
                                                     d_err + 1);
        RS_CUDA(cudaGetLastError());
        RS_CUDA(cub::DeviceScan::ExclusiveSum(part[7], scan, count, offset, (long long)(nc + 1), st));
        RS_CUDA(cudaMemcpyAsync(&crossings, offset + nc, 8, cudaMemcpyDeviceToHost, st));
        return FG_OK;
    };
    int stray = 0, rc = count_all();
    if (rc) return rc;
    RS_CUDA(cudaMemcpyAsync(&stray, d_err + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    RS_CUDA(cudaStreamSynchronize(st));
    if (stray) {
        const Boxes boxes(tris, size_t(ntri));
        RS_CUDA(cudaMalloc(&m.p[2], size_t(ntri) * 48));
        RS_CUDA(cudaMemcpyAsync(m.p[2], boxes.out.data(), size_t(ntri) * 48, cudaMemcpyHostToDevice, st));
        leaf = static_cast<const double*>(m.p[2]);
        RS_CUDA(cudaMemsetAsync(count, 0, (nc + 1) * 8, st));
        if ((rc = count_all())) return rc;
        RS_CUDA(cudaStreamSynchronize(st));
    }
    // the columns in runs whose lists fit the room: all at once for an ordinary mesh, else at most 2^26
    // crossings (or one column's) at a time
    struct Piece { int axis; long long c0, c1; unsigned long long base; };
    std::vector<Piece> pieces;
    if (crossings <= room) {
        for (int a = 0; a < 3; ++a) pieces.push_back(Piece{a, 0, cols[a], 0});
    } else {
        std::vector<unsigned long long> off(nc + 1);
        RS_CUDA(cudaMemcpy(off.data(), offset, (nc + 1) * 8, cudaMemcpyDeviceToHost));
        unsigned long long most = 0;
        for (int a = 0; a < 3; ++a)
            for (long long c = 0; c < cols[a];) {
                const unsigned long long base = off[size_t(col0[a] + c)];
                long long e = c + 1;
                while (e < cols[a] && off[size_t(col0[a] + e + 1)] - base <= (1ull << 26)) ++e;
                most = std::max(most, off[size_t(col0[a] + e)] - base);
                pieces.push_back(Piece{a, c, e, base});
                c = e;
            }
        RS_CUDA(cudaMalloc(&m.p[1], size_t(most) * 8));
        hits = static_cast<double*>(m.p[1]);
    }
    RS_CUDA(cudaMemsetAsync(count, 0, nc * 8, st));   // counted again as the lists fill
    for (const Piece& p : pieces) {
        const long long o = col0[p.axis];
        k_crossings<true><<<grid, 128, 0, st>>>(f[p.axis], tri, (long long)ntri, count + o, offset + o, hits, p.base, p.c0, p.c1, leaf,
                                                d_err + 1);
        k_fill_axis<<<unsigned((p.c1 - p.c0 + 127) / 128), 128, 0, st>>>(f[p.axis], count + o, offset + o, hits, p.base, p.c0, p.c1,
                                                                       d_in, d_thin, d_err);
    }
    k_thin_only<<<unsigned(std::min<size_t>((total + 255) / 256, 148 * 16)), 256, 0, st>>>(d_in, d_thin, total);
    RS_CUDA(cudaGetLastError());
    int error = 0;
    RS_CUDA(cudaMemcpyAsync(&error, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    RS_CUDA(cudaMemcpyAsync(inside, d_in, total, cudaMemcpyDeviceToHost, st));
    RS_CUDA(cudaMemcpyAsync(thin, d_thin, total, cudaMemcpyDeviceToHost, st));
    RS_CUDA(cudaStreamSynchronize(st));
    if (error) {
        err = "a column crosses the mesh too often";
        return FG_ERR_INVALID;
    }
    return FG_OK;
}

// fill (raster.rs:24-104) on the device: inside / thin get 1 at the filled samples, indexed in the
// space of dimensions dims (order 0: (i m1 + j) m2 + k, 1: i + (j + k m1) m0; every sample index
// is below its dimension); thin is then cleared where inside is set. A fill that fails leaves both clear.
int raster_fill(Gpu* gpu, const double* tris, uint64_t ntri, const std::vector<double>* samples, const size_t* dims,
                int order, uint8_t* inside, uint8_t* thin, std::string& err) {
    for (int a = 0; a < 3; ++a)
        if (samples[a].size() > dims[a]) { err = "a sample line is longer than its index dimension"; return FG_ERR_INVALID; }
    const int rc = fill_masks(gpu, tris, ntri, samples, dims, order, inside, thin, err);
    if (rc) {
        std::memset(inside, 0, dims[0] * dims[1] * dims[2]);
        std::memset(thin, 0, dims[0] * dims[1] * dims[2]);
        cudaGetLastError();   // a failed allocation is not the next call's error
    }
    return rc;
}

int raster_sheet_edges(Gpu* gpu, const double* tris, uint64_t ntri, const std::vector<double>* lines, uint8_t* mask,
                       std::string& err) {
    using namespace raster;
    const size_t nn = lines[0].size() * lines[1].size() * lines[2].size();
    std::memset(mask, 0, 3 * nn);
    if (ntri == 0 || nn == 0) return FG_OK;
    for (int a = 0; a < 3; ++a)
        if (lines[a].size() < 2) { err = "a grid axis needs two lines"; return FG_ERR_INVALID; }
    RS_CUDA(cudaSetDevice(gpu->device));
    cudaStream_t st;
    RS_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    struct Bufs {
        void* p[3] = {};
        cudaStream_t st;
        ~Bufs() {
            cudaStreamSynchronize(st);
            for (void* q : p) if (q) cudaFree(q);
            cudaStreamDestroy(st);
        }
    } m;
    m.st = st;
    const size_t lens[3] = {lines[0].size(), lines[1].size(), lines[2].size()};
    RS_CUDA(cudaMalloc(&m.p[0], size_t(ntri) * 9 * sizeof(double)));
    RS_CUDA(cudaMalloc(&m.p[1], (lens[0] + lens[1] + lens[2]) * sizeof(double)));
    RS_CUDA(cudaMalloc(&m.p[2], 3 * nn));
    RS_CUDA(cudaMemcpyAsync(m.p[0], tris, size_t(ntri) * 9 * sizeof(double), cudaMemcpyHostToDevice, st));
    double* dl = static_cast<double*>(m.p[1]);
    RS_CUDA(cudaMemcpyAsync(dl, lines[0].data(), lens[0] * 8, cudaMemcpyHostToDevice, st));
    RS_CUDA(cudaMemcpyAsync(dl + lens[0], lines[1].data(), lens[1] * 8, cudaMemcpyHostToDevice, st));
    RS_CUDA(cudaMemcpyAsync(dl + lens[0] + lens[1], lines[2].data(), lens[2] * 8, cudaMemcpyHostToDevice, st));
    RS_CUDA(cudaMemsetAsync(m.p[2], 0, 3 * nn, st));
    SheetArgs g{};
    g.line[0] = dl;
    g.line[1] = dl + lens[0];
    g.line[2] = dl + lens[0] + lens[1];
    for (int a = 0; a < 3; ++a) g.n[a] = int(lens[a]);
    const unsigned blocks = unsigned(std::min<uint64_t>(ntri, 148 * 32));
    k_sheet_edges<<<blocks, 256, 0, st>>>(g, static_cast<const double*>(m.p[0]), (long long)ntri,
                                          static_cast<uint8_t*>(m.p[2]));
    RS_CUDA(cudaGetLastError());
    RS_CUDA(cudaMemcpyAsync(mask, m.p[2], 3 * nn, cudaMemcpyDeviceToHost, st));
    RS_CUDA(cudaStreamSynchronize(st));
    return FG_OK;
}

// closed (raster.rs:127-143): every edge of the non-degenerate triangles, keyed by its quantised
// end points, is shared by an even number of them.
bool raster_closed(const double* tris, uint64_t ntri) {
    if (ntri == 0) return false;
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (uint64_t q = 0; q < ntri * 3; ++q)
        for (int a = 0; a < 3; ++a) {
            lo[a] = std::fmin(lo[a], tris[q * 3 + a]);
            hi[a] = std::fmax(hi[a], tris[q * 3 + a]);
        }
    double size = 0.0;
    for (int a = 0; a < 3; ++a) size = std::fmax(size, hi[a] - lo[a]);
    size = std::fmax(size, 1e-30);
    const double base = std::fmin(std::fmin(lo[0], lo[1]), lo[2]);
    struct Key {
        int64_t a[3], b[3];
        bool operator==(const Key& o) const { return std::memcmp(this, &o, sizeof(Key)) == 0; }
    };
    struct Hash {
        size_t operator()(const Key& k) const {
            uint64_t h = 1469598103934665603ull;
            const int64_t* v = k.a;
            for (int q = 0; q < 6; ++q) h = (h ^ uint64_t(v[q])) * 1099511628211ull;
            return size_t(h);
        }
    };
    std::unordered_map<Key, uint32_t, Hash> edges;
    auto key = [&](const double* p, int64_t* o) {
        for (int a = 0; a < 3; ++a) o[a] = int64_t(std::round((p[a] - base) / size * 1e9));
    };
    for (uint64_t t = 0; t < ntri; ++t) {
        int64_t k[3][3];
        for (int v = 0; v < 3; ++v) key(tris + t * 9 + v * 3, k[v]);
        auto same = [&](int x, int y) { return k[x][0] == k[y][0] && k[x][1] == k[y][1] && k[x][2] == k[y][2]; };
        if (same(0, 1) || same(1, 2) || same(0, 2)) continue;
        const int pairs[3][2] = {{0, 1}, {1, 2}, {2, 0}};
        for (auto& pr : pairs) {
            const int64_t* a = k[pr[0]];
            const int64_t* b = k[pr[1]];
            const bool less = std::lexicographical_compare(a, a + 3, b, b + 3);
            Key e;
            std::memcpy(e.a, less ? a : b, sizeof e.a);
            std::memcpy(e.b, less ? b : a, sizeof e.b);
            edges[e] += 1;
        }
    }
    if (edges.empty()) return false;
    for (auto& kv : edges)
        if (kv.second % 2 != 0) return false;
    return true;
}

}  // namespace fg
