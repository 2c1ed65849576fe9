// Far field of the NTFF box on the device: Far::field (sims-field ntff.rs:90-116) for many directions
// at once, all sums in f64.
//
// Each patch adds its six complex currents times a e^{jk r.d} to a direction's sums: 24 fused
// multiply-adds, and a sine and cosine of about as many operations again where each (patch, direction)
// forms its own phase. The patches of a box come as lines along an axis: consecutive patches that share
// two coordinates and differ in the third, with the same sequence of third coordinates from line to line.
// So the phase is that of the line (one per line and direction) times that of the coordinate (one per
// sequence entry and direction), and k_far_lines sums a line with the latter alone, from a table in
// shared memory: 24 fused multiply-adds per pair and nothing else. A lane owns a direction, a warp sums
// four lines at a time (a table entry serves four, the lines' currents come as broadcasts, staged with
// cp.async), and a block's warps share the table of 32 directions. Its floor is the FP64 rate: 174,760
// patches x 2664 directions are 11.2 G multiply-adds, 0.6 ms at 64 per SM and clock; a repeated call takes
// 2.0 ms, the first on a handle, which lays its patches out on the device, 4.5 to 6; a block per direction took
// 13.4 with its copies each time.
// Patches that do not come in lines (fewer than 8 per line on average), or whose lines hardly share their
// sequences (FAR_SEQUENCES, FAR_PADDING), go through k_far_field, a block per direction, which forms every
// phase.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "../../include/fieldgrid.h"
#include "engine.hpp"

namespace fg {

namespace {

constexpr int FAR_THREADS = 256;

// The far field of one direction from its twelve sums (N then L, re and im): ntff.rs:100-116.
__device__ __forceinline__ void far_finish(const double (&s)[12], const double d[3], double kw, double* o) {
    double rn0 = 0, rn1 = 0;
    for (int c = 0; c < 3; ++c) { rn0 += s[2 * c] * d[c]; rn1 += s[2 * c + 1] * d[c]; }
    const double eta0 = 376.730313668;
    const double scale = kw / (4.0 * 3.14159265358979323846);
    const double* l = s + 6;
    const double rl[3][2] = {{d[1] * l[4] - d[2] * l[2], d[1] * l[5] - d[2] * l[3]},
                             {d[2] * l[0] - d[0] * l[4], d[2] * l[1] - d[0] * l[5]},
                             {d[0] * l[2] - d[1] * l[0], d[0] * l[3] - d[1] * l[1]}};
    for (int c = 0; c < 3; ++c) {
        const double p0 = s[2 * c] - rn0 * d[c], p1 = s[2 * c + 1] - rn1 * d[c];
        o[2 * c] = (rl[c][0] - p0 * eta0) * scale;
        o[2 * c + 1] = (rl[c][1] - p1 * eta0) * scale;
    }
}

__global__ void __launch_bounds__(FAR_THREADS) k_far_field(const double* __restrict__ pos, const double* __restrict__ jm,
                                                           long long count, double kw, const double* __restrict__ dirs,
                                                           double* __restrict__ out) {
    __shared__ double red[12][FAR_THREADS / 32];
    const double* dir = dirs + 3 * (long long)blockIdx.x;
    const double d[3] = {dir[0], dir[1], dir[2]};
    double acc[12];
#pragma unroll
    for (int q = 0; q < 12; ++q) acc[q] = 0.0;
    for (long long i = threadIdx.x; i < count; i += blockDim.x) {
        const double* p = pos + 3 * i;
        const double arg = kw * (d[0] * p[0] + d[1] * p[1] + d[2] * p[2]);
        double s, c;
        sincos(arg, &s, &c);
        const double* x = jm + 12 * i;   // the currents times the patch's area
#pragma unroll
        for (int q = 0; q < 12; q += 2) {
            acc[q] = __fma_rn(x[q], c, __fma_rn(-x[q + 1], s, acc[q]));
            acc[q + 1] = __fma_rn(x[q], s, __fma_rn(x[q + 1], c, acc[q + 1]));
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 12; ++q) {
        double v = acc[q];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[q][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s[12];
        for (int q = 0; q < 12; ++q) {
            s[q] = 0.0;
            for (int w = 0; w < FAR_THREADS / 32; ++w) s[q] += red[q][w];
        }
        far_finish(s, d, kw, out + 6 * (long long)blockIdx.x);
    }
}

// Up to four lines with one sequence: their first patches (consecutive lines' patches need not touch).
struct FarGroup {
    int first[4];       // a missing line repeats the first one, its sums are dropped
    double base[4][3];  // the lines' coordinates, 0 along the sequence's axis
    int lines, pad;
};
// One block's share: groups [g0, g1) of a sequence of `len` coordinates along `axis`.
struct FarPart {
    int axis, len, seq, g0, g1;
};

constexpr int FAR_LEN = 320;      // a line's patches at most (longer lines are cut into equal pieces)
constexpr int FAR_WARPS = 8;
constexpr int FAR_TILE = 8;       // patches of four lines a warp stages at a time
constexpr int FAR_STAGE = 4 * FAR_TILE * 12;   // doubles
// Sequences at most, each a block's table at least and sums of its own: a box has one or two per axis. Past
// that, and where the slots of the blocks' passes (FAR_WARPS groups of four lines) would be more than
// FAR_PADDING times the patches, k_far_field takes over: a pair costs it 6.7 times a filled slot (174,760
// patches, 2664 directions: 13.4 ms against 2.0).
constexpr size_t FAR_SEQUENCES = 4096;
constexpr long long FAR_PADDING = 4;
constexpr uint64_t FAR_PARTIAL = uint64_t(256) << 20;   // bytes of partial sums at a time, above 32 directions
constexpr int FAR_SMEM = FAR_LEN * 32 * 16 + FAR_WARPS * 2 * FAR_STAGE * 8;

__device__ __forceinline__ void cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(unsigned(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

// Block (t, p): directions 32 t .. 32 t + 31, part p; the twelve sums of each to partial[(p n + dir) 12].
__global__ void __launch_bounds__(32 * FAR_WARPS, 1)
    k_far_lines(const FarPart* __restrict__ parts, const FarGroup* __restrict__ groups, const double* __restrict__ seqs,
                const double* __restrict__ jm, double kw, const double* __restrict__ dirs, int n, double* __restrict__ partial) {
    extern __shared__ __align__(16) unsigned char far_sm[];
    double2* table = reinterpret_cast<double2*>(far_sm);   // [coordinate][direction]: (cos, sin)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* stage = reinterpret_cast<double*>(far_sm + FAR_LEN * 32 * 16) + warp * 2 * FAR_STAGE;
    const FarPart p = parts[blockIdx.y];
    const int q = min(int(blockIdx.x) * 32 + lane, n - 1);
    const double d[3] = {dirs[3 * q], dirs[3 * q + 1], dirs[3 * q + 2]};
    const double* seq = seqs + p.seq;
    for (int v = warp; v < p.len; v += FAR_WARPS) {
        double s, c;
        sincos(kw * (d[p.axis] * seq[v]), &s, &c);
        table[v * 32 + lane] = make_double2(c, s);
    }
    __syncthreads();
    double sum[12];
#pragma unroll
    for (int x = 0; x < 12; ++x) sum[x] = 0.0;
    const int tiles = (p.len + FAR_TILE - 1) / FAR_TILE;
    for (int gi = p.g0 + warp; gi < p.g1; gi += FAR_WARPS) {
        const FarGroup& G = groups[gi];
        // a tile: FAR_TILE patches of each line, 96 bytes a patch, six 16-byte copies a lane
        auto fetch = [&](int t, int buf) {
            const int m = min(FAR_TILE, p.len - t * FAR_TILE) * 6;
            for (int l = 0; l < 4; ++l) {
                const double* src = jm + ((long long)G.first[l] + t * FAR_TILE) * 12;
                double* dst = stage + buf * FAR_STAGE + l * (FAR_TILE * 12);
                for (int x = lane; x < m; x += 32) cp16(dst + 2 * x, src + 2 * x);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        double acc[4][12];
#pragma unroll
        for (int l = 0; l < 4; ++l)
#pragma unroll
            for (int x = 0; x < 12; ++x) acc[l][x] = 0.0;
        __syncwarp();
        fetch(0, 0);
        for (int t = 0; t < tiles; ++t) {
            if (t + 1 < tiles) {
                fetch(t + 1, (t + 1) & 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncwarp();
            const double* st = stage + (t & 1) * FAR_STAGE;
            const int m = min(FAR_TILE, p.len - t * FAR_TILE);
            for (int v = 0; v < m; ++v) {
                const double2 e = table[(t * FAR_TILE + v) * 32 + lane];
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    const double2* x = reinterpret_cast<const double2*>(st + (l * FAR_TILE + v) * 12);
#pragma unroll
                    for (int y = 0; y < 6; ++y) {
                        const double2 z = x[y];
                        acc[l][2 * y] = __fma_rn(z.x, e.x, __fma_rn(-z.y, e.y, acc[l][2 * y]));
                        acc[l][2 * y + 1] = __fma_rn(z.x, e.y, __fma_rn(z.y, e.x, acc[l][2 * y + 1]));
                    }
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            double s, c;
            sincos(kw * (d[0] * G.base[l][0] + d[1] * G.base[l][1] + d[2] * G.base[l][2]), &s, &c);
            if (l >= G.lines) s = c = 0.0;
#pragma unroll
            for (int x = 0; x < 12; x += 2) {
                sum[x] = __fma_rn(acc[l][x], c, __fma_rn(-acc[l][x + 1], s, sum[x]));
                sum[x + 1] = __fma_rn(acc[l][x], s, __fma_rn(acc[l][x + 1], c, sum[x + 1]));
            }
        }
    }
    __syncthreads();   // the table's room now holds the warps' sums
    double* red = reinterpret_cast<double*>(far_sm);
#pragma unroll
    for (int x = 0; x < 12; ++x) red[(warp * 12 + x) * 32 + lane] = sum[x];
    __syncthreads();
    for (int x = warp; x < 12; x += FAR_WARPS) {
        double v = 0.0;
        for (int w = 0; w < FAR_WARPS; ++w) v += red[(w * 12 + x) * 32 + lane];
        const int at = int(blockIdx.x) * 32 + lane;
        if (at < n) partial[((long long)blockIdx.y * n + at) * 12 + x] = v;
    }
}

// Each direction's parts summed in order, and its field.
__global__ void k_far_finish(const double* __restrict__ partial, int parts, int n, double kw, const double* __restrict__ dirs,
                             double* __restrict__ out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    double s[12];
    for (int x = 0; x < 12; ++x) s[x] = 0.0;
    for (int p = 0; p < parts; ++p)
        for (int x = 0; x < 12; ++x) s[x] += partial[((long long)p * n + q) * 12 + x];
    const double d[3] = {dirs[3 * q], dirs[3 * q + 1], dirs[3 * q + 2]};
    far_finish(s, d, kw, out + 6 * (long long)q);
}

// Each patch's currents times its area.
__global__ void k_far_areas(double* __restrict__ jm, const double* __restrict__ area, long long count) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < 12 * count; q += (long long)gridDim.x * blockDim.x)
        jm[q] *= area[q / 12];
}

// The patches as lines with shared sequences.
struct Line {
    int first, len, axis, seq;   // seq: offset into the sequence values
};

void find_lines(const double* pos, int count, std::vector<Line>& lines, std::vector<double>& seqs) {
    struct Known { int first, len, axis; };
    std::vector<Known> known;   // the sequences so far, newest last
    for (int i = 0; i < count;) {
        const double* a = pos + 3 * (size_t)i;
        int axis = -1, n = 1;
        for (; i + n < count; ++n) {
            const double* b = a + 3 * (size_t)n;
            int diff = -1, many = 0;
            for (int x = 0; x < 3; ++x)
                if (std::memcmp(a + x, b + x, 8) != 0) { diff = x; ++many; }
            if (many != 1 || (axis >= 0 && diff != axis)) break;
            axis = diff;
        }
        if (axis < 0) axis = known.empty() ? 0 : known.back().axis;
        const int pieces = (n + FAR_LEN - 1) / FAR_LEN;
        for (int c = 0; c < pieces; ++c) {
            const int v0 = int((long long)n * c / pieces), m = int((long long)n * (c + 1) / pieces) - v0;
            const double* p = a + 3 * (size_t)v0;
            // its sequence: a recent one with the same values, or a new one
            int seq = -1;
            for (size_t k = known.size(); k-- > 0 && known.size() - k <= 16 && seq < 0;) {
                if (known[k].len != m || known[k].axis != axis) continue;
                bool same = true;
                for (int v = 0; v < m && same; ++v) same = std::memcmp(&seqs[size_t(known[k].first + v)], p + 3 * (size_t)v + axis, 8) == 0;
                if (same) seq = known[k].first;
            }
            if (seq < 0) {
                seq = int(seqs.size());
                for (int v = 0; v < m; ++v) seqs.push_back(p[3 * (size_t)v + axis]);
                known.push_back(Known{seq, m, axis});
            }
            lines.push_back(Line{i + v0, m, axis, seq});
        }
        i += n;
    }
}

}  // namespace

// What a Far keeps on its device: the currents times their areas, and the patches' lines (or, where
// they form none, the positions). Laid out on the first call with the device's handle. All handles
// together keep at most FAR_KEEP bytes: a call that ends above it gives its handle's back.
constexpr long long FAR_KEEP = 1LL << 30;
std::atomic<long long> far_kept{0};

struct FarDevice {
    int device = 0;
    long long count = 0;
    char* mem = nullptr;              // one allocation: the layout, and behind it the first call's work
    double *pos = nullptr, *jm = nullptr, *seqs = nullptr;
    FarGroup* groups = nullptr;
    bool lined = false;
    struct Run { int axis, len, seq, g0, g1; };   // groups of one sequence
    std::vector<Run> runs;
    char *work = nullptr, *own_work = nullptr;   // the calls' directions, parts and partial sums; an allocation of its own once outgrown
    size_t work_bytes = 0;
    long long bytes = 0, kept = 0;    // allocated; what far_kept counts for this one
    ~FarDevice() {
        far_kept -= kept;
        int prev = 0;
        const bool back = cudaGetDevice(&prev) == cudaSuccess;
        cudaSetDevice(device);
        cudaFree(mem);
        if (own_work) cudaFree(own_work);
        if (back) cudaSetDevice(prev);
    }
};

void far_device_free(FarDevice* d) { delete d; }

namespace {

// The patches' lines in groups of four, where they form lines that share their sequences.
void far_groups(const double* pos, uint64_t count, FarDevice& D, std::vector<FarGroup>& groups, std::vector<double>& seqs) {
    std::vector<Line> lines;
    D.lined = false;
    if (count > 0 && count < (uint64_t(1) << 31)) {
        find_lines(pos, int(count), lines, seqs);
        D.lined = lines.size() * 8 <= count;
    }
    if (!D.lined) return;
    // lines of one sequence, in their order, four to a group
    std::stable_sort(lines.begin(), lines.end(), [](const Line& a, const Line& b) { return a.seq < b.seq; });
    long long slots = 0;
    for (size_t i = 0; i < lines.size();) {
        size_t e = i;
        while (e < lines.size() && lines[e].seq == lines[i].seq) ++e;
        FarDevice::Run r{lines[i].axis, lines[i].len, lines[i].seq, int(groups.size()), 0};
        for (size_t q = i; q < e; q += 4) {
            FarGroup G{};
            G.lines = int(std::min<size_t>(4, e - q));
            for (int l = 0; l < 4; ++l) {
                const Line& L = lines[q + size_t(l < G.lines ? l : 0)];
                G.first[l] = L.first;
                for (int x = 0; x < 3; ++x) G.base[l][x] = x == L.axis ? 0.0 : pos[3 * (size_t)L.first + x];
            }
            groups.push_back(G);
        }
        r.g1 = int(groups.size());
        D.runs.push_back(r);
        slots += (long long)((r.g1 - r.g0 + FAR_WARPS - 1) / FAR_WARPS) * FAR_WARPS * 4 * r.len;
        i = e;
    }
    D.lined = D.runs.size() <= FAR_SEQUENCES && slots <= FAR_PADDING * (long long)count;
}

// Allocates and fills a handle's layout, with `work` bytes behind it.
int far_layout(Gpu* g, const double* pos, const double* area, const double* jm, uint64_t count, FarDevice& D,
               const std::vector<FarGroup>& groups, const std::vector<double>& seqs, size_t work, std::string& err) {
    auto check = [&](cudaError_t e, const char* what) {
        if (e != cudaSuccess) { err = std::string(what) + ": " + cudaGetErrorString(e); return false; }
        return true;
    };
    auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t jb = al(13 * count * 8), gb = D.lined ? al(groups.size() * sizeof(FarGroup)) : 0;
    const size_t sb = D.lined ? al(seqs.size() * 8) : al(3 * count * 8);
    if (!check(cudaMalloc(&D.mem, jb + gb + sb + work), "cudaMalloc")) return FG_ERR_CUDA;
    D.bytes = (long long)(jb + gb + sb + work);
    D.jm = reinterpret_cast<double*>(D.mem);
    D.work = D.mem + jb + gb + sb;
    D.work_bytes = work;
    // the currents, then their areas behind them for the products
    if (count) {
        double* a = D.jm + 12 * count;
        if (!check(cudaError_t(staged_upload(g, D.jm, jm, 12 * count * 8, nullptr)), "cudaMemcpy") ||
            !check(cudaError_t(staged_upload(g, a, area, count * 8, nullptr)), "cudaMemcpy"))
            return FG_ERR_CUDA;
        k_far_areas<<<unsigned(std::min<uint64_t>((12 * count + 255) / 256, 148 * 8)), 256>>>(D.jm, a, (long long)count);
        if (!check(cudaGetLastError(), "k_far_areas")) return FG_ERR_CUDA;
    }
    if (D.lined) {
        D.groups = reinterpret_cast<FarGroup*>(D.mem + jb);
        D.seqs = reinterpret_cast<double*>(D.mem + jb + gb);
        if (!check(cudaMemcpy(D.groups, groups.data(), groups.size() * sizeof(FarGroup), cudaMemcpyHostToDevice), "cudaMemcpy") ||
            !check(cudaMemcpy(D.seqs, seqs.data(), seqs.size() * 8, cudaMemcpyHostToDevice), "cudaMemcpy") ||
            !check(cudaFuncSetAttribute(k_far_lines, cudaFuncAttributeMaxDynamicSharedMemorySize, FAR_SMEM), "cudaFuncSetAttribute"))
            return FG_ERR_CUDA;
    } else if (count) {
        D.pos = reinterpret_cast<double*>(D.mem + jb);
        if (!check(cudaMemcpy(D.pos, pos, 3 * count * 8, cudaMemcpyHostToDevice), "cudaMemcpy")) return FG_ERR_CUDA;
    }
    return FG_OK;
}

}  // namespace

int far_field_gpu(Gpu* g, std::vector<FarDevice*>& devices, const double* pos, const double* area, const double* jm, uint64_t count,
                  double freq, const double* dirs, uint64_t n, double* out, std::string& err) {
    if (n == 0) return FG_OK;
    auto check = [&](cudaError_t e, const char* what) {
        if (e != cudaSuccess) { err = std::string(what) + ": " + cudaGetErrorString(e); return false; }
        return true;
    };
    if (!check(cudaSetDevice(g->device), "cudaSetDevice")) return FG_ERR_CUDA;
    FarDevice* dev = nullptr;   // the handle's layout on this device, made on first use
    for (FarDevice* d : devices)
        if (d->device == g->device) dev = d;
    std::unique_ptr<FarDevice> made;
    std::vector<FarGroup> groups;
    std::vector<double> seqs;
    if (!dev) {
        made.reset(dev = new FarDevice);
        dev->device = g->device;
        dev->count = (long long)count;
        far_groups(pos, count, *dev, groups, seqs);
    }
    FarDevice& D = *dev;
    const double kw = 2.0 * 3.14159265358979323846 * freq / 299792458.0;
    constexpr uint64_t MOST = 65535;   // directions at a time
    const int m0 = int(std::min<uint64_t>(n, MOST));
    // parts of about equal work, in whole passes of a block's warps, for about seven waves of blocks over
    // the direction tiles (the last wave's loss against each block's table of phases); where there is
    // less work than one pass per SM, a group a block
    std::vector<FarPart> parts;
    if (D.lined) {
        long long work = 0, all = 0;
        for (const auto& r : D.runs) {
            work += (long long)(r.g1 - r.g0) * r.len;
            all += r.g1 - r.g0;
        }
        const long long tiles = (m0 + 31) / 32, per = std::max<long long>(work * tiles / (148 * 7), 1);
        const bool few = tiles * all < 148 * FAR_WARPS;
        for (const auto& r : D.runs) {
            const long long pass = (long long)r.len * FAR_WARPS;
            const int m = few ? 1 : FAR_WARPS * int(std::max<long long>(1, (per + pass / 2) / pass));
            for (int q = r.g0; q < r.g1; q += m) parts.push_back(FarPart{r.axis, r.len, r.seq, q, std::min(q + m, r.g1)});
        }
    }
    // directions at a time: no more partial sums than FAR_PARTIAL
    const uint64_t step = parts.empty() ? MOST : std::min<uint64_t>(MOST, std::max<uint64_t>(32, FAR_PARTIAL / (96 * parts.size()) / 32 * 32));
    const int ms = int(std::min<uint64_t>(n, step));
    const size_t pb = (parts.size() * sizeof(FarPart) + 255) & ~size_t(255);
    const size_t bytes = pb + (size_t(9) + size_t(12) * parts.size()) * size_t(ms) * 8 + 256;
    if (made) {
        if (const int rc = far_layout(g, pos, area, jm, count, D, groups, seqs, bytes, err)) return rc;
        devices.push_back(made.release());
    } else if (D.work_bytes < bytes) {
        if (D.own_work) {
            cudaFree(D.own_work);
            D.bytes -= (long long)D.work_bytes;
        }
        D.work = D.own_work = nullptr;
        D.work_bytes = 0;
        if (!check(cudaMalloc(&D.own_work, bytes), "cudaMalloc")) return FG_ERR_CUDA;
        D.work = D.own_work;
        D.work_bytes = bytes;
        D.bytes += (long long)bytes;
    }
    char* buf = D.work;
    double* d_dirs = reinterpret_cast<double*>(buf + pb);
    double* d_out = d_dirs + 3 * size_t(ms);
    double* d_part = d_out + 6 * size_t(ms);
    bool ok = parts.empty() || check(cudaMemcpyAsync(buf, parts.data(), parts.size() * sizeof(FarPart), cudaMemcpyHostToDevice, nullptr), "cudaMemcpy");
    for (uint64_t first = 0; first < n && ok; first += step) {
        const int m = int(std::min<uint64_t>(step, n - first));
        ok = check(cudaMemcpyAsync(d_dirs, dirs + 3 * first, size_t(m) * 24, cudaMemcpyHostToDevice, nullptr), "cudaMemcpy");
        if (!ok) break;
        if (D.lined) {
            const dim3 grid(unsigned((m + 31) / 32), unsigned(parts.size()));
            k_far_lines<<<grid, 32 * FAR_WARPS, FAR_SMEM>>>(reinterpret_cast<const FarPart*>(buf), D.groups, D.seqs, D.jm, kw,
                                                             d_dirs, m, d_part);
            k_far_finish<<<unsigned((m + 127) / 128), 128>>>(d_part, int(parts.size()), m, kw, d_dirs, d_out);
        } else {
            k_far_field<<<unsigned(m), FAR_THREADS>>>(D.pos, D.jm, D.count, kw, d_dirs, d_out);
        }
        ok = check(cudaGetLastError(), "far field") &&
             check(cudaMemcpyAsync(out + 6 * first, d_out, size_t(m) * 48, cudaMemcpyDeviceToHost, nullptr), "cudaMemcpy");
    }
    ok = check(cudaStreamSynchronize(nullptr), "far field") && ok;
    const long long all = far_kept += D.bytes - D.kept;
    D.kept = D.bytes;
    if (all > FAR_KEEP) {
        devices.erase(std::find(devices.begin(), devices.end(), dev));
        delete dev;
    }
    return ok ? FG_OK : FG_ERR_CUDA;
}

}  // namespace fg
