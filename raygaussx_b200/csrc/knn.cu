// rgx_knn_mean_dist2: for every point the mean of the squared distances to its three
// nearest other points -- what the reference's point-cloud initialisation asks of
// simple-knn (classes/point_cloud.py:252,592 -> submodules/simple-knn/simple_knn.cu,
// SimpleKNN::knn) to size the first Gaussians.
//
// Exact, like the reference: points are sorted along a Hilbert curve, every 32
// consecutive points get a box, every 32 boxes a box of their own, and 32 of those
// again.  A warp owns 32 consecutive sorted points, one query per lane.  It descends
// the three levels with lanes as nodes: 32 boxes at a time against the box of its 32
// queries and the worst third-best distance among them.  A box of points that passes is
// opened if it is nearer to some lane's query than that lane's third-best; its points
// are then read by all lanes at once from shared memory.
//   Queries of a warp are neighbours in space, so after the seed (the warp's own box and
// its two neighbours) few boxes are opened and what bounds the kernel is the distance
// arithmetic of those.  Testing every upper box by every warp, as an earlier version did, took 15.3 ms
// for 3 M points (now 0.85 ms); the whole call, whose eleven allocations and frees cost more than
// its kernels on small clouds, took 19.9 ms for 3 M (now 1.27) and 0.4 ms (in a process with a large
// workspace several ms) for 100 k points (now 0.17, scratch from the caller).
#include "rgx_internal.cuh"
#include "device_math.cuh"
#include "cluster_sort.cuh"
#include <cub/device/device_radix_sort.cuh>
#include <algorithm>

namespace rgx {

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kKnnWarps = 8;

// bounds: [0, 3) largest coordinates, [3, 6) largest negated coordinates, as ordered integers that start at zero
__global__ void __launch_bounds__(256) knn_bounds_kernel(const float* pts, int n, unsigned* bounds) {
    after_previous();
    __shared__ unsigned s_max[6];
    if (threadIdx.x < 6) s_max[threadIdx.x] = 0u;
    __syncthreads();
    unsigned m[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float v = pts[3 * (size_t)i + a];
            m[a] = max(m[a], ordered(v));
            m[3 + a] = max(m[3 + a], ordered(-v));
        }
#pragma unroll
    for (int a = 0; a < 6; ++a) {
        const unsigned v = __reduce_max_sync(kAll, m[a]);
        if ((threadIdx.x & 31) == 0) atomicMax(&s_max[a], v);
    }
    __syncthreads();
    if (threadIdx.x < 6) atomicMax(&bounds[threadIdx.x], s_max[threadIdx.x]);
}

// Positions along a Hilbert curve.  A cell that holds many points leaves them in no order, their boxes of 32 all as large as
// the cell, so a cloud whose extent is set by a few far points needs fine cells: sixteen points at 1,000 times the size of a cloud of
// 1 M on surfaces take the whole call from 6.1 ms to 38.2 with 10 bits per axis instead of 16, 300 k from 2.0 to 5.3, 100 k from 0.70 to
// 1.19, 65 k from 0.48 to 0.67, 30 k from 0.31 to 0.35, and 3 M points of a core and a shell from 1.43 to 1.78.  Where there are none,
// sorting 64-bit keys costs 0.02 to 0.07 ms (100 k on surfaces 0.153 -> 0.177, 1 M 0.446 -> 0.509).  The extent cannot be told without
// waiting for the device, so the line is the count from which the loss outweighs that price.
template <class Key>
__global__ void __launch_bounds__(256) knn_keys_kernel(const float* pts, int n, const unsigned* bounds,
                                                       Key* keys, unsigned* vals) {
    after_previous();
    constexpr int kBits = sizeof(Key) == 8 ? 16 : 10;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float top = (float)((1 << kBits) - 1);
    uint32_t q[3];
    for (int a = 0; a < 3; ++a) {
        float lo = -unordered(bounds[3 + a]), hi = unordered(bounds[a]);
        float ext = hi - lo;
        float u = ext > 0.f ? (pts[3 * (size_t)i + a] - lo) / ext : 0.f;
        q[a] = (uint32_t)fminf(fmaxf(u * top, 0.f), top);
    }
    hilbert_transpose(q, kBits);
    keys[i] = (Key)((spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]));
    vals[i] = (unsigned)i;
}
inline bool wide_keys(int n) { return n >= 65536; }

// Boxes of one level: lo and hi per node.
struct KnnLevel {
    float4 *lo, *hi;
    int count;
};

// The box of the warp's 32 boxes (an empty one is (+inf, -inf): at infinite distance), on lane 0.
__device__ __forceinline__ void warp_box(float (&lo)[3], float (&hi)[3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(kAll, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(kAll, hi[a], o));
        }
}

// Sorted copies of the points, padded to a multiple of 32 with points at infinity, their boxes and, a block of 1,024 points
// being one node of the level above, that node's.  A point of which a coordinate is no number goes to infinity, where it is nobody's
// neighbour, and into no box: the reference's comparisons pass by it too.
__global__ void __launch_bounds__(1024) knn_gather_kernel(const float* pts, int n, const unsigned* order,
                                                          float4* sorted, KnnLevel leaf, KnnLevel mid) {
    after_previous();
    __shared__ float s_lo[32][3], s_hi[32][3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * 1024 + threadIdx.x, b = blockIdx.x * 32 + warp;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n) {
        const size_t s = order[i];
        p = make_float4(pts[3 * s], pts[3 * s + 1], pts[3 * s + 2], 0.f);
    }
    const bool is = i < n && p.x == p.x && p.y == p.y && p.z == p.z;
    if (!is) p = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
    if (b < leaf.count) sorted[i] = p;
    float lo[3] = {p.x, p.y, p.z}, hi[3] = {is ? p.x : -INFINITY, is ? p.y : -INFINITY, is ? p.z : -INFINITY};
    warp_box(lo, hi);
    if (lane == 0) {
        if (b < leaf.count) {
            leaf.lo[b] = make_float4(lo[0], lo[1], lo[2], 0.f);
            leaf.hi[b] = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
        for (int a = 0; a < 3; ++a) { s_lo[warp][a] = lo[a]; s_hi[warp][a] = hi[a]; }
    }
    __syncthreads();
    if (warp == 0) {
        for (int a = 0; a < 3; ++a) { lo[a] = s_lo[lane][a]; hi[a] = s_hi[lane][a]; }
        warp_box(lo, hi);
        if (lane == 0) {
            mid.lo[blockIdx.x] = make_float4(lo[0], lo[1], lo[2], 0.f);
            mid.hi[blockIdx.x] = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
    }
}

// LATE: the query is set up when the gathering is done, not beside it.  Where it has few blocks they crowd otherwise on the SMs without a
// block of knn_gather_kernel: with 3,125 warps, 391 blocks of eight, beside 98 of those, on 50 SMs.  Up to four blocks per SM (151 k points
// on 148); whole call, us, beside it and behind it: 40 k points of an object 122.7 and 116.1, 65 k 152.6 and 141.4, 80 k on surfaces 161.1
// and 148.3, 100 k 182.5 and 174.1, 130 k 187.8 and 182.5, 150 k 193.2 and 192.6; beyond that either may be the faster (180 k on surfaces
// 206.9 and 200.1, 230 k 214.3 and 221.3).
template <bool LATE>
__global__ void __launch_bounds__(256) knn_upper_kernel(KnnLevel below, KnnLevel level) {
    if (LATE) after_previous_then_next();
    else after_previous();
    const int node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (node >= level.count) return;
    const int b = node * 32 + lane;
    const float4 l = b < below.count ? below.lo[b] : make_float4(INFINITY, INFINITY, INFINITY, 0.f);
    const float4 h = b < below.count ? below.hi[b] : make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
    float lo[3] = {l.x, l.y, l.z}, hi[3] = {h.x, h.y, h.z};
    warp_box(lo, hi);
    if (lane == 0) {
        level.lo[node] = make_float4(lo[0], lo[1], lo[2], 0.f);
        level.hi[node] = make_float4(hi[0], hi[1], hi[2], 0.f);
    }
}

// squared distance from a point to a box (0 inside; +inf for an empty box)
__device__ __forceinline__ float box_dist2(float4 lo, float4 hi, float4 p) {
    float dx = fmaxf(fmaxf(lo.x - p.x, p.x - hi.x), 0.f), dy = fmaxf(fmaxf(lo.y - p.y, p.y - hi.y), 0.f),
          dz = fmaxf(fmaxf(lo.z - p.z, p.z - hi.z), 0.f);
    return dx * dx + dy * dy + dz * dz;
}

struct KnnTree {
    KnnLevel leaf, mid, top;
};

// FILTER: eight points at a time are passed by where none of them is nearer to its query than what a lane has.  Of the points opened
// few are, so that saves most of the bookkeeping where the kernel is bound by arithmetic (whole call, 3 M points of a core and a shell
// 1,424 -> 1,271 us, 1 M of an object 539 -> 489, 1 M on surfaces 493 -> 483); with fewer warps than the device holds, 64 on each SM (303 k
// points on 148), the vote is one more thing to wait for (30 k points 225 -> 235 us, 100 k 176 -> 178).
template <bool FILTER>
__global__ void __launch_bounds__(kKnnWarps * 32) knn_query_kernel(const float4* sorted, const unsigned* order,
                                                                   int n, KnnTree tree, float* out) {
    after_previous();
    __shared__ float s_pts[kKnnWarps][3][32];
    const int warp = blockIdx.x * kKnnWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (warp >= tree.leaf.count) return;
    float (*pts)[32] = s_pts[threadIdx.x >> 5];
    const int self = warp * 32 + lane;
    const bool live = self < n;
    const float4 q = sorted[self];
    // the box of the queries
    float qlo[3] = {live ? q.x : INFINITY, live ? q.y : INFINITY, live ? q.z : INFINITY};
    float qhi[3] = {live ? q.x : -INFINITY, live ? q.y : -INFINITY, live ? q.z : -INFINITY};
    warp_box(qlo, qhi);
    float best0 = FLT_MAX, best1 = FLT_MAX, best2 = FLT_MAX;             // the three smallest, ascending
    float worst = FLT_MAX;                                               // largest best2 of the warp
    auto keep = [&](float2 d) {                                          // the three smallest of those and two more
        const float lo = fminf(d.x, d.y), hi = fmaxf(d.x, d.y);
        const float second = fminf(fminf(fmaxf(best0, lo), best1), hi), third = fminf(fminf(best2, fmaxf(best1, lo)), fmaxf(best0, hi));
        best0 = fminf(best0, lo);
        best1 = second;
        best2 = third;
    };
    auto dist2 = [&](int k, bool own, const float (*pts)[32]) {          // to points k and k + 1 in packed fp32x2 arithmetic, same bits
        const float2 dx = __fadd2_rn(*reinterpret_cast<const float2*>(&pts[0][k]), make_float2(-q.x, -q.x)),
                     dy = __fadd2_rn(*reinterpret_cast<const float2*>(&pts[1][k]), make_float2(-q.y, -q.y)),
                     dz = __fadd2_rn(*reinterpret_cast<const float2*>(&pts[2][k]), make_float2(-q.z, -q.z));
        float2 d = __fadd2_rn(__fadd2_rn(__fmul2_rn(dx, dx), __fmul2_rn(dy, dy)), __fmul2_rn(dz, dz));   // +inf for the padding points
        if (own && k == lane) d.x = INFINITY;
        if (own && k + 1 == lane) d.y = INFINITY;
        return d;
    };
    auto open_box = [&](int b, bool own) {
        const float4 mine = sorted[b * 32 + lane];
        __syncwarp();
        pts[0][lane] = mine.x; pts[1][lane] = mine.y; pts[2][lane] = mine.z;
        __syncwarp();
        constexpr int kPairs = FILTER ? 4 : 1;
#pragma unroll(FILTER ? 1 : 4)
        for (int k = 0; k < 32; k += 2 * kPairs) {
            float2 d[kPairs];
            float least = INFINITY;
#pragma unroll
            for (int i = 0; i < kPairs; ++i) {
                d[i] = dist2(k + 2 * i, own, pts);
                least = fminf(fminf(d[i].x, d[i].y), least);
            }
            if (FILTER && !__any_sync(kAll, least < best2)) continue;
#pragma unroll
            for (int i = 0; i < kPairs; ++i) keep(d[i]);
        }
    };
    auto settle = [&]() { worst = __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(live ? best2 : 0.f))); };
    // nodes [base, base + 32) of a level that may hold something near enough for some query of the warp
    auto near = [&](const KnnLevel& level, int base) -> unsigned {
        const int b = base + lane;
        bool ok = false;
        if (b < level.count) {
            const float4 lo = level.lo[b], hi = level.hi[b];
            const float dx = fmaxf(fmaxf(lo.x - qhi[0], qlo[0] - hi.x), 0.f), dy = fmaxf(fmaxf(lo.y - qhi[1], qlo[1] - hi.y), 0.f),
                        dz = fmaxf(fmaxf(lo.z - qhi[2], qlo[2] - hi.z), 0.f);
            ok = dx * dx + dy * dy + dz * dz <= worst;
        }
        return __ballot_sync(kAll, ok);
    };
    // seed: the warp's own box and its neighbours along the curve
    open_box(warp, true);
    if (warp > 0) open_box(warp - 1, false);
    if (warp + 1 < tree.leaf.count) open_box(warp + 1, false);
    settle();
    for (int t0 = 0; t0 < tree.top.count; t0 += 32)
        for (unsigned mt = near(tree.top, t0); mt; mt &= mt - 1) {
            const int t = t0 + __ffs(mt) - 1;
            for (unsigned mm = near(tree.mid, t * 32); mm; mm &= mm - 1) {
                const int m = t * 32 + __ffs(mm) - 1;
                for (unsigned ml = near(tree.leaf, m * 32); ml; ml &= ml - 1) {
                    const int b = m * 32 + __ffs(ml) - 1;
                    if (b >= warp - 1 && b <= warp + 1) continue;        // seeded above
                    if (!__any_sync(kAll, live && box_dist2(tree.leaf.lo[b], tree.leaf.hi[b], q) <= best2)) continue;
                    open_box(b, false);
                    settle();
                }
            }
        }
    if (live) out[order[self]] = (best0 + best1 + best2) / 3.0f;         // simple_knn.cu: mean of the three
}

// The scratch of a call, carved out of one piece of memory.
struct KnnScratch {
    unsigned *bounds, *vals_in, *vals_out;
    void *keys_in, *keys_out;          // 32 or 64 bits each, see wide_keys
    float4* sorted;
    KnnTree tree;
    unsigned char* temp;
    size_t temp_bytes, bytes;
};

template <class Key>
cudaError_t sort_keys(KnnScratch& w, int n, int bits, cudaStream_t s) {
    return cub::DeviceRadixSort::SortPairs(w.temp, w.temp_bytes, (const Key*)w.keys_in, (Key*)w.keys_out, w.vals_in, w.vals_out, n, 0,
                                           bits, s);
}
cudaError_t sort_points(KnnScratch& w, int n, cudaStream_t s) {
    return wide_keys(n) ? sort_keys<uint64_t>(w, n, 48, s) : sort_keys<uint32_t>(w, n, 30, s);
}

cudaError_t plan_scratch(int n, unsigned char* base, KnnScratch& w) {
    size_t at = 0;
    auto take = [&](size_t bytes) -> unsigned char* {
        unsigned char* p = base + at;
        at += (bytes + 255) & ~(size_t)255;
        return p;
    };
    const size_t N = (size_t)n;
    w.tree.leaf.count = (n + 31) / 32;
    w.tree.mid.count = (w.tree.leaf.count + 31) / 32;
    w.tree.top.count = (w.tree.mid.count + 31) / 32;
    w.bounds = (unsigned*)take(6 * sizeof(unsigned));
    const size_t key = wide_keys(n) ? 8 : 4;
    w.keys_in = take(key * N); w.keys_out = take(key * N);
    w.vals_in = (unsigned*)take(4 * N); w.vals_out = (unsigned*)take(4 * N);
    w.sorted = (float4*)take(sizeof(float4) * 32 * (size_t)w.tree.leaf.count);
    for (KnnLevel* l : {&w.tree.leaf, &w.tree.mid, &w.tree.top}) {
        l->lo = (float4*)take(sizeof(float4) * (size_t)l->count);
        l->hi = (float4*)take(sizeof(float4) * (size_t)l->count);
    }
    w.temp = nullptr;
    w.temp_bytes = 0;
    cudaError_t e = sort_points(w, n, (cudaStream_t)0);                   // size query
    w.temp = take(w.temp_bytes);
    w.bytes = at;
    return e;
}

cudaError_t run_knn(int device, const float* points, int n, float* out, KnnScratch& w, cudaStream_t s) {
    const int tb = 256;
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(w.bounds, 0, 6 * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    if ((e = launch_after(knn_bounds_kernel, std::min((n + tb - 1) / tb, 4 * sms), tb, 0, s, points, n, w.bounds)) != cudaSuccess) return e;
    if (wide_keys(n)) e = launch_after(knn_keys_kernel<uint64_t>, (n + tb - 1) / tb, tb, 0, s, points, n, w.bounds, (uint64_t*)w.keys_in, w.vals_in);
    else e = launch_after(knn_keys_kernel<uint32_t>, (n + tb - 1) / tb, tb, 0, s, points, n, w.bounds, (uint32_t*)w.keys_in, w.vals_in);
    if (e != cudaSuccess) return e;
    e = wide_keys(n) ? cluster_sort((const uint64_t*)w.keys_in, (uint64_t*)w.keys_out, w.vals_in, w.vals_out, n, 48, s)
                     : cluster_sort((const uint32_t*)w.keys_in, (uint32_t*)w.keys_out, w.vals_in, w.vals_out, n, 30, s);
    if (e == cudaErrorNotSupported) e = sort_points(w, n, s);
    if (e != cudaSuccess) return e;
    launch_after(knn_gather_kernel, w.tree.mid.count, 1024, 0, s, points, n, w.vals_out, w.sorted, w.tree.leaf, w.tree.mid);
    const int blocks = (w.tree.leaf.count + kKnnWarps - 1) / kKnnWarps, upper = (w.tree.top.count + 7) / 8;
    if (blocks <= 4 * sms) launch_after(knn_upper_kernel<true>, upper, 256, 0, s, w.tree.mid, w.tree.top);
    else launch_after(knn_upper_kernel<false>, upper, 256, 0, s, w.tree.mid, w.tree.top);
    if (w.tree.leaf.count > 64 * sms) launch_after(knn_query_kernel<true>, blocks, kKnnWarps * 32, 0, s, w.sorted, w.vals_out, n, w.tree, out);
    else launch_after(knn_query_kernel<false>, blocks, kKnnWarps * 32, 0, s, w.sorted, w.vals_out, n, w.tree, out);
    return cudaGetLastError();
}

}  // namespace

}  // namespace rgx

using namespace rgx;

extern "C" RGX_API size_t rgx_knn_scratch_bytes(int n) {
    KnnScratch w;
    return n > 0 && n <= (1 << 30) && plan_scratch(n, nullptr, w) == cudaSuccess ? w.bytes : 0;
}

extern "C" RGX_API int rgx_knn_mean_dist2_scratch(int device, const float* points, int n, float* mean_dist2, void* scratch,
                                                  size_t scratch_bytes, rgx_stream stream) {
    if (n < 0 || (n > 0 && (!points || !mean_dist2 || !scratch || (reinterpret_cast<uintptr_t>(scratch) & 255u)))) return RGX_E_INVALID;
    if (n > (1 << 30)) return RGX_E_TOO_LARGE;
    if (n == 0) return RGX_OK;
    DeviceGuard guard(device);
    if (!guard.ok) { (void)cudaGetLastError(); return RGX_E_CUDA; }
    KnnScratch w;
    cudaError_t e = plan_scratch(n, (unsigned char*)scratch, w);
    if (e == cudaSuccess && w.bytes > scratch_bytes) return RGX_E_INVALID;
    if (e == cudaSuccess) e = run_knn(device, points, n, mean_dist2, w, (cudaStream_t)stream);
    if (e != cudaSuccess) { (void)cudaGetLastError(); return RGX_E_CUDA; }
    return RGX_OK;
}

extern "C" RGX_API int rgx_knn_mean_dist2(int device, const float* points, int n, float* mean_dist2, rgx_stream stream) {
    if (n < 0 || (n > 0 && (!points || !mean_dist2))) return RGX_E_INVALID;
    if (n > (1 << 30)) return RGX_E_TOO_LARGE;
    if (n == 0) return RGX_OK;
    DeviceGuard guard(device);
    if (!guard.ok) { (void)cudaGetLastError(); return RGX_E_CUDA; }
    cudaStream_t s = (cudaStream_t)stream;
    void* scratch = nullptr;
    const size_t bytes = rgx_knn_scratch_bytes(n);
    cudaError_t e = bytes ? cudaMalloc(&scratch, bytes) : cudaErrorUnknown;
    if (e != cudaSuccess) { (void)cudaGetLastError(); return RGX_E_CUDA; }
    int rc = rgx_knn_mean_dist2_scratch(device, points, n, mean_dist2, scratch, bytes, stream);
    if (rc == RGX_OK && cudaStreamSynchronize(s) != cudaSuccess) { (void)cudaGetLastError(); rc = RGX_E_CUDA; }   // the scratch is freed below
    cudaFree(scratch);
    return rc;
}
