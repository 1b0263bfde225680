// Stable sort of a few thousand to some 80 thousand (key, 32-bit value) pairs by one cluster of sixteen blocks.
//
// The pairs stay in the shared memory of the cluster from the first pass to the last.  Per pass of eight bits every warp counts the
// digits of its share and numbers its pairs among those of the same digit, the counts are added up over the warps of a block
// and over the blocks, and every pair goes to its place in the blocks' other buffers.  Bound by latency (three barriers and a dozen
// rounds of votes a pass); one launch, where the library's sort takes a histogram, a scan and, per pass, a clear and a kernel, each
// with microseconds until it gets going.  30-bit / 48-bit keys, us, library and here: 4 k 14 and 21 / 74 and 31, 8 k 60 and 23, 30 k 66
// and 31 / 86 and 47, 66 k 69 and 50 / 93 and 75, 100 k 74 and 75 / 100 and 113.  (Votes on the bits of a digit: with
// __match_any_sync, which takes as long as there are digits, 30 k took 41 us.)
#pragma once
#include "rgx_internal.cuh"
#include <cooperative_groups.h>

namespace rgx {
namespace {

constexpr int kSortCluster = 16, kClusterThreads = 1024, kClusterWarps = kClusterThreads / 32, kDigits = 256;

// Pairs a block holds at most.  A call deals its pairs out in pieces of a multiple of 1,024, the last blocks get what is left or nothing;
// where the pieces grow the time does, by 4 to 12 us: builds with 30-bit / 60-bit keys of 16,384 and 16,385 Gaussians 35.2 and 41.3 / 55.6 and
// 67.9 us, of 32,768 and 32,769 43.4 and 51.6 / 76.0 and 86.3 (with the library 70.3 to 76.2 / 114 to 124).
constexpr int kClusterPiece = 5 * kClusterThreads;
// From and to how many pairs the cluster is the faster, by the width of the keys (whole calls, us, library and here).  Up to 4,864 short keys
// are one block's work for the library: builds of 4,864 Gaussians 25 and 32, distances of as many points 46 and 54, of 4,865 65 and 31, 86 and
// 54.  Long keys take six or eight passes: builds with 60-bit keys of 76,000 130 and 123, of 78,000 131 and 129, of 81,920 131 and
// 135; distances (48 bits) of 76,000 points 136 and 130, of 78,000 144 and 140, of 81,920 144 and 145.  Short keys end with the memory of the
// blocks: builds of 81,920 84 and 77.
template <class Key> constexpr int kClusterSortFrom = sizeof(Key) == 4 ? 4865 : 4097;
template <class Key> constexpr int kClusterSortTo = sizeof(Key) == 4 ? kSortCluster * kClusterPiece : 78000;
template <class Key>
size_t cluster_sort_smem(int piece) { return 2 * (size_t)piece * (sizeof(Key) + sizeof(unsigned) + 1) + sizeof(unsigned) * (kClusterWarps + 2) * kDigits; }

template <class Key>
__global__ void __launch_bounds__(kClusterThreads) cluster_sort_kernel(const Key* keys_in, Key* keys_out, const unsigned* vals_in, unsigned* vals_out,
                                                                       int n, int bits, int piece) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char cluster_sort_mem[];
    Key* key = reinterpret_cast<Key*>(cluster_sort_mem);                           // [2][piece]
    unsigned* val = reinterpret_cast<unsigned*>(key + 2 * piece);                  // [2][piece]
    unsigned* count = val + 2 * piece;                                             // [warps][digits]: pairs, then places
    unsigned* total = count + kClusterWarps * kDigits;                             // [digits] of this block, read by all
    unsigned* base = total + kDigits;                                              // [digits] place of this block's first
    unsigned short* rank = reinterpret_cast<unsigned short*>(base + kDigits);      // [piece] among the warp's pairs of the same digit
    __shared__ unsigned s_scan[kDigits / 32];
    cg::cluster_group cluster = cg::this_cluster();
    const int block = (int)cluster.block_rank(), t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int mine = min(max(n - block * piece, 0), piece), share = piece / kClusterWarps;
    const float inv_piece = 1.0f / (float)piece;
    unsigned* warp_count = count + warp * kDigits;
    for (int i = t; i < mine; i += kClusterThreads) {
        key[i] = keys_in[(size_t)block * piece + i];
        val[i] = vals_in[(size_t)block * piece + i];
    }
    const int first = warp * share, last = min(first + share, mine);
    __syncthreads();
    int from = 0;
    for (int shift = 0; shift < bits; shift += 8, from ^= 1) {
        const Key* k_at = key + from * piece;
        const unsigned* v_at = val + from * piece;
        for (int d = lane; d < kDigits; d += 32) warp_count[d] = 0u;
        __syncwarp();
        for (int i = first; i < last; i += 32) {
            const bool valid = i + lane < last;
            const unsigned d = valid ? (unsigned)(k_at[i + lane] >> shift) & (kDigits - 1u) : kDigits;
            unsigned same = __ballot_sync(0xffffffffu, valid);                     // lanes of the same digit
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const bool set = (d >> b) & 1u;
                const unsigned with = __ballot_sync(0xffffffffu, set);
                same &= set ? with : ~with;
            }
            const unsigned lower = same & ((1u << lane) - 1u), so_far = valid ? warp_count[d] : 0u;
            __syncwarp();
            if (valid) {
                rank[i + lane] = (unsigned short)(so_far + (unsigned)__popc(lower));
                if (lower == 0u) warp_count[d] = so_far + (unsigned)__popc(same);
            }
            __syncwarp();
        }
        __syncthreads();
        if (t < kDigits) {                                                         // over the warps of the block
            unsigned run = 0u;
#pragma unroll 8
            for (int w = 0; w < kClusterWarps; ++w) { const unsigned c = count[w * kDigits + t]; count[w * kDigits + t] = run; run += c; }
            total[t] = run;
        }
        cluster.sync();
        if (t < kDigits) {                                                         // over the blocks, then over the digits
            unsigned before = 0u, all = 0u;
#pragma unroll
            for (int b = 0; b < kSortCluster; ++b) {
                const unsigned c = cluster.map_shared_rank(total, b)[t];
                before += b < block ? c : 0u;
                all += c;
            }
            unsigned incl = all;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const unsigned u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
            if (lane == 31) s_scan[warp] = incl;
            base[t] = incl - all + before;
        }
        __syncthreads();
        if (t < kDigits) {
            unsigned smaller = 0u;
            for (int w = 0; w < warp; ++w) smaller += s_scan[w];
            base[t] += smaller;
        }
        __syncthreads();
        const bool done = shift + 8 >= bits;
        for (int i = first + lane; i < last; i += 32) {
            const Key k = k_at[i];
            const unsigned v = v_at[i], d = (unsigned)(k >> shift) & (kDigits - 1u), at = base[d] + warp_count[d] + rank[i];
            if (done) {
                keys_out[at] = k;
                vals_out[at] = v;
            } else {
                const unsigned b = __float2uint_rz(((float)at + 0.5f) * inv_piece), slot = at - b * (unsigned)piece;      // at / piece: at < 2^18
                cluster.map_shared_rank(key, b)[(from ^ 1) * piece + slot] = k;
                cluster.map_shared_rank(val, b)[(from ^ 1) * piece + slot] = v;
            }
        }
        cluster.sync();                          // all sent; after the last pass: no block ends while another reads its counts
    }
}

// What says that this device, or what is left of it, does not take the cluster.  Any other error is no reason to go on.
inline bool cluster_refused(cudaError_t e) {
    return e == cudaErrorInvalidClusterSize || e == cudaErrorInvalidConfiguration || e == cudaErrorInvalidValue || e == cudaErrorLaunchOutOfResources ||
           e == cudaErrorNotSupported;
}

// cudaErrorNotSupported, and nothing enqueued, where there are too few or too many pairs or the device does not take the cluster.  Clears
// that error: the caller has looked at the results of its launches before.
template <class Key>
cudaError_t cluster_sort(const Key* keys_in, Key* keys_out, const unsigned* vals_in, unsigned* vals_out, int n, int bits, cudaStream_t s) {
    if (n < kClusterSortFrom<Key> || n > kClusterSortTo<Key>) return cudaErrorNotSupported;
    const int per_block = (n + kSortCluster - 1) / kSortCluster, piece = (per_block + kClusterThreads - 1) / kClusterThreads * kClusterThreads;
    const size_t smem = cluster_sort_smem<Key>(piece);
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(cluster_sort_kernel<Key>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) == cudaSuccess &&
        (e = cudaFuncSetAttribute(cluster_sort_kernel<Key>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cluster_sort_smem<Key>(kClusterPiece))) == cudaSuccess) {
        cudaLaunchAttribute cluster = {};
        cluster.id = cudaLaunchAttributeClusterDimension;
        cluster.val.clusterDim.x = kSortCluster;
        cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
        cudaLaunchConfig_t c = {};
        c.gridDim = kSortCluster;
        c.blockDim = kClusterThreads;
        c.dynamicSmemBytes = smem;
        c.stream = s;
        c.attrs = &cluster;
        c.numAttrs = 1;
        if ((e = cudaLaunchKernelEx(&c, cluster_sort_kernel<Key>, keys_in, keys_out, vals_in, vals_out, n, bits, piece)) == cudaSuccess) note_launch();
    }
    if (!cluster_refused(e)) return e;
    (void)cudaGetLastError();
    return cudaErrorNotSupported;
}

}  // namespace
}  // namespace rgx
