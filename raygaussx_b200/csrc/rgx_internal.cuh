// Internal declarations shared by the translation units of librgx.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <float.h>
#include "../../include/rgx.h"

namespace rgx {

constexpr int kFan = 32;          // children per hierarchy node = lanes per warp
constexpr int kMaxLevels = 8;     // level 0 = Gaussians; 32^7 > 3e10 primitives
constexpr int kSlab = 32;         // samples per slab  (BUFFER_SIZE, cuda_train/forward/gaussians_aabb.h:2)
constexpr int kChunk = 16;        // samples per chunk (CHUNK_SIZE, :3)
constexpr int kMaxLobes = 8;

// Pointers that kernels read or write 16 bytes at a time (float4) must start on a 16-byte boundary.
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Makes `device` current for the duration of an entry point and puts the caller's device back afterwards.
struct DeviceGuard {
    int prev = -1, dev;
    bool ok;
    explicit DeviceGuard(int device) : dev(device) {
        if (cudaGetDevice(&prev) != cudaSuccess) { prev = -1; (void)cudaGetLastError(); }
        ok = prev == device || cudaSetDevice(device) == cudaSuccess;
    }
    ~DeviceGuard() { if (prev >= 0 && prev != dev) cudaSetDevice(prev); }
    DeviceGuard(const DeviceGuard&) = delete;
    DeviceGuard& operator=(const DeviceGuard&) = delete;
};

// Hierarchy over the Morton-sorted Gaussians.  Level 0 holds one box per Gaussian,
// node j of level l+1 bounds boxes [32j, 32j+32) of level l.  All levels live in
// one set of arrays; every level is padded to a multiple of 32 entries with
// inverted (never hit) boxes.
struct Hierarchy {
    const float2* bx;  // per box: (min, max) along x
    const float2* by;
    const float2* bz;
    int num_levels;            // including level 0
    int offset[kMaxLevels];    // first box of each level
    int count[kMaxLevels];     // valid boxes of each level (unpadded)
};

// Per-Gaussian data in sorted order (index j), n_pad = roundup(n, 32) entries.
struct SortedGaussians {
    // g0 = (p.x, p.y, p.z, m00), g1 = (m01, m02, m10, m11), g2 = (m12, m20, m21, m22)
    // with M = S^-1 R^T / k, so that the truncation ellipsoid is |M (x - p)|^2 < 1.
    const float4* g0;
    const float4* g1;
    const float4* g2;
    const float* hk;     // log2(sigma / sigma_threshold): exp(-power/2) = exp2(-hk * |M(x-p)|^2)
    const float4* rgba;  // per view: (r*sigma, g*sigma, b*sigma, sigma)
    const float4* quat;  // raw quaternion (backward)
    const float4* sdens; // (s.x, s.y, s.z, sigma) raw (backward)
    const uint32_t* perm;// sorted index -> caller's index
    int n;
    int n_pad;
};

struct DeviceCounters {   // mirrors rgx_counters
    unsigned long long v[20];
};
enum { C_RAYS, C_SLABS, C_SLABS_HIT, C_CLOSEST, C_HITS, C_PAIRS, C_OVF, C_NODE_TESTS, C_PRIM_TESTS, C_ELL_TESTS,
       C_STACK_OVF, C_HASH, C_CANDS, C_CYC_WINDOW, C_CYC_SEEK, C_CYC_SEARCH,
       C_CYC_EVAL, C_CYC_COMP, C_CYC_WAIT, C_CYC_TOTAL, C_NUM };

struct SceneBox {         // written by the build, read by the march kernels
    float lo[3];
    float hi[3];
};

// Pixels per side of a binning tile.  16 for images of ordinary size; a small image has few tiles of that size, each as wide as
// a large part of the scene and with a list as long, and walking it by the warps of a few SMs is then all the time there is.
// Forward march with tiles of 16 / 8 / 4 pixels: 600 k object at 64x64 28.0 / 0.87 / 0.86 ms, at 128x128 4.3 / 1.0 / 0.5, at
// 256x256 1.65 / 0.99 / 0.78; but smaller tiles mean more pairs, and from 256x256 on (8) and 128x128 on (4) the lists of
// scenes with large Gaussians cost more than the march gains.  Depends on the image alone, so that a row range of it meets
// its Gaussians in the same order.
inline int bin_tile_size(const rgx_camera& c) {
    const long long rays = (long long)c.width * c.height;
    return rays <= 128 * 128 ? 4 : rays <= 256 * 256 ? 8 : 16;
}
constexpr int kMaxPatchesPerTile = 64;  // patches of rays that a warp marches together: 4 rays at least (march_lists.cu)
constexpr int kTapeBlockInts = 16384;   // ints of the recording that a warp reserves at a time

// Per-view, per-tile candidate lists (binning.cu).  Tile t owns entries
// [tile_pbegin[t], tile_pbegin[t] + roundup32(tile_cnt[t])), sorted by near distance;
// padding entries have the empty range (+inf, -inf).
struct TileLists {
    const int* ent_id;         // sorted slot of the candidate
    const float2* ent_range;   // (near, far) distance of its box from the eye, conservative
    const float2* blk;         // per 32 entries: (smallest near, largest far)
    const int* tile_pbegin;
    const int* tile_cnt;
    const int* tile_order;     // tiles by falling list length: CTA b marches tile tile_order[b] (null: tile b)
    int tiles_x, tiles_y, ty_first;
    int tile;                  // pixels per side
};

// Horizon of a culled emission (binning.cu): picked on the device from a histogram of the Gaussians' nearest
// distances, read by the emission kernels of the same stream and, afterwards, by the host.
struct HorizonPick {
    unsigned int cut;                   // last histogram bucket kept; kAllBuckets: every pair is kept
    unsigned int chord_bits;            // largest chord of a tile (float bits), from bin_tile_dirs_kernel
    unsigned long long est_kept;        // estimated pairs up to the cut (tile rectangles, an upper bound)
    unsigned long long est_total;       // estimated pairs of the view
    unsigned long long reserved;
};
constexpr unsigned int kAllBuckets = 0xffffffffu;

// What an emission leaves for the host, first in the piece of memory that it starts from zero.
struct BinResult {
    unsigned long long total[6];        // [0] pairs met (may exceed the capacity); Gaussians listed for the emission: [1] of few tiles, [3] of
                                        // many; [2], [4] the next of each
    HorizonPick pick;
    unsigned int longest, long_tiles;   // pairs of the longest list; lists of more than kSortShort pairs (bin_layout_kernel)
};
constexpr int kSortShort = 2048, kSortLong = 16384;   // lists that a block sorts in shared memory (binning.cu)
// That piece, as byte offsets: the result, the histogram of nearest distances, per tile first and last pair and padded count,
// corners of culled rectangles, tiles that have more pairs.
struct ZeroedBins {
    size_t hist, first, pcnt, diff, more, bytes;     // pcnt: pairs per tile, counted by the emission
};
inline ZeroedBins zeroed_bins(int tiles_x, int tiles_y) {
    const size_t tiles = (size_t)tiles_x * tiles_y, align = 255;
    ZeroedBins z;
    z.hist = (sizeof(BinResult) + align) & ~align;
    z.first = z.hist + 2048 * sizeof(unsigned long long);
    z.pcnt = (z.first + sizeof(int) * (tiles + 1) + align) & ~align;
    z.diff = (z.pcnt + sizeof(int) * (tiles + 1) + align) & ~align;
    z.more = (z.diff + sizeof(int) * (size_t)(tiles_x + 1) * (tiles_y + 1) + align) & ~align;
    z.bytes = z.more + sizeof(int) * tiles;
    return z;
}

struct Projector {     // pixel coordinates of a world point: px = (a / (2 tan) + pp) * size - 0.5
    float eye[3], du[3], dv[3], dw[3];   // dual basis of (u, v, w)
    float sx, sy, ox, oy;                // px = a * sx + ox, py = b * sy + oy
    float plane[4][4];                   // the view's four side planes through the eye: inward normal, and its length
};

struct BinLaunch {
    Projector proj;                        // of cam, for the rows at hand
    int n, n_pad;
    const float2 *bx, *by, *bz;            // level-0 boxes
    const float4 *g0, *g1, *g2, *quat, *sdens;
    const float* hk;
    rgx_camera cam;
    float dual[3][3];                      // dual basis of (u, v, w): rows u*, v*, w*
    int row_begin, row_end, tile, tiles_x, tiles_y, ty_first;
    uint64_t *keys_in, *keys_out;          // [pair capacity] (tile, near distance, sorted slot)
    uint32_t *vals_in, *vals_out;          // [pair capacity] far distance (float bits)
    uint32_t* ranks;                       // [pair capacity] the pair's number among its tile's, in no particular order
    BinResult* result;
    BinResult* result_host;                // pinned: bin_layout_kernel, the last of the emission, leaves the result there too
    unsigned long long pair_cap;
    int *tile_first, *tile_cnt, *tile_pcnt, *tile_pbegin;   // [tiles + 1]
    int *tile_iota, *tile_cnt_sorted, *tile_order;                      // [tiles]
    int* ent_id; float2* ent_range; float2* blk;
    float4* tile_dir;                      // [tiles] central ray direction, chord to the farthest corner ray
    void* cub_temp; size_t cub_bytes;
    unsigned char* zero; size_t zero_bytes;// cleared before an emission; total_dev, pick ... tile_more point into it
    unsigned long long* total_dev;         // [6], see BinResult
    int* big_slot; uint2* big_rect;        // [n_pad] complete emission: the Gaussians that touch a tile, and their tile rectangles
    int big_grid, sm_count;                // CTAs that work the list off (a few per SM)
    // culled emission (null / unused for a complete one): only the pairs that begin before a horizon are emitted
    HorizonPick* pick;
    unsigned long long* near_hist;         // [2048] estimated pairs by nearest distance of the Gaussian
    uint2* g_rect; unsigned int* g_code;   // [n_pad] tile rectangle (x = ~0: none) and histogram bucket of every Gaussian
    int* kept_slot;                        // [n_pad] the Gaussians before the cut, in no particular order: from the front, of many tiles from the back
    int* tile_diff;                        // [(tiles_x + 1) * (tiles_y + 1)] corners of the rectangles of culled Gaussians
    int* tile_more;                        // [tiles] the tile has pairs that were not emitted
    unsigned long long near_target;        // estimated pairs to keep
    unsigned long long near_min_total;     // views with fewer estimated pairs are emitted completely ...
    int near_half;                         // ... and so are views of which the cut would keep all (0) or half or more (1)
    const int* tile_flag;                  // null, or [tiles]: pairs of unflagged tiles are not emitted
};

struct MarchLaunch {
    Hierarchy h;
    SortedGaussians g;
    TileLists lists;
    rgx_camera cam;
    rgx_march m;
    const SceneBox* box;
    DeviceCounters* counters;
    // forward outputs / backward inputs
    float* rgb;           // [R,3]; may be null when frame is given
    float* alpha;
    float* depth;
    uchar4* frame;        // [R] 8-bit colour (cuda_gui/helpers.h:45-58), or null
    const float* rgb_in;
    const float* dl_drgb;
    // "tape": what the forward met, kept for the backward (RGX_FLAG_SAVE_HITS); layout in march_lists.cu.
    int* tape;
    unsigned long long* tape_used;   // ints reserved so far
    long long tape_cap;
    long long* patch_head;           // [tiles * patches per tile] first chunk of every patch of rays, -1: nothing to replay
    unsigned char* ray_unrecorded;   // [R] the ray could not be recorded: the backward searches it again
    int* tile_unrecorded;            // per tile (of the lists): set by the forward when a ray of the tile is unrecorded
    const int* replay_order;  // backward replay: tiles in the order of the recording forward (own copy: the lists may be remade meanwhile)
    unsigned int* next_unit;  // [2] the warps of the forward and of the replay fetch their patches from it; zero before and after
    int sm_count;
    // two-depth forward (march_lists.cu, HZ variant): 0 = off, 1 = first phase (lists up to `horizon`), 2 = second
    int hz_phase;
    float horizon;
    float4* hz_state;         // [R, 2] what a ray put aside: (tbuffer, T, tenter, mode), colour and depth
    const int* tile_more;     // per tile: has pairs that begin beyond the horizon
    int* tile_resume;         // per tile: some ray stopped at the horizon
    unsigned int* hz_count;   // rays that stopped
    unsigned long long *tape_used_host, *hz_count_host;   // pinned, or null: where the counts of a finished march go
    int* hz_rays;             // hz_phase 3: their numbers, for march_forward_listed_rays_kernel
    float4* grad_rows;    // [grad_copies, n_pad, 4] float4 of accumulated moments, layout in emit_global
    int grad_copies;      // power of two
};

struct ColorLaunch {
    rgx_scene sc;
    float eye[3];
    const uint32_t* perm;  // null: identity order, write rgb_out [n,3]
    float4* rgba;          // sorted order output (when perm != null)
    float* rgb_out;
    float sigma_threshold;
    // lists that stop at a horizon (binning.cu): the Gaussians none of whose pairs were emitted keep whatever rgba holds
    const uint2* listed_rect;
    const unsigned int* listed_code;
    unsigned int listed_cut;
    unsigned char* listed_out;   // [n_pad] 1 where the Gaussian is on some list of the view (written with listed_code)
    const unsigned int* only_if; // not null: the kernel does nothing when this counter is zero
    int sm_count;                // wanted with only_if
};

struct FinalizeLaunch {
    rgx_scene sc;
    rgx_grads gr;
    float eye[3];
    const uint32_t* perm;
    float4* grad_rows;         // [grad_copies, n_pad, 4], see emit_global; the kernel leaves them cleared for the next backward
    const unsigned char* listed;   // null, or [n_pad]: the march can only have met the Gaussians marked here
    int grad_copies, n_pad;
    const float4 *quat, *sdens;   // sorted copies the march used
    const float* hk;
    int flags;
};

struct BuildLaunch {
    rgx_scene sc;
    float sigma_threshold;
    int morton_bits;
    int curve;
    int n_pad;
    // outputs
    uint64_t* keys_in; uint64_t* keys_out;
    uint32_t* vals_in; uint32_t* vals_out;
    float2 *bx, *by, *bz;
    float4 *g0, *g1, *g2, *quat, *sdens;
    float* hk;
    int* bounds;           // 12 words: largest -lo[3], hi[3] of the scene box, then of the centres, ordered (device_math.cuh); zero
                           // before and after a build, as are the refit counters
    SceneBox* box;
    unsigned int* refit_counters;
    int num_levels;
    int offset[kMaxLevels];
    int count[kMaxLevels];
    void* cub_temp; size_t cub_temp_bytes;
};

// Counts the kernels of this library that were launched by this process (rgx_kernel_launches).
void note_launch();

// Kernels that follow one another on a stream are set up while the one before still runs (programmatic dependent launch): a gap of
// one to three microseconds less between any two.  A kernel launched by launch_after begins with after_previous(): it lets the
// next one be set up, and waits until everything before it is done and visible.  What it reads may have just been written by the kernel
// before it -- the caller's points and parameters, too, by Adam -- and a load through the read-only path (__ldg, const __restrict__), or by an
// intrinsic with a cache hint, is bound to nothing and may be moved above that wait: such kernels use plain loads and the two below.  Iterations of 4 k Gaussians at 64x64 0.390 -> 0.376 ms, of 30 k at
// 399x301 0.751 -> 0.721, RGB + alpha + depth of 1 M at 640x360 1.058 -> 1.039, neighbour distances of 30 k points 0.227 -> 0.218.
//   Not for the march and the colours: blocks that are set up early live with the division between shared memory and L1 cache that
// the kernel before them asked for (colours behind the sort of the tile lists 33 -> 104 us, march of the 300 k object +3 %).
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// The other way round: the next kernel is set up only when everything before this one is done.  For a short kernel that is followed by one
// of a few blocks per SM: set up beside the kernel before last, those would all go to the SMs that it leaves free.
__device__ __forceinline__ void after_previous_then_next() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}
__device__ __forceinline__ float load_streaming(const float* p) {
    float v;
    asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ float4 load_streaming(const float4* p) {
    float4 v;
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ float2 load_from_l2(const float2* p) {
    float2 v;
    asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(__cvta_generic_to_global(p)) : "memory");
    return v;
}
template <class... Params, class... Args>
inline cudaError_t launch_after(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &early;
    c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, static_cast<Args&&>(args)...);
    if (e == cudaSuccess) note_launch();
    return e;
}

// host launchers (each returns the cudaError_t of its last launch)
cudaError_t launch_build(const BuildLaunch& b, cudaStream_t s);
size_t build_cub_temp_bytes(int n_pad);
cudaError_t launch_colors(const ColorLaunch& c, cudaStream_t s);
cudaError_t launch_finalize(const FinalizeLaunch& f, cudaStream_t s);
size_t binning_cub_temp_bytes(size_t pair_cap, int ntiles);
Projector make_projector(const BinLaunch& b);
cudaError_t launch_bin_emit(const BinLaunch& b, cudaStream_t s);
cudaError_t launch_bin_fill(const BinLaunch& b, int total, const BinResult& r, cudaStream_t s);
float bin_hist_bucket_end(const BinLaunch& b, int bucket);
cudaError_t launch_march_forward(const MarchLaunch& m, cudaStream_t s);
// The rays listed in m.hz_rays by a march over lists that stop at a horizon, again by per-ray search (march.cu); the march's counts go to
// pinned memory with it.
cudaError_t launch_march_forward_listed_rays(const MarchLaunch& m, int ctas, cudaStream_t s);
// The ints that a recording march has used, to pinned memory, where no launch of the above does it.
cudaError_t launch_report(const MarchLaunch& m, cudaStream_t s);
// The backward in two launches: rays without a recording (searches the lists or the hierarchy), then the replay of
// the recording, which reads neither lists nor hierarchy.
cudaError_t launch_march_backward_search(const MarchLaunch& m, cudaStream_t s);
cudaError_t launch_march_backward_replay(const MarchLaunch& m, cudaStream_t s);

}  // namespace rgx
