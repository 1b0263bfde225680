// Forward and backward ray march over per-view tile lists: the default path.
//
// binning.cu leaves, for every tile of the view (16x16 pixels; 8x8 or 4x4 of small images), a front-to-back list
// of the Gaussians that any ray of the tile can meet, each with the range of
// distances from the eye that its box spans, plus a (nearest near, farthest far)
// summary per 32 entries.
//
// A warp marches a patch of neighbouring pixels (4x4; less of a small image): its rays go through the list
// together.  Neighbouring rays begin and end their slabs within a fraction of a slab of each
// other and meet the same Gaussians (measured: 15 of 16 rays of a patch share a hit on
// the 3 M-Gaussian scene, 10 of 16 on the 300 k object), so a list entry is fetched,
// whitened and culled once per patch instead of once per ray, and everything a ray does by
// itself -- planning a slab, compositing, bookkeeping -- costs a lane or two of a warp
// instruction, not a whole one.  The deciding test of a hit is the per-ray one of
// march_common.cuh, so hit sets equal those of the per-ray and exhaustive variants; hits are
// met in list order (near distance, then sorted slot), the same in the forward and the backward.
//
// Reference semantics: cuda_train/forward/gaussians_aabb.cu:205-340 and
// cuda_train/backward/gaussians_aabb.cu:209-497 (see march_common.cuh).
#include "march_common.cuh"

namespace rgx {

namespace {

constexpr int kThreads = kWarps * 32;

// Shape of a patch.  P lanes carry a ray; the 32 / P rays of a warp lie in a block of W x H pixels.
template <int P>
struct Patch {
    static constexpr int kLanes = P, kRays = 32 / P;
    static constexpr int kW = P == 8 ? 2 : 4, kH = kRays / kW;
    static constexpr unsigned kRayBits = (1u << kRays) - 1u;          // the lanes of one list entry in a ballot
    static constexpr int kSamples = kSlab / P;                        // samples of a lane
    // A slab is evaluated in this many parts.  Each costs a branch per entry, 4 % of the kernel: with two lanes per ray eight parts
    // are 15 % slower than four, and two (ten samples in three evaluated for nothing more) 4 to 10 %; with four lanes, whose quarter is one
    // pair of samples, two are faster (150x140: 60 k object 0.314 -> 0.305 ms, 60 k unbounded 0.066 -> 0.061).
    static constexpr int kParts = P == 2 ? 4 : 2;
    static constexpr int kPairs = kSamples / 2, kPairsPerPart = kPairs / kParts;
    // recording, in ints: header, tbuffer and sample spacing per ray, sums, list
    static constexpr int kTapeDt = 8 + kRays, kTapeSums = 8 + 2 * kRays, kTapeList = kTapeSums + 4 * kSamples * 32;
};

constexpr int kHitList = 256;      // hits of a slab remembered between the two passes of the backward search

// Recording of the forward for the backward ("tape"), in ints, everything 16-byte aligned.  A patch has a chain of chunks,
// one per slab step in which some of its rays had hits:
//   [0] entries in this piece   [1] rays (bits) the step belongs to   [2,3] offset of the next piece of the list (-1: none)
//   [4,5] offset of the patch's next chunk (-1: last)                 [6,7] -
//   tbuffer, then sample spacing, of the patch's rays
//   the per-sample sums (sigma, r sigma, g sigma, b sigma): float4 [samples of a lane][lane]
//   list: (sorted slot, rays that hit it as bits) in the order met
// A list that outgrows the block goes on in a piece elsewhere: [0] entries, [2,3] next piece, [4, ...) list.
// 140 ints per ray and slab on the 3 M-Gaussian scene: sharing the list among the rays makes the hits nearly free.
constexpr int kTapeBlock = kTapeBlockInts;
constexpr int kTapePiece = 4;

struct ListShared {                // backward search: per warp and ray
    int next_ray;
    int pend[kWarps][2 * kFan];
    int prim_of[kWarps][kFan];
    WarpStage ws[kWarps];
};

struct TileView {      // one tile's list: entries begin, begin + 1, ... of the view's
    int begin, nblk;
};

__device__ __forceinline__ TileView tile_view(const TileLists& l, int tile) {
    return {__ldg(&l.tile_pbegin[tile]), (__ldg(&l.tile_cnt[tile]) + 31) / 32};
}
__device__ __forceinline__ int entry_id(const MarchLaunch& L, const TileView& tv, int k) { return __ldg(&L.lists.ent_id[tv.begin + k]); }
__device__ __forceinline__ float2 entry_range(const MarchLaunch& L, const TileView& tv, int k) {
    return __ldg(&L.lists.ent_range[tv.begin + k]);
}
__device__ __forceinline__ float2 block_range(const MarchLaunch& L, const TileView& tv, int b) {
    return b < tv.nblk ? __ldg(&L.lists.blk[tv.begin / 32 + b]) : make_float2(INFINITY, -INFINITY);
}

// Runs the exact test on the first min(npend, 32) pending candidates and hands them to leaf.
template <bool COUNT, class LeafFn>
__device__ __forceinline__ bool test_pending(const MarchLaunch& L, const Ray& r, float tmin, float tmax, int* pend,
                                             int& npend, int lane, Tally& tl, LeafFn&& leaf) {
    const bool valid = lane < npend;
    const int j = valid ? pend[lane] : 0;
    LeafTest t = test_gaussian(L, r, j, valid, tmin, tmax, tl, COUNT, false);
    const bool go = leaf(t, j);
    const int moved = (lane + kFan < npend) ? pend[lane + kFan] : 0;
    __syncwarp();
    pend[lane] = moved;
    npend = npend > kFan ? npend - kFan : 0;
    __syncwarp();
    return go;
}

// Any-hit query over a tile list.  `cursor` is the ray's first block that may still
// matter; it only moves forward because a ray's tmin never decreases.
template <bool COUNT, class LeafFn>
__device__ __forceinline__ void search_tile(const MarchLaunch& L, const Ray& r, float tmin, float tmax,
                                            const TileView& tv, int& cursor, int* pend, int lane, Tally& tl,
                                            LeafFn&& leaf) {
    int npend = 0;
    bool advancing = true;
    for (int b0 = cursor; b0 < tv.nblk; b0 += kFan) {
        const int bi = b0 + lane;
        const bool valid = bi < tv.nblk;
        const float2 s = block_range(L, tv, bi);
        const bool reaches = valid && s.y >= tmin;          // something in the block extends to tmin or beyond
        const bool beyond = valid && s.x > tmax;            // the block, and every later one, starts after tmax
        unsigned live = __ballot_sync(kFull, reaches && !beyond);
        const unsigned any_beyond = __ballot_sync(kFull, beyond);
        if (advancing) {
            const unsigned alive = __ballot_sync(kFull, reaches);
            if (alive == 0u) cursor = min(b0 + kFan, tv.nblk);
            else { cursor = b0 + __ffs(alive) - 1; advancing = false; }
        }
        while (live) {
            const int bb = b0 + __ffs(live) - 1;
            live &= live - 1;
            const int k = bb * kFan + lane;
            const float2 rg = entry_range(L, tv, k);
            const bool pass = rg.x <= tmax && rg.y >= tmin;
            const unsigned m = __ballot_sync(kFull, pass);
            if (pass) pend[npend + __popc(m & ((1u << lane) - 1u))] = entry_id(L, tv, k);
            npend += __popc(m);
            if (COUNT) tl.v[C_CANDS] += 32;
            __syncwarp();
            if (npend >= kFan) {
                const long long c_t = COUNT ? clock64() : 0;
                const bool go = test_pending<COUNT>(L, r, tmin, tmax, pend, npend, lane, tl, leaf);
                if (COUNT) tl.v[C_CYC_WAIT] += clock64() - c_t;       // exact tests and what the caller does with the hits
                if (!go) return;
            }
        }
        if (any_beyond) break;
    }
    while (npend > 0) {
        const long long c_t = COUNT ? clock64() : 0;
        const bool go = test_pending<COUNT>(L, r, tmin, tmax, pend, npend, lane, tl, leaf);
        if (COUNT) tl.v[C_CYC_WAIT] += clock64() - c_t;
        if (!go) return;
    }
}


// Closest hit over [tmin,tmax] in a tile list, +inf on a miss.
template <bool COUNT>
__device__ __forceinline__ float closest_in_tile(const MarchLaunch& L, const Ray& r, float tmin, float tmax,
                                                 const TileView& tv, int& cursor, int* pend, int lane, Tally& tl) {
    float best = INFINITY;
    if (COUNT) tl.v[C_CLOSEST] += 1;
    if (!(tmin <= tmax)) return best;
    int npend = 0;
    bool advancing = true, done = false;
    auto leaf = [&](const LeafTest& t, int) {
        best = fminf(best, warp_min_f(t.hit ? t.t_hit : INFINITY));
        return true;
    };
    for (int b0 = cursor; b0 < tv.nblk && !done; b0 += kFan) {
        const int bi = b0 + lane;
        const bool valid = bi < tv.nblk;
        const float2 s = block_range(L, tv, bi);
        const bool reaches = valid && s.y >= tmin;
        unsigned live = __ballot_sync(kFull, reaches && s.x <= tmax);
        const unsigned any_beyond = __ballot_sync(kFull, valid && s.x > tmax);
        if (advancing) {
            const unsigned alive = __ballot_sync(kFull, reaches);
            if (alive == 0u) cursor = min(b0 + kFan, tv.nblk);
            else { cursor = b0 + __ffs(alive) - 1; advancing = false; }
        }
        while (live) {
            const int src = __ffs(live) - 1;
            live &= live - 1;
            // entries are sorted by near distance: nothing from here on can start before `best`
            if (__shfl_sync(kFull, s.x, src) > best) { done = true; break; }
            const int k = (b0 + src) * kFan + lane;
            const float2 rg = entry_range(L, tv, k);
            const bool pass = rg.x <= fminf(tmax, best) && rg.y >= tmin;
            const unsigned m = __ballot_sync(kFull, pass);
            if (pass) pend[npend + __popc(m & ((1u << lane) - 1u))] = entry_id(L, tv, k);
            npend += __popc(m);
            if (COUNT) tl.v[C_CANDS] += 32;
            __syncwarp();
            if (npend >= kFan) test_pending<COUNT>(L, r, tmin, fminf(tmax, best), pend, npend, lane, tl, leaf);
        }
        // do not run far ahead with untested candidates: they may already hold the answer
        while (npend > 0) test_pending<COUNT>(L, r, tmin, fminf(tmax, best), pend, npend, lane, tl, leaf);
        if (any_beyond) break;
    }
    return best;
}

// pixel of the tile's ray number `ray` (row-major inside the tile)
__device__ __forceinline__ bool ray_pixel(const MarchLaunch& L, int tile_x, int tile_y, int ray, int& px, int& py) {
    px = tile_x * L.lists.tile + ray % L.lists.tile;
    py = (L.lists.ty_first + tile_y) * L.lists.tile + ray / L.lists.tile;
    return px < L.cam.width && py >= L.m.row_begin && py < L.m.row_end;
}

// A ray stops at the horizon of its lists: counted; in the counting-only variant its number is kept as well, for the
// per-ray search that finishes it (march.cu).
template <int HZ>
__device__ __forceinline__ void hz_note(const MarchLaunch& L, int ray_id) {
    const unsigned int at = atomicAdd(L.hz_count, 1u);
    if (HZ == 2) L.hz_rays[at] = ray_id;
}

// ---------------------------------------------------------------- what the sixteen rays of a patch share
constexpr int kPatchWarps = 1;     // warps per CTA of the patch kernels, see forward_ctas
constexpr int kGroup = 8;          // entries that are tested before their hits are evaluated
// The next patch.  Every warp of the grid fetches one number past the end; the one that fetches the last of those puts the counter
// back to zero for the next launch.
__device__ __forceinline__ unsigned fetch_unit(unsigned* next, unsigned units) {
    const unsigned u = atomicAdd(next, 1u);
    if (u == units + gridDim.x * (blockDim.x >> 5) - 1u) *next = 0u;
    return u;
}

constexpr int kStaged = 64;        // ring of list entries that passed the patch's filters

template <int N>
struct Staged {                    // per warp
    float4 m0[N];                  // M = S^-1 R^T / k, and the eye in the whitened frame, the first two rows side by side for
    float4 m1[N];                  // packed instructions: (m00, m10, m01, m11), (m02, m12, Oe.x, Oe.y), (m20, m21, m22, Oe.z)
    float4 m2[N];
    float4 ex[N];                  // hk, |Oe|^2 - 1, sorted slot (bits), rays that hit it (bits, set once tested)
    float4 rgba[N];                // (r sigma, g sigma, b sigma, sigma)
};
using PatchStage = Staged<kStaged>;

template <int N>
__device__ __forceinline__ unsigned& hit_by(Staged<N>& st, int q) { return reinterpret_cast<unsigned*>(&st.ex[q])[3]; }

// smallest / largest of non-negative floats over the warp (they order like their bits)
__device__ __forceinline__ float warp_min_pos(float v) { return __uint_as_float(__reduce_min_sync(kFull, __float_as_uint(v))); }
__device__ __forceinline__ float warp_max_pos(float v) { return __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(v))); }

// One Gaussian's record, as the sorted arrays hold it, into slot `q` (by one lane): what is computed from the geometry, then the rest.
template <int N>
__device__ __forceinline__ void stage_geometry(Staged<N>& st, int q, int j, float4 g0, float4 g1, float4 g2, float3 Oe) {
    st.m0[q] = make_float4(g0.w, g1.z, g1.x, g1.w);
    st.m1[q] = make_float4(g1.y, g2.x, Oe.x, Oe.y);
    st.m2[q] = make_float4(g2.y, g2.z, g2.w, Oe.z);
    st.ex[q].y = whitened_c(Oe);
    st.ex[q].z = __int_as_float(j);
}
// BYTES (4 or 16, aligned to as many) from global into shared memory, without a register on the way.
template <int BYTES>
__device__ __forceinline__ void copy_async(void* to, const void* from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ float3 whiten_eye(const MarchLaunch& L, float4 g0, float4 g1, float4 g2) {
    const float3 O = make_float3(L.cam.eye[0] - g0.x, L.cam.eye[1] - g0.y, L.cam.eye[2] - g0.z);
    float3 Oe;
    Oe.x = fmaf(g0.w, O.x, fmaf(g1.x, O.y, __fmul_rn(g1.y, O.z)));
    Oe.y = fmaf(g1.z, O.x, fmaf(g1.w, O.y, __fmul_rn(g2.x, O.z)));
    Oe.z = fmaf(g2.y, O.x, fmaf(g2.z, O.y, __fmul_rn(g2.w, O.z)));
    return Oe;
}
__device__ __forceinline__ float3 whiten_dir(float4 m0, float4 m1, float4 m2, float3 d) {
    return make_float3(fmaf(m0.x, d.x, fmaf(m0.y, d.y, __fmul_rn(m0.z, d.z))),
                       fmaf(m1.x, d.x, fmaf(m1.y, d.y, __fmul_rn(m1.z, d.z))),
                       fmaf(m2.x, d.x, fmaf(m2.y, d.y, __fmul_rn(m2.z, d.z))));
}

// whiten_dir for a staged record: the same bits, six instructions instead of nine (recording forward of four 3 M views 12.38 -> 12.29 ms, of
// the 300 k object 2.91 -> 2.87).
__device__ __forceinline__ float3 staged_dir(float4 m0, float4 m1, float4 m2, float3 d) {
    const float2 xy = __ffma2_rn(make_float2(m0.x, m0.y), make_float2(d.x, d.x), __ffma2_rn(make_float2(m0.z, m0.w), make_float2(d.y, d.y),
                                 __fmul2_rn(make_float2(m1.x, m1.y), make_float2(d.z, d.z))));
    return make_float3(xy.x, xy.y, fmaf(m2.x, d.x, fmaf(m2.y, d.y, __fmul_rn(m2.z, d.z))));
}
__device__ __forceinline__ float3 staged_eye(float4 m1, float4 m2) { return make_float3(m1.z, m1.w, m2.w); }

// No ray of the patch can meet the Gaussian at a parameter in [wlo, whi].  The rays' directions lie in the parallelogram
// mid +- e1 +- e2 (cone[0..2], the directions scaled to the middle one's projection; what the normalisation of each ray takes off only
// shortens its reach), so at parameter t <= far a ray is within far |M (e1 +- e2)| of the middle ray in the whitened frame, the longer
// of the two diagonals: the middle ray would have to come that close to the unit sphere, and do so where the rays' windows lie, give
// or take the stretch by which the rays' parameters differ from the middle one's (cone[1].w of themselves).  With a slack well above
// the rounding.  Without the last condition -- the list's ranges are those of a whole tile, grown by its angular radius -- every second
// entry tested on the 300 k object and every third on 7 M needles was met by no ray (forward 3.34 -> 3.17 ms, three frames of the
// needles 16.95 -> 14.70).  A bound of the stretch that tells E's share along the ray from that across it turns away 4 % more of the needles
// and takes as long as it saves (14.37 against 14.31 ms, the object 3.35 against 3.17: registers).
__device__ __forceinline__ bool patch_misses(const float4* cone, float4 g0, float4 g1, float4 g2, float3 Oe, float far, float wlo, float whi) {
    const float4 m0 = make_float4(g0.w, g1.x, g1.y, 0.f), m1 = make_float4(g1.z, g1.w, g2.x, 0.f), m2 = make_float4(g2.y, g2.z, g2.w, 0.f);
    const float4 c = cone[0], p = cone[1], q = cone[2];
    const float3 de = whiten_dir(m0, m1, m2, make_float3(c.x, c.y, c.z));
    const float3 dp = whiten_dir(m0, m1, m2, make_float3(p.x, p.y, p.z)), dq = whiten_dir(m0, m1, m2, make_float3(q.x, q.y, q.z));
    const float inv_a = rcp_approx(dot3(de, de)), t = -dot3(Oe, de) * inv_a;
    const float3 P = make_float3(fmaf(t, de.x, Oe.x), fmaf(t, de.y, Oe.y), fmaf(t, de.z, Oe.z));
    const float rho = fmaf(__fmul_rn(far, c.w), sqrt_approx(fmaxf(dot3(dp, dp), dot3(dq, dq))), 1.0f);
    const float room = fmaf(__fmul_rn(rho, rho), 1.0005f, 1e-5f) - dot3(P, P);
    // (no number where room is none -- a Gaussian without end may have an endless range and no width across the cone --, and then kept)
    const float h = sqrt_approx(room * inv_a) * 1.01f;
    return room < 0.0f || t - h > fmaf(p.w, whi, whi) || t + h < fmaf(-p.w, wlo, wlo);
}

// The cone of a patch: the unit direction of its middle ray with the scale of the diagonals, and the two half diagonals.
__device__ __forceinline__ void patch_cone(const rgx_camera& c, int x0, int y0, int w, int h, float4* cone) {
    float3 mid;
    make_ray_dir(c, (float)x0 + 0.5f * (float)w, (float)y0 + 0.5f * (float)h, mid);
    // a pixel to the right adds su u to the unnormalised direction, a row down adds sv v; rays reach (w - 1) / 2 and (h - 1) / 2
    // pixels from the middle.  |unnormalised direction| of the middle one and of any ray of the patch: at least the shortest of
    // the patch's, which the corner below bounds from below.
    const float su = 2.0f * c.tan_half_fov[0] / (float)c.width * 0.5f * (float)(w - 1), sv = 2.0f * c.tan_half_fov[1] / (float)c.height * 0.5f * (float)(h - 1);
    const float3 e1 = make_float3(su * c.u[0], su * c.u[1], su * c.u[2]), e2 = make_float3(sv * c.v[0], sv * c.v[1], sv * c.v[2]);
    const float a = 2.0f * (((float)x0 + 0.5f * (float)w) / (float)c.width - c.pp[0]) * c.tan_half_fov[0];
    const float b = 2.0f * (((float)y0 + 0.5f * (float)h) / (float)c.height - c.pp[1]) * c.tan_half_fov[1];
    const float3 d = make_float3(a * c.u[0] + b * c.v[0] + c.w[0], a * c.u[1] + b * c.v[1] + c.w[1], a * c.u[2] + b * c.v[2] + c.w[2]);
    const float len = sqrtf(dot3(d, d)), reach = sqrtf(dot3(e1, e1)) + sqrtf(dot3(e2, e2));
    // a ray d + e, |e| <= reach: its point at parameter t is t (d + e) / |d + e|; the middle ray passes t / |d + e| d, so the
    // distance between the two is t |e| / |d + e| <= t |e| / (len - reach)
    const float scale = reach < 0.5f * len ? 1.001f / (len - reach) : INFINITY;
    cone[0] = make_float4(mid.x, mid.y, mid.z, scale);
    // a ray's parameter t is t len / |d + e| along the middle ray
    cone[1] = make_float4(e1.x + e2.x, e1.y + e2.y, e1.z + e2.z, reach * scale + 1e-4f);
    cone[2] = make_float4(e1.x - e2.x, e1.y - e2.y, e1.z - e2.z, 0.f);
}

// Walks the entries of the list that can matter to rays whose windows lie within [wlo, whi]: 32 block summaries per step,
// the blocks that overlap, their entries filtered by range and by the patch's cone; what is left is staged, and handed to
// process(first, count) in list order, four groups or more at a time and whatever remains at the end.  `cursor`: first block that
// may still matter to a ray of the patch that has got as far as `wall`; it only moves forward.  whi may shrink while walking (closest hit).
// One loop with one place that processes: the code that follows is long, and a second copy of it did not fit the instruction
// cache beside the first (a third of all stalls on the 300 k object).  Fetching a block ahead with asynchronous copies was no
// faster: the registers it takes cost what it hides.  What the filters do not look at -- exponent scale and payload -- is copied
// straight to shared memory while the walk goes on: it waited for these loads, entry after entry, and for an entry's slot after its
// range (forward, ms: object without recording 2.45 -> 2.32, three frames of 7 M needles 12.22 -> 11.76, four 3 M views 11.57 -> 11.32;
// through registers, issued before the filters: 2.53, 12.62, 12.16).
template <bool COUNT, class Process>
__device__ __forceinline__ void walk_list(const MarchLaunch& L, const TileView& tv, const float4* cone_at, float wall, float wlo,
                                          float& whi, int& cursor, PatchStage& st, int batch, int lane, Tally& tl,
                                          Process&& process) {
    int head = 0, n = 0, b0 = cursor - kFan;
    bool advancing = true, more = true;
    unsigned live = 0u;
    float near_of = 0.f;                                              // smallest near distance of this lane's block
    while (true) {
        while (more && n < batch) {
            if (live == 0u) {
                b0 += kFan;
                if (b0 >= tv.nblk) { more = false; break; }
                const float2 s = block_range(L, tv, b0 + lane);        // (inf, -inf) past the last block
                near_of = s.x;
                live = __ballot_sync(kFull, s.y >= wlo && s.x <= whi);
                if (advancing) {
                    const unsigned alive = __ballot_sync(kFull, s.y >= wall);
                    if (alive == 0u) cursor = min(b0 + kFan, tv.nblk);
                    else { cursor = b0 + __ffs(alive) - 1; advancing = false; }
                }
                if (live == 0u) {
                    if (__any_sync(kFull, s.x > whi)) more = false;
                    continue;
                }
            }
            const int src = __ffs(live) - 1;
            live &= live - 1;
            // sorted by near: once a block begins beyond whi, nothing further on can matter
            if (__shfl_sync(kFull, near_of, src) > whi) { more = false; break; }
            const int k = (b0 + src) * kFan + lane;
            const float2 rg = entry_range(L, tv, k);
            const int j = entry_id(L, tv, k);                          // wanted or not: with the range, not after it
            bool keep = rg.x <= whi && rg.y >= wlo;
            float4 g0, g1, g2;
            float3 Oe;
            if (keep) {
                g0 = __ldg(&L.g.g0[j]); g1 = __ldg(&L.g.g1[j]); g2 = __ldg(&L.g.g2[j]);
                Oe = whiten_eye(L, g0, g1, g2);
                keep = !patch_misses(cone_at, g0, g1, g2, Oe, rg.y, wlo, whi);
            }
            const unsigned m = __ballot_sync(kFull, keep);
            if (keep) {
                const int q = (head + n + __popc(m & ((1u << lane) - 1u))) & (kStaged - 1);
                stage_geometry(st, q, j, g0, g1, g2, Oe);
                copy_async<4>(&st.ex[q].x, &L.g.hk[j]);
                copy_async<16>(&st.rgba[q], &L.g.rgba[j]);
            }
            n += __popc(m);
            if (COUNT && lane == 0) tl.v[C_CANDS] += 32;
        }
        copies_done();
        __syncwarp();
        const int take = more ? n & ~(kGroup - 1) : n;
        if (take > 0) process(head, take);
        __syncwarp();
        head = (head + take) & (kStaged - 1);
        n -= take;
        if (!more) break;
    }
}

// Where a warp stands on the tape (lane 0 writes, all lanes read).
struct TapeState {
    long long off;      // next free int of the warp's current block
    long long head;     // first chunk of the patch (-1: none yet)
    long long prev;     // latest chunk of the patch
    long long chunk;    // chunk of the current step (-1: the step is not recorded)
    long long piece;    // piece the list is being written to (the chunk itself, or a later piece)
    int left;           // ints left in the block
    int ok;             // 0: the patch cannot be recorded (no room)
    int n;              // entries in the current piece
};

template <int P>
struct PatchShared {
    static constexpr int kPatchRays = Patch<P>::kRays;
    PatchStage st;
    float4 cone[3];                   // see patch_misses
    float2 clip[kPatchRays];          // tenter, texit
    int slabs[kPatchRays];            // slabs begun so far
    float4 rec[kGroup][kPatchRays];   // what eval_forward's record is in march_common.cuh, per entry and ray (y = -1: no hit)
    float4 color[kPatchRays];      // colour and depth of the patch's rays so far
    TapeState tq;
};

// Room for `need` ints at tq.off, from the warp's block or a new one.  Lane 0 only.
__device__ __forceinline__ bool tape_room(const MarchLaunch& L, TapeState& tq, int need) {
    if (need > tq.left) {
        const unsigned long long o = atomicAdd(L.tape_used, (unsigned long long)kTapeBlock);
        if ((long long)(o + kTapeBlock) > L.tape_cap) return false;
        tq.off = (long long)o;
        tq.left = kTapeBlock;
    }
    return true;
}
__device__ __forceinline__ void put_offset(int* at, long long off) {
    *reinterpret_cast<int2*>(at) = make_int2((int)(off & 0xffffffffll), (int)(off >> 32));
}
__device__ __forceinline__ long long get_offset(int lo, int hi) { return ((long long)hi << 32) | (unsigned int)lo; }

// Appends the staged entries [first, first + count) that some ray hit to the list of the current step.
__device__ __forceinline__ void tape_append(const MarchLaunch& L, TapeState& tq, PatchStage& st, int first, int count, int lane) {
    if (tq.chunk < 0) return;
    for (int base = 0; base < count; base += 32) {
        const int q = (first + base + lane) & (kStaged - 1);
        const unsigned mask = base + lane < count ? hit_by(st, q) : 0u;
        const unsigned m = __ballot_sync(kFull, mask != 0u);
        const int n = __popc(m);
        if (n == 0) continue;
        if (lane == 0 && tq.left < 2 * n) {                          // the block is full: the list goes on elsewhere
            const long long old = tq.piece;
            L.tape[old] = tq.n;
            if (tape_room(L, tq, kTapePiece + 64)) {
                put_offset(L.tape + old + 2, tq.off);
                put_offset(L.tape + tq.off + 2, -1);
                tq.piece = tq.off;
                tq.n = 0;
                tq.off += kTapePiece;
                tq.left -= kTapePiece;
            } else {
                tq.chunk = -1;
                tq.ok = 0;
            }
        }
        __syncwarp();
        if (tq.chunk < 0) return;
        if (mask != 0u)
            reinterpret_cast<int2*>(L.tape + tq.off)[__popc(m & ((1u << lane) - 1u))] =
                make_int2(__float_as_int(st.ex[q].z), (int)mask);
        __syncwarp();
        if (lane == 0) { tq.off += 2 * n; tq.left -= 2 * n; tq.n += n; }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- forward
// One warp per patch of 32 / P rays.  Lane r + h (32 / P) belongs to ray r; the P lanes of a ray carry the same state.  While list
// entries are tested, lane group h tests entry e + h for all the rays; while hits are evaluated, lane h of a ray holds the samples
// P i + h of its slab, 32 / P samples times four sums in registers.  Hits are evaluated only in the parts of the slab that some ray's
// stretch inside the Gaussian reaches.
//   What bounds it: instruction issue (66 % of the slots on 2 M Gaussians at 628x414, 63 % on the 300 k object at 400x400; the rest
// waits on dependent chains at sixteen warps per SM; 12 warp instructions per hit, 16 before the tests were culled by the rays' windows) and, recording, the 512 bytes of sums per ray and slab.  With P = 1 the sums of a slab would be 128 registers and eight
// warps would fill an SM; P = 2 halves them at the price of one exchange per sample in the compositing.
//   Tests of a group of entries come before their evaluation, through shared memory: the loops are short (a unit of tests and the
// evaluation of both halves in one body missed the instruction cache) and the evaluation runs over entries that were hit only.
//   Slabs of the rays are taken in steps: the ray that is furthest behind leads, and every ray whose slab begins before the
// leader's ends marches with it.  The list is walked once per step over the union of the windows.
//   Measured against a warp per ray with lanes as samples (forward ms): 3 M-Gaussian view 9.3 -> 2.8, 300 k object 9.3 -> 2.6 (7.8 -> 2.3
// without recording), 7 M needles 14.6 -> 3.85 (two depths), 1 M at 640x360 1.83 -> 0.48.
//
// HZ: the two-depth variant for forward-only views whose rays end early (binning.cu).  In its first phase
// (L.hz_phase == 1) the tile lists hold only the pairs that begin before L.horizon; a ray that would need more
// -- its next slab reaches past the horizon, or a closest-hit query finds nothing before it, in a tile that has
// pairs beyond (L.tile_more) -- puts its state aside (L.hz_state), flags its tile (L.tile_resume) and stops.
// The second phase (L.hz_phase == 2) has the complete lists of the flagged tiles and takes those rays up where
// they stopped: same slabs, same hits in the same order, same image.
// L.hz_phase == 3 is the first phase without a second one, for recording forwards (training views, whose rays
// are expected to end before the horizon): a ray that would need more is counted and listed (L.hz_rays), marked as
// not recorded, and finished by march_forward_listed_rays_kernel, which the caller launches next.
// HZ = 1: the two phases (L.hz_phase 1 or 2); HZ = 2: counting only (L.hz_phase 3), nothing is put aside.
enum RayMode { kSeekFirst, kSeekNext, kInSlab, kDone };

// Packed a b + c, evaluated where it stands: left to itself the compiler lifts the sample positions of a slab, sixteen registers,
// out of the loop over its hits and spills others for them (recording forward of the 300 k object 3.66 ms, 3.34 this way).
__device__ __forceinline__ float2 fma2_in_place(float2 a, float2 b, float2 c) {
    float2 r;
    asm volatile("{ .reg .b64 a, b, c, r; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mov.b64 c, {%6, %7};"
                 " fma.rn.f32x2 r, a, b, c; mov.b64 {%0, %1}, r; }" : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

// Sample numbers plus a half of a lane's pairs with two lanes per ray (the first lane's; the other's are one more).  From constant memory,
// where an instruction takes them as an operand, and not literals (four 3 M views 13.47 -> 13.28 ms, three frames of 7 M needles
// 13.98 -> 13.73, the object 3.05 -> 3.03).
__constant__ float2 kPairAt[8] = {{0.5f, 2.5f}, {4.5f, 6.5f}, {8.5f, 10.5f}, {12.5f, 14.5f}, {16.5f, 18.5f}, {20.5f, 22.5f}, {24.5f, 26.5f}, {28.5f, 30.5f}};

// Sum of one value over the P lanes of a ray (P consecutive samples), as a balanced tree; `before`: over the lanes before this one.
template <int P>
__device__ __forceinline__ float across_ray(float x, int sub, float& before) {
    before = 0.f;
#pragma unroll
    for (int o = 1; o < P; o <<= 1) {
        const float other = __shfl_xor_sync(kFull, x, o * Patch<P>::kRays);
        if (sub & o) before = __fadd_rn(before, other);
        x = __fadd_rn(x, other);
    }
    return x;
}
// Balanced sum of the values of sixteen consecutive samples, fed P at a time (indices known at compile time): what decides
// the course of a ray is summed in the order of warp_scan in march_common.cuh, whichever way samples are dealt out to lanes.
template <int P>
struct SampleTree {
    static constexpr int kLeaves = 16 / P;
    float part[4];
    float half;                        // complete after kLeaves values, again after twice as many
    __device__ __forceinline__ void add(int i, float v) {
        int k = i % kLeaves, level = 0;
        while (k & 1) { v = __fadd_rn(part[level], v); k >>= 1; ++level; }
        if ((1 << level) == kLeaves) half = v;
        else part[level] = v;
    }
};
// CTAs of one warp per SM that a forward kernel is compiled for and launched with: 128 registers with 16.  The warps of a
// patch kernel share nothing, and in CTAs of one warp their number per SM can be chosen one by
// one; against CTAs of four warps (12 of 168 registers per SM when recording, 16 of 128 otherwise) the recording forward took 3.52
// instead of 4.09 ms on the 3 M view and 3.39 instead of 3.73 on the 300 k object.  15 warps are slower (four 3 M views 13.98 against
// 13.46 ms, the object 3.09 against 3.05), 18 of 112 registers much slower (15.25, 3.89): the sums of a slab alone are 64.
// All of that with two lanes per ray.  Four and eight, whose sums are 32 and 16 registers, have the same number; more was not tried there.
template <bool COUNT>
__host__ __device__ constexpr int forward_ctas() { return COUNT ? 4 : 16; }
// The replay, of 96 registers and 8.9 KB: 20 warps per SM.  18 are 1.5 to 3 % slower (four 3 M views 10.57 against 10.40 ms, the 300 k
// object 1.95 against 1.89), 17 another 4 % on the 3 M views, 21 (80 registers) as slow as 18.  With two lanes per ray, and taken over for
// four and eight.
constexpr int kReplayCtas = 20;

template <int P, bool COUNT, bool SAVE, int HZ>
__global__ void __launch_bounds__(kPatchWarps * 32, forward_ctas<COUNT>()) march_forward_patches_kernel(const __grid_constant__ MarchLaunch L) {
    using Pt = Patch<P>;
    __shared__ PatchShared<P> shared[kPatchWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane / Pt::kRays, r = lane % Pt::kRays;
    PatchShared<P>& sh = shared[warp];
    PatchStage& st = sh.st;
    TapeState& tq = sh.tq;
    const float eps = L.m.transmittance_eps;
    const float sub_half = (float)sub + 0.5f;
    const int cap = L.m.max_prim_slice;
    const unsigned per_row = (unsigned)(L.lists.tile / Pt::kW), per_tile = per_row * (unsigned)(L.lists.tile / Pt::kH);
    const unsigned units = (unsigned)(L.lists.tiles_x * L.lists.tiles_y) * per_tile;
    Tally tl;
#pragma unroll
    for (int i = 0; i < C_NUM; ++i) tl.v[i] = 0;
    if (SAVE && lane == 0) { tq.off = 0; tq.left = 0; }

    while (true) {
        unsigned unit = 0;
        if (lane == 0) unit = fetch_unit(L.next_unit, units);
        unit = __shfl_sync(kFull, unit, 0);
        if (unit >= units) break;
        const int tile = __ldg(&L.lists.tile_order[unit / per_tile]), patch = (int)(unit % per_tile);   // longest lists first
        if (HZ == 1 && L.hz_phase == 2 && !L.tile_resume[tile]) continue;    // no ray of this tile stopped at the horizon
        const int x0 = (tile % L.lists.tiles_x) * L.lists.tile + (patch % (int)per_row) * Pt::kW;
        const int y0 = (L.lists.ty_first + tile / L.lists.tiles_x) * L.lists.tile + (patch / (int)per_row) * Pt::kH;
        if (x0 >= L.cam.width || y0 >= L.m.row_end || y0 + Pt::kH <= L.m.row_begin) continue;
        // the tile has pairs beyond the horizon that its lists do not hold
        const bool hz_more = HZ != 0 && (HZ == 2 || L.hz_phase == 1) && L.tile_more[tile] != 0;
        const int px = x0 + r % Pt::kW, py = y0 + r / Pt::kW;
        const bool in_image = px < L.cam.width && py >= L.m.row_begin && py < L.m.row_end;
        const int ray_id = py * L.cam.width + px;
        const TileView tv = tile_view(L.lists, tile);
        float3 dir;
        float t;                           // where the ray stands: start of its next slab, or of its next query
        {
            Ray ray;
            float tenter, texit;
            make_ray(L.cam, px, py, ray);                                    // rays outside the image or the rows stay idle
            clip_scene(*L.box, ray, tenter, texit);
            dir = ray.d;
            t = tenter;
            // what a ray needs now and then lives in shared memory: its registers are wanted by the sums of the slab
            if (lane == 0) patch_cone(L.cam, x0, y0, Pt::kW, Pt::kH, sh.cone);
            if (sub == 0) {
                sh.clip[r] = make_float2(tenter, texit);
                sh.color[r] = make_float4(0.f, 0.f, 0.f, 0.f);
                sh.slabs[r] = 0;
            }
        }
        int mode = in_image ? kSeekFirst : kDone;
        float T = 1.0f;
        bool suspended = false;
        int cursor = 0;
        if (HZ == 1 && L.hz_phase == 2 && in_image) {
            // what was put aside is (t, T, tenter, mode) + colour; mode 1: at a slab, 2: before the first query, 3: at a query
            // after an empty slab, 0: finished
            const float4 a = L.hz_state[2 * (size_t)ray_id];
            const int was = (int)a.w;
            if (was == 0) { mode = kDone; suspended = true; }                // nothing to do, nothing to write
            else if (was != 2) {
                mode = was == 1 ? kInSlab : kSeekNext;
                t = a.x; T = a.y;
                if (sub == 0) sh.clip[r].x = a.z;
                if (sub == 0) sh.color[r] = L.hz_state[2 * (size_t)ray_id + 1];
            }
        }
        if (SAVE && lane == 0) { tq.head = -1; tq.prev = -1; tq.chunk = -1; tq.ok = 1; }
        if (COUNT && in_image && sub == 0) tl.v[C_RAYS] += 1;
        __syncwarp();
        const long long c_patch = COUNT ? clock64() : 0;
        // a ray that would need pairs from beyond the horizon: put aside (HZ = 1, first phase), counted and listed
        auto suspend = [&](float at, float how) {
            suspended = true;
            mode = kDone;
            if (sub == 0) {
                if (HZ == 1 && L.hz_phase == 1) {
                    L.hz_state[2 * (size_t)ray_id] = make_float4(at, T, sh.clip[r].x, how);
                    L.hz_state[2 * (size_t)ray_id + 1] = sh.color[r];
                    L.tile_resume[tile] = 1;
                }
                hz_note<HZ>(L, ray_id);
            }
        };

        while (__any_sync(kFull, mode != kDone)) {
            const float wall = warp_min_pos(mode != kDone ? t : INFINITY);
            // ---- closest-hit queries (:249-260, :297-319)
            if (__any_sync(kFull, mode == kSeekFirst || mode == kSeekNext)) {
                const long long c_t = COUNT ? clock64() : 0;
                const bool seeking = mode == kSeekFirst || mode == kSeekNext;
                if (COUNT && seeking && sub == 0) tl.v[C_CLOSEST] += 1;
                const float from = seeking ? t : INFINITY, texit = sh.clip[r].y;
                float best = seeking && t <= texit ? texit : -INFINITY;     // nothing from here on can matter
                bool found = false;
                float whi = warp_max_pos(fmaxf(best, 0.0f));
                walk_list<COUNT>(L, tv, sh.cone, wall, warp_min_pos(from), whi, cursor, st, kGroup, lane, tl, [&](int first, int count) {
#pragma unroll 1
                    for (int e = 0; e < count; e += P) {
                        const int q = (first + e + sub) & (kStaged - 1);
                        const float4 m0 = st.m0[q], m1 = st.m1[q], m2 = st.m2[q];
                        RayParabola pb;
                        const float3 Oe = staged_eye(m1, m2), de = staged_dir(m0, m1, m2, dir);
                        // no branch: a miss's root is whatever it is (three frames of 7 M needles 11.54 -> 11.50 ms, four 3 M views 11.17 -> 11.14)
                        const bool meets = ellipsoid_stretch(Oe, de, pb) & (e + sub < count) & (from <= best) & stretch_meets(pb, from, best);
                        const float at = fmaxf(from, entry_root(Oe, de, st.ex[q].y, pb));
                        const bool nearer = meets & (at <= best);
                        best = nearer ? at : best;
                        found |= nearer;
                        if (COUNT && seeking && e + sub < count) { tl.v[C_PRIM_TESTS] += 1; tl.v[C_ELL_TESTS] += 1; }
                    }
                    whi = warp_max_pos(fmaxf(best, 0.0f));                  // each lane prunes by what it has found itself
                });
                if (!found) best = INFINITY;
                for (int o = Pt::kRays; o < 32; o <<= 1) best = fminf(best, __shfl_xor_sync(kFull, best, o));
                if (seeking) {
                    if (HZ && hz_more && !(best < L.horizon)) {                      // nothing before the horizon: ask again later
                        suspend(t, mode == kSeekFirst ? 2.0f : 3.0f);
                    } else if (mode == kSeekFirst) {
                        if (best < INFINITY && best < texit) { t = best; if (sub == 0) sh.clip[r].x = best; mode = kInSlab; }
                        else mode = kDone;
                    } else {
                        if (best < INFINITY) { t = best; mode = kInSlab; }
                        else mode = kDone;
                    }
                }
                if (COUNT && lane == 0) tl.v[C_CYC_SEEK] += clock64() - c_t;
            }
            __syncwarp();
            const float2 clip = sh.clip[r];
            if (mode == kInSlab && !(t < clip.y && T > eps && sh.slabs[r] < kMaxSlabs)) mode = kDone;   // :266

            // ---- one slab of every ray that is near the one furthest behind
            SlabPlan p = plan_slab(L.m, t, T, clip.x, clip.y);
            const bool ready = mode == kInSlab;
            const float lead = warp_min_pos(ready ? t : INFINITY);
            const float lead_end = warp_min_pos(ready && t == lead ? p.tmax : INFINITY);
            bool act = ready && (t < lead_end || t == lead);
            if (HZ && hz_more && act && !(p.tmax < L.horizon)) { suspend(t, 1.0f); act = false; }   // this slab needs pairs from beyond
            if (act) {
                if (COUNT && sub == 0) tl.v[C_SLABS] += 1;
                if (sub == 0) sh.slabs[r] += 1;
                if (!p.traced) { t = __fadd_rn(t, p.slab); act = false; }
            }
            if (!__any_sync(kFull, act)) continue;
            const long long c_q = COUNT ? clock64() : 0;
            const float tmin = act ? p.tmin : INFINITY, tmax = act ? p.tmax : -INFINITY;
            const float dt = p.dt, sub_dt = sub ? dt : 0.f, inv_part = quotient((float)Pt::kParts / (float)kSlab, p.dt);
            float2 S[Pt::kPairs], R[Pt::kPairs], G[Pt::kPairs], B[Pt::kPairs];
#pragma unroll
            for (int i = 0; i < Pt::kPairs; ++i) S[i] = R[i] = G[i] = B[i] = make_float2(0.f, 0.f);
            int nhit = 0, most = 0;                     // hits of this ray that this lane found; bound on the hits of any ray of the patch
            bool overflow = false;
            if (SAVE) {
                if (lane == 0 && tq.ok) {
                    if (tape_room(L, tq, Pt::kTapeList + 64)) {
                        tq.chunk = tq.piece = tq.off;
                        tq.n = 0;
                        tq.off += Pt::kTapeList;
                        tq.left -= Pt::kTapeList;
                        put_offset(L.tape + tq.chunk + 2, -1);
                        put_offset(L.tape + tq.chunk + 4, -1);
                    } else {
                        tq.chunk = -1;
                        tq.ok = 0;                     // no room: the backward will search these rays
                    }
                }
                __syncwarp();
            }
            float whi = warp_max_pos(fmaxf(tmax, 0.0f));
            walk_list<COUNT>(L, tv, sh.cone, wall, warp_min_pos(tmin), whi, cursor, st, 4 * kGroup, lane, tl, [&](int first, int count) {
#pragma unroll 1
                for (int base = 0; base < count; base += kGroup) {
                    const int f = (first + base) & (kStaged - 1), n = min(count - base, kGroup), nhit0 = nhit;   // a group does not wrap around the ring
                    // test: lane group h of the warp takes entry e + h
                    unsigned reach = 0u;               // kParts bits per entry: parts of the slab that some ray's stretch inside reaches
#pragma unroll 1
                    for (int e = 0; e < n; e += P) {
                        const int q = f + e + sub;
                        const float4 m0 = st.m0[q], m1 = st.m1[q], m2 = st.m2[q];
                        RayParabola pb;
                        bool hit = ellipsoid_stretch(staged_eye(m1, m2), staged_dir(m0, m1, m2, dir), pb);
                        hit = hit & (e + sub < n) & stretch_meets(pb, tmin, tmax);
                        if (COUNT && act && e + sub < n) { tl.v[C_PRIM_TESTS] += 1; tl.v[C_ELL_TESTS] += 1; }
                        const unsigned m = __ballot_sync(kFull, hit);
                        nhit += hit ? 1 : 0;
                        // by all lanes alike: a branch around the store, as any in this loop, costs 4 % of the kernel
                        if (SAVE || COUNT) hit_by(st, q) = (m >> (Pt::kRays * sub)) & Pt::kRayBits;
                        float4 A = parabola_record(pb, t, st.ex[q].x);
                        // parts of the slab that the ray's stretch inside reaches, with a fiftieth of one on either side against
                        // rounding (the test of each sample decides)
                        const float begin = fmaxf(fmaf(A.x - pb.hw, inv_part, -0.5f * Pt::kParts / kSlab - 0.02f), 0.f);
                        const float end = fminf(fmaf(A.x + pb.hw, inv_part, -0.5f * Pt::kParts / kSlab + 0.02f), (float)Pt::kParts - 1e-6f);
                        // their whole numbers are the last bits of the sums with 2^23, rounded down (a shift takes the last five): with conversions
                        // and short-circuit logic in place of this and of `hit` above the object took 2.67 ms instead of 2.58, four 3 M views 11.32
                        // instead of 11.19
                        const unsigned lo = __float_as_uint(__fadd_rd(begin, 8388608.0f)), hi = __float_as_uint(__fadd_rd(end, 8388608.0f));
                        const unsigned groups = hit && begin <= end ? (2u << (hi & 31u)) - (1u << (lo & 31u)) : 0u;
                        if (!hit) A.y = -1.0f;
                        sh.rec[e + sub][r] = A;
                        reach |= __reduce_or_sync(kFull, groups << (Pt::kParts * sub)) << (Pt::kParts * e);
                    }
                    __syncwarp();
                    most += n;
                    if (most > cap) {                   // cuda_train/forward/gaussians_aabb.cu:352-356: hits past the cap are dropped
                        int seen = nhit0;
                        for (int o = Pt::kRays; o < 32; o <<= 1) seen += __shfl_xor_sync(kFull, seen, o);
                        for (int e = 0; e < n; ++e) {
                            const int q = f + e;
                            bool hit = sh.rec[e][r].y != -1.0f;
                            __syncwarp();
                            if (hit && seen >= cap) { hit = false; overflow = true; if (sub == 0) sh.rec[e][r].y = -1.0f; }
                            seen += hit ? 1 : 0;
                            const unsigned m = __ballot_sync(kFull, hit) & Pt::kRayBits;
                            if (lane == 0) hit_by(st, q) = m;
                            __syncwarp();
                        }
                        nhit = sub == 0 ? seen : 0;
                    }
                    if (COUNT)
                        for (int e = 0; e < n; ++e) {
                            const int q = f + e;
                            if (sub == 0 && ((hit_by(st, q) >> r) & 1u))
                                tl.v[C_HASH] += mix64(((unsigned long long)ray_id << 40) ^ ((unsigned long long)sh.slabs[r] << 24) ^
                                                      (unsigned long long)__ldg(&L.g.perm[__float_as_int(st.ex[q].z)]));
                        }
                    // Evaluate, entry after entry: to pick those that reach something out of the bits costs more than to pass by the
                    // others (four 3 M views 12.17 -> 11.72 ms, three frames of 7 M needles 12.83 -> 12.30, the object 2.81 -> 2.79).
                    // The records of the next entry fetched ahead: 12.57 and 13.09, registers.
                    const float4 *rec = &sh.rec[0][r], *payload = &st.rgba[f];
#pragma unroll 1
                    for (; reach; reach >>= Pt::kParts, rec += Pt::kRays, ++payload) {
                        const float4 A = *rec, c = *payload;
#pragma unroll
                        for (int g = 0; g < Pt::kParts; ++g) {
                            if (!((reach >> g) & 1u)) continue;
#pragma unroll
                            for (int i = Pt::kPairsPerPart * g; i < Pt::kPairsPerPart * (g + 1); ++i) {
                                // (s + 1/2) dt rounded once, as in eval_forward: with two lanes per ray sub dt is exact
                                const float2 tau = P == 2 ? fma2_in_place(kPairAt[i], make_float2(dt, dt), make_float2(sub_dt, sub_dt))
                                                          : __fmul2_rn(make_float2((float)(2 * P * i) + sub_half, (float)(2 * P * i + P) + sub_half), make_float2(dt, dt));
                                const float2 d = __fadd2_rn(tau, make_float2(-A.x, -A.x));
                                const float2 d2 = __fmul2_rn(d, d);
                                const float2 arg = __ffma2_rn(make_float2(A.z, A.z), d2, make_float2(A.w, A.w));
                                const float2 ee = make_float2(d2.x < A.y ? ex2_approx(arg.x) : 0.0f, d2.y < A.y ? ex2_approx(arg.y) : 0.0f);
                                R[i] = __ffma2_rn(make_float2(c.x, c.x), ee, R[i]);
                                G[i] = __ffma2_rn(make_float2(c.y, c.y), ee, G[i]);
                                B[i] = __ffma2_rn(make_float2(c.z, c.z), ee, B[i]);
                                S[i] = __ffma2_rn(make_float2(c.w, c.w), ee, S[i]);
                                if (COUNT) tl.v[C_PAIRS] += (d2.x < A.y ? 1 : 0) + (d2.y < A.y ? 1 : 0);
                            }
                        }
                    }
                    __syncwarp();
                }
                if (SAVE) tape_append(L, tq, st, first, count, lane);
            });
            for (int o = Pt::kRays; o < 32; o <<= 1) nhit += __shfl_xor_sync(kFull, nhit, o);
            const bool hits = act && nhit > 0;
            if (COUNT) {
                if (lane == 0) tl.v[C_CYC_SEARCH] += clock64() - c_q;
                if (act && sub == 0) { tl.v[C_HITS] += nhit; tl.v[C_OVF] += overflow ? 1 : 0; tl.v[C_SLABS_HIT] += hits ? 1 : 0; }
            }
            const unsigned with_hits = __ballot_sync(kFull, hits) & Pt::kRayBits;
            if (SAVE && with_hits && tq.chunk >= 0) {
                int* chunk = L.tape + tq.chunk;
                if (lane == 0) {
                    L.tape[tq.piece] = tq.n;
                    chunk[1] = (int)with_hits;
                    if (tq.prev >= 0) put_offset(L.tape + tq.prev + 4, tq.chunk);
                    if (tq.head < 0) tq.head = tq.chunk;
                    tq.prev = tq.chunk;
                    const int pad = (int)(-tq.off & 3);                  // the next chunk starts on 16 bytes again
                    tq.off += pad;
                    tq.left -= pad;
                }
                if (lane < 2 * Pt::kRays) chunk[8 + lane] = __float_as_int(sub == 0 ? t : dt);
                float4* sums = reinterpret_cast<float4*>(chunk + Pt::kTapeSums) + lane;
#pragma unroll
                for (int i = 0; i < Pt::kPairs; ++i) {
                    __stcs(sums + 64 * i, make_float4(S[i].x, R[i].x, G[i].x, B[i].x));
                    __stcs(sums + 64 * i + 32, make_float4(S[i].y, R[i].y, G[i].y, B[i].y));
                }
                __syncwarp();
            } else if (SAVE && !with_hits && tq.chunk >= 0) {
                __syncwarp();
                if (lane == 0) { tq.off -= Pt::kTapeList; tq.left += Pt::kTapeList; tq.chunk = -1; }    // nothing met: the room is handed back
                __syncwarp();
            }
            // ---- compositing (march_common.cuh, composite_forward): transmittance before sample s = T exp(-sum of the x before it);
            // what decides the ray's course -- T after 16 and after 32 samples -- is summed in the same order there and here
            if (with_hits) {
                const long long c_c = COUNT ? clock64() : 0;
                float run = 0.f, cr = 0.f, cg = 0.f, cb = 0.f, cd = 0.f, T16 = T, x16 = 0.f;
                bool live = true;
                SampleTree<P> tree;
#pragma unroll
                for (int i = 0; i < Pt::kPairs; ++i) {                   // two samples of the lane at a time, in packed instructions
                    const float2 dt2 = make_float2(dt, dt), log2e = make_float2(-1.4426950408889634f, -1.4426950408889634f);
                    const float2 x = __fmul2_rn(S[i], dt2), wx = __fmul2_rn(x, log2e);
                    if (i == Pt::kPairs / 2) {
                        x16 = tree.half;
                        T16 = __fmul_rn(T, exp_neg(x16));
                        live = T16 > eps;                                // :190-201: the second chunk only counts while T is above the threshold
                    }
                    float2 before, excl;
                    const float all0 = across_ray<P>(x.x, sub, before.x), all1 = across_ray<P>(x.y, sub, before.y);
                    excl.x = __fadd_rn(run, before.x);
                    run = __fadd_rn(run, all0);
                    excl.y = __fadd_rn(run, before.y);
                    run = __fadd_rn(run, all1);
                    tree.add(2 * i, all0);
                    tree.add(2 * i + 1, all1);
                    const float2 one_m_w = __fadd2_rn(make_float2(1.0f, 1.0f), make_float2(-ex2_approx(wx.x), -ex2_approx(wx.y)));
                    const float2 tx = __fmul2_rn(excl, log2e);
                    const float T_live = live ? T : 0.f;
                    const float2 Ts = __fmul2_rn(make_float2(T_live, T_live), make_float2(ex2_approx(tx.x), ex2_approx(tx.y)));
                    const float2 per_x = __fmul2_rn(one_m_w, make_float2(rcp_approx(fmaxf(x.x, 1e-6f)), rcp_approx(fmaxf(x.y, 1e-6f))));
                    const float2 f = __fmul2_rn(Ts, __fmul2_rn(dt2, per_x));
                    cr = fmaf(f.y, R[i].y, fmaf(f.x, R[i].x, cr));
                    cg = fmaf(f.y, G[i].y, fmaf(f.x, G[i].x, cg));
                    cb = fmaf(f.y, B[i].y, fmaf(f.x, B[i].x, cb));
                    if (L.depth) {
                        const float2 lost = __fmul2_rn(Ts, one_m_w);
                        cd = fmaf(lost.x, __fadd_rn(t, __fmul_rn((float)(2 * P * i) + sub_half, dt)), cd);
                        cd = fmaf(lost.y, __fadd_rn(t, __fmul_rn((float)(2 * P * i + P) + sub_half, dt)), cd);
                    }
                }
                for (int o = Pt::kRays; o < 32; o <<= 1) {
                    cr = __fadd_rn(cr, __shfl_xor_sync(kFull, cr, o));
                    cg = __fadd_rn(cg, __shfl_xor_sync(kFull, cg, o));
                    cb = __fadd_rn(cb, __shfl_xor_sync(kFull, cb, o));
                    if (L.depth) cd = __fadd_rn(cd, __shfl_xor_sync(kFull, cd, o));
                }
                if (hits) {
                    if (sub == 0) {
                        const float4 a = sh.color[r];
                        sh.color[r] = make_float4(__fadd_rn(a.x, cr), __fadd_rn(a.y, cg), __fadd_rn(a.z, cb), __fadd_rn(a.w, cd));
                    }
                    T = live ? __fmul_rn(T, exp_neg(__fadd_rn(x16, tree.half))) : T16;
                }
                if (COUNT && lane == 0) tl.v[C_CYC_COMP] += clock64() - c_c;
            }
            if (act) {
                t = __fadd_rn(t, p.slab);                                // :324
                if (!hits) mode = kSeekNext;                             // :297-319
            }
        }
        __syncwarp();
        if (in_image && sub == 0) {                                     // :326-339
            if (!suspended) {
                const float4 acc = sh.color[r];
                const RayColor out = {T, acc.x, acc.y, acc.z, acc.w};
                write_ray(L, ray_id, out, L.m.white_background ? 1.0f : 0.0f);
                if (HZ == 1 && L.hz_phase == 1) L.hz_state[2 * (size_t)ray_id] = make_float4(0.f, 0.f, 0.f, 0.f);   // done
            }
            if (SAVE) {
                const bool unrecorded = !tq.ok || (HZ == 2 && suspended);   // the backward searches this ray again
                L.ray_unrecorded[ray_id] = unrecorded ? 1 : 0;
                if (unrecorded) L.tile_unrecorded[tile] = 1;
            }
        }
        if (SAVE && lane == 0) L.patch_head[tile * (int)per_tile + patch] = tq.ok ? tq.head : -1;
        __syncwarp();
        if (COUNT && lane == 0) tl.v[C_CYC_TOTAL] += clock64() - c_patch;
    }
    if (COUNT) {
#pragma unroll
        for (int i = 0; i < C_NUM; ++i)
            if (tl.v[i]) atomicAdd(&L.counters->v[i], tl.v[i]);
    }
}

// ---------------------------------------------------------------- backward, by replaying the forward's recording
//
// For rays whose forward was recorded.  Per slab step the recording holds the per-sample sums of the patch's rays and the list of
// Gaussians they hit, so what is left is the second pass of the reference's backward
// (cuda_train/backward/gaussians_aabb.cu:354-470): the gradient of every (slab, Gaussian) pair.
// One warp per patch.  First the step's per-sample terms beta and gamma, P lanes per ray as in the forward (same arithmetic:
// T comes out bit for bit), into shared memory.  Then the listed Gaussians, P at a time: lane group h takes entry e + h for the
// patch's rays; a lane walks the samples that lie inside that Gaussian on its ray (a handful of the 32) and keeps the four
// moment sums in registers.  The thirteen sums of the Gaussian's gradient row are then added up over the rays in shared memory and
// leave the SM as one coalesced reduction of 52 bytes, where a reduction per ray and hit kept the L2 and the L1 data pipe busy.
// Bound by instruction issue (76 % of the slots) and the FMA pipe.  Against a warp per ray: 3 M-Gaussian view 7.7 -> 2.55 ms, 300 k object 4.7 -> 1.87 ms.
template <int P>
struct ReplayShared {
    Staged<kFan> st;
    float2 bg[kSlab + kRun - 1][Patch<P>::kRays];  // beta, gamma of every sample; zero past the last, where a run may end
    float red[13][36];             // one row per component, 32 lanes (+4: rows start in other banks)
};

template <int P>
__global__ void __launch_bounds__(kPatchWarps * 32, kReplayCtas) march_backward_patches_kernel(const __grid_constant__ MarchLaunch L) {
    using Pt = Patch<P>;
    __shared__ ReplayShared<P> sh;
    const int lane = threadIdx.x, sub = lane / Pt::kRays, r = lane % Pt::kRays;
    Staged<kFan>& st = sh.st;
    const float eps = L.m.transmittance_eps;
    const unsigned per_row = (unsigned)(L.lists.tile / Pt::kW), per_tile = per_row * (unsigned)(L.lists.tile / Pt::kH);
    const unsigned units = (unsigned)(L.lists.tiles_x * L.lists.tiles_y) * per_tile;
    for (int i = lane; i < (kRun - 1) * Pt::kRays; i += 32) (&sh.bg[kSlab][0])[i] = make_float2(0.f, 0.f);

    while (true) {
        unsigned unit = 0;
        if (lane == 0) unit = fetch_unit(L.next_unit + 1, units);
        unit = __shfl_sync(kFull, unit, 0);
        if (unit >= units) break;
        const int tile = __ldg(&L.replay_order[unit / per_tile]), patch = (int)(unit % per_tile);
        const int x0 = (tile % L.lists.tiles_x) * L.lists.tile + (patch % (int)per_row) * Pt::kW;
        const int y0 = (L.lists.ty_first + tile / L.lists.tiles_x) * L.lists.tile + (patch / (int)per_row) * Pt::kH;
        if (x0 >= L.cam.width || y0 >= L.m.row_end || y0 + Pt::kH <= L.m.row_begin) continue;
        long long off = L.patch_head[tile * (int)per_tile + patch];
        if (off < 0) continue;                     // the patch met nothing, or is left to the search kernel
        const int px = x0 + r % Pt::kW, py = y0 + r / Pt::kW;
        const int ray_id = py * L.cam.width + px;
        const bool mine = px < L.cam.width && py >= L.m.row_begin && py < L.m.row_end && !L.ray_unrecorded[ray_id];
        const unsigned recorded = __ballot_sync(kFull, mine) & Pt::kRayBits;
        float3 dir, dl = make_float3(0.f, 0.f, 0.f);
        float D = 0.f, T = 1.0f;
        {
            Ray ray;
            make_ray(L.cam, px, py, ray);
            dir = ray.d;
        }
        if (mine) {
            const float* g = L.dl_drgb + 3 * (size_t)ray_id;
            const float* c = L.rgb_in + 3 * (size_t)ray_id;
            dl = make_float3(g[0], g[1], g[2]);
            D = fmaf(dl.x, c[0], fmaf(dl.y, c[1], __fmul_rn(dl.z, c[2])));
        }
        while (off >= 0) {
            const int* chunk = L.tape + off;
            const int4 h0 = __ldcs(reinterpret_cast<const int4*>(chunk)), h1 = __ldcs(reinterpret_cast<const int4*>(chunk) + 1);
            // The next chunk's sums on their way from memory into the L2 while this one is worked on (a chunk and the 64 ints behind its fixed
            // part lie within the recording: that much room was asked for).  Their loads are what a step waits for most: replay of the 300 k object
            // 2.05 -> 1.95 ms, of 4 k Gaussians at 64x64 0.089 -> 0.082, of four 3 M views 10.51 -> 10.45.
            const long long next = get_offset(h1.x, h1.y);
            if (lane == 0 && next >= 0)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(L.tape + next), "r"(4 * (Pt::kTapeList + 64)) : "memory");
            const unsigned rays = (unsigned)h0.y & recorded;
            const bool act = (rays >> r) & 1u;
            const float tbuffer = __int_as_float(chunk[8 + r]), dt = __int_as_float(chunk[Pt::kTapeDt + r]);
            // ---- first pass: transmittance and the per-sample terms (slab_back_terms of march_common.cuh)
            {
                const float4* sums = reinterpret_cast<const float4*>(chunk + Pt::kTapeSums) + lane;
                float run = 0.f, back = 0.f, T16 = T, x16 = 0.f;
                bool live = true;
                SampleTree<P> tree;
                constexpr int kAhead = Pt::kSamples < 4 ? Pt::kSamples : 4;
                float4 ahead[kAhead];
#pragma unroll
                for (int i = 0; i < kAhead; ++i) ahead[i] = __ldcs(sums + 32 * i);
#pragma unroll
                for (int i = 0; i < Pt::kSamples; ++i) {
                    const float4 c = ahead[i % kAhead];
                    if (i + kAhead < Pt::kSamples) ahead[i % kAhead] = __ldcs(sums + 32 * (i + kAhead));
                    const float x = __fmul_rn(c.x, dt);
                    float before, earlier;
                    const float all = across_ray<P>(x, sub, before);
                    if (i == Pt::kSamples / 2) {
                        x16 = tree.half;
                        T16 = __fmul_rn(T, exp_neg(x16));
                        live = T16 > eps;
                    }
                    const float excl = __fadd_rn(run, before);
                    run = __fadd_rn(run, all);
                    const float one_m_w = 1.0f - exp_neg(x);
                    const float Ts = __fmul_rn(T, exp_neg(excl));
                    const float inv_s = c.x > 0.f ? rcp_approx(c.x) : 0.f;
                    const float chat = __fmul_rn(fmaf(dl.x, c.y, fmaf(dl.y, c.z, __fmul_rn(dl.z, c.w))), inv_s);
                    const float tw = __fmul_rn(Ts, one_m_w);
                    const float step = __fmul_rn(tw, chat);                       // T_s (1 - w_s) chat_s
                    const float steps = across_ray<P>(step, sub, earlier);
                    const float Ds = __fadd_rn(D, -__fadd_rn(back, earlier));
                    back = __fadd_rn(back, steps);
                    const float beta = live ? __fmul_rn(tw, inv_s) : 0.f;
                    const float alpha = __fmul_rn(fmaf(Ts, chat, -Ds), dt);
                    sh.bg[P * i + sub][r] = make_float2(beta, live ? fmaf(-beta, chat, alpha) : 0.f);
                    tree.add(i, all);
                }
                if (act) {
                    D = __fadd_rn(D, -back);
                    T = live ? __fmul_rn(T, exp_neg(__fadd_rn(x16, tree.half))) : T16;
                }
            }
            __syncwarp();
            // ---- second pass: the Gaussians of the step
            const float inv_dt = rcp_approx(dt);
            const float2* bg = &sh.bg[0][r];
            const int2* list = reinterpret_cast<const int2*>(chunk + Pt::kTapeList);
            int n = h0.x;
            long long piece = get_offset(h0.z, h0.w);
            while (true) {
                for (int base = 0; base < n; base += 32) {
                    const int cnt = min(n - base, 32);
                    if (lane < cnt) {
                        const int2 en = __ldcs(list + base + lane);
                        const int j = en.x;
                        const float4 g0 = __ldg(&L.g.g0[j]), g1 = __ldg(&L.g.g1[j]), g2 = __ldg(&L.g.g2[j]);
                        stage_geometry(st, lane, j, g0, g1, g2, whiten_eye(L, g0, g1, g2));
                        st.ex[lane].x = __ldg(&L.g.hk[j]);
                        st.rgba[lane] = __ldg(&L.g.rgba[j]);
                        hit_by(st, lane) = (unsigned)en.y & rays;
                    } else {
                        hit_by(st, lane) = 0u;
                    }
                    __syncwarp();
                    for (int e = 0; e < cnt; e += P) {
                        const int q = e + sub;
                        const bool hit = (hit_by(st, q) >> r) & 1u;
                        const float4 m0 = st.m0[q], m1 = st.m1[q], m2 = st.m2[q];
                        const float2 ex = make_float2(st.ex[q].x, st.ex[q].z);
                        const float4 c = st.rgba[q];
                        const float3 Oe = staged_eye(m1, m2), de = staged_dir(m0, m1, m2, dir);
                        const float a = dot3(de, de), inv_a = rcp_approx(a), b = -dot3(Oe, de);
                        // the closest approach as in ellipsoid_stretch; a lane without a hit adds up nothing, and whatever its ray is to the
                        // Gaussian, zero times a point near it is zero
                        const float t0 = __fmul_rn(b, inv_a), tca = hit ? fmaf(fmaf(-t0, a, b), inv_a, t0) : 0.f;
                        const float3 yc = make_float3(fmaf(tca, de.x, Oe.x), fmaf(tca, de.y, Oe.y), fmaf(tca, de.z, Oe.z));
                        const float qmin = dot3(yc, yc);
                        const float ay = __fmul_rn(1.0f - qmin, inv_a), az = __fmul_rn(-ex.x, a), aw = __fmul_rn(-ex.x, qmin);
                        // runs of samples that may lie inside (first_run), up to the last one within a twentieth of a sample of the
                        // ellipsoid (positions are good to a few 2^-24 t, so up to t = 10^5 dt); d^2 < ay decides
                        const float hw = sqrt_approx(fmaxf(ay, 0.f));
                        const int s_lo = first_run(tca, hw, tbuffer, inv_dt);
                        const int s_hi = min(__float2int_rd(slab_sample(__fadd_rn(tca, hw), tbuffer, inv_dt) + 0.05f), kSlab - 1);
                        const int runs = hit && s_hi >= s_lo ? (s_hi - s_lo) / kRun + 1 : 0;
                        // moments about the closest approach: there the whitened ray is at right angles to its direction, so the
                        // terms do not cancel, and inside the ellipsoid none is larger than one
                        const float ci = quotient(fmaf(dl.x, c.x, fmaf(dl.y, c.y, __fmul_rn(dl.z, c.z))), c.w);
                        const float off_d = __fadd_rn(tbuffer, -tca);
                        float2 sn = make_float2(0.f, 0.f), n12 = make_float2(0.f, 0.f);          // sums of beta g and of w; of w d and w d^2
                        float x = (float)s_lo + 0.5f;
                        const float2 *at = bg + s_lo * Pt::kRays, *const end = at + runs * (kRun * Pt::kRays);
#pragma unroll 1
                        for (; at != end; at += kRun * Pt::kRays) {
                            float d = __fadd_rn(__fmul_rn(x, dt), off_d);
#pragma unroll
                            for (int i = 0; i < kRun; ++i) {
                                const float d2 = __fmul_rn(d, d);
                                const float2 w = at[i * Pt::kRays];
                                // 2^-inf is the zero outside: what is chosen is the exponent, before the slow unit (1.5 % of the kernel)
                                const float g = ex2_approx(d2 < ay ? fmaf(az, d2, aw) : -INFINITY);
                                const float u = fmaf(ci, w.x, w.y), ga = __fmul_rn(g, u);  // w = g * (alpha + beta*(chat_i - chat_s))
                                sn = __ffma2_rn(make_float2(g, g), make_float2(w.x, u), sn);
                                n12 = __ffma2_rn(make_float2(ga, ga), make_float2(d, d2), n12);
                                d = __fadd_rn(d, dt);
                            }
                            x += (float)kRun;
                        }
                        const float4 A = make_float4(yc.x, yc.y, yc.z, 0.f);
                        const GaussGrad gg = expand_gradient(c.w, A, make_float4(de.x, de.y, de.z, 0.f), sn.x, sn.y, n12.x, n12.y);
                        sh.red[0][lane] = gg.mu.x; sh.red[1][lane] = gg.mu.y; sh.red[2][lane] = gg.mu.z;
                        sh.red[3][lane] = gg.y00; sh.red[4][lane] = gg.y11; sh.red[5][lane] = gg.y22;
                        sh.red[6][lane] = gg.y01; sh.red[7][lane] = gg.y02; sh.red[8][lane] = gg.y12;
                        sh.red[9][lane] = gg.dsigma;
                        sh.red[10][lane] = __fmul_rn(dl.x, gg.drgb_scale);
                        sh.red[11][lane] = __fmul_rn(dl.y, gg.drgb_scale);
                        sh.red[12][lane] = __fmul_rn(dl.z, gg.drgb_scale);
                        __syncwarp();
                        // the lanes of entry e + h add its components over the rays (row layout: emit_global); lanes past the thirteenth add up
                        // the last one too and keep it to themselves
                        float* row = reinterpret_cast<float*>(L.grad_rows) +
                                     16 * ((size_t)((unsigned)tile & (unsigned)(L.grad_copies - 1)) * (size_t)L.g.n_pad + (size_t)__float_as_int(ex.y));
#pragma unroll
                        for (int k0 = 0; k0 < 13; k0 += Pt::kRays) {
                            const int k = min(k0 + r, 12);
                            const float4* v = reinterpret_cast<const float4*>(&sh.red[k][Pt::kRays * sub]);
                            float2 sum = make_float2(0.f, 0.f);
#pragma unroll
                            for (int i = 0; i < Pt::kRays / 4; ++i) { const float4 a4 = v[i]; sum = __fadd2_rn(sum, __fadd2_rn(make_float2(a4.x, a4.y), make_float2(a4.z, a4.w))); }
                            if (q < cnt && k0 + r < 13) atomicAdd(row + k, __fadd_rn(sum.x, sum.y));
                        }
                        __syncwarp();
                    }
                }
                if (piece < 0) break;
                const int4 h = *reinterpret_cast<const int4*>(L.tape + piece);
                list = reinterpret_cast<const int2*>(L.tape + piece + kTapePiece);
                n = h.x;
                piece = get_offset(h.z, h.w);
            }
            off = next;
        }
    }
}

// ---------------------------------------------------------------- backward, by searching again
// For rays without a recording: all of them when the forward did not record, else only those
// it could not record (ray_unrecorded).
__global__ void __launch_bounds__(kThreads) march_backward_lists_kernel(const __grid_constant__ MarchLaunch L) {
    __shared__ ListShared sh;
    __shared__ int hit_lists[kWarps][kHitList];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    WarpStage& ws = sh.ws[warp];
    int* pend = sh.pend[warp];
    const int tile = L.lists.tile_order ? __ldg(&L.lists.tile_order[blockIdx.x]) : blockIdx.x;
    if (L.tape && !L.tile_unrecorded[tile]) return;             // every ray of the tile was recorded: the replay kernel's
    const int tile_x = tile % L.lists.tiles_x, tile_y = tile / L.lists.tiles_x;
    const float eps = L.m.transmittance_eps;
    const SceneBox box = *L.box;
    const TileView tv = tile_view(L.lists, tile);
    Tally tl;
#pragma unroll
    for (int i = 0; i < C_NUM; ++i) tl.v[i] = 0;
    if (tid == 0) sh.next_ray = 0;
    __syncthreads();

    while (true) {
        int ray = 0;
        if (lane == 0) ray = atomicAdd(&sh.next_ray, 1);
        ray = __shfl_sync(kFull, ray, 0);
        if (ray >= L.lists.tile * L.lists.tile) break;
        int px, py;
        if (!ray_pixel(L, tile_x, tile_y, ray, px, py)) continue;
        const int ray_id = py * L.cam.width + px;
        if (L.tape && !L.ray_unrecorded[ray_id]) continue;      // recorded: the replay kernel's
        Ray r;
        make_ray(L.cam, px, py, r);
        float tenter, texit;
        clip_scene(box, r, tenter, texit);
        int cursor = 0;
        const float3 dl = make_float3(L.dl_drgb[3 * (size_t)ray_id], L.dl_drgb[3 * (size_t)ray_id + 1],
                                      L.dl_drgb[3 * (size_t)ray_id + 2]);
        float D = fmaf(dl.x, L.rgb_in[3 * (size_t)ray_id],
                       fmaf(dl.y, L.rgb_in[3 * (size_t)ray_id + 1], __fmul_rn(dl.z, L.rgb_in[3 * (size_t)ray_id + 2])));
        float T = 1.0f;
        float first = closest_in_tile<false>(L, r, tenter, texit, tv, cursor, pend, lane, tl);
        if (!(first < INFINITY && first < texit)) continue;                       // backward .cu:249-254
        tenter = first;
        float tbuffer = tenter;
        int slab_index = 0;
        while (tbuffer < texit && T > eps && slab_index < kMaxSlabs) {
            SlabPlan p = plan_slab(L.m, tbuffer, T, tenter, texit);
            ++slab_index;
            if (!p.traced) { tbuffer = __fadd_rn(tbuffer, p.slab); continue; }
            const float tau = __fmul_rn((float)lane + 0.5f, p.dt);
            auto enumerate = [&](auto&& leaf) { search_tile<false>(L, r, p.tmin, p.tmax, tv, cursor, pend, lane, tl, leaf); };
            float s, dc, u0, u1;
            bool overflow;
            int* hits = hit_lists[warp];
            int nhit = slab_sums<false, true>(L, L.m, tbuffer, p.dt, ray_id, slab_index, dl, ws, lane, tl, enumerate, s, dc,
                                              u0, u1, overflow, &hits, kHitList);
            if (nhit == 0) {
                tbuffer = __fadd_rn(tbuffer, p.slab);
                float nxt = closest_in_tile<false>(L, r, tbuffer, texit, tv, cursor, pend, lane, tl);
                if (!(nxt < INFINITY)) break;
                tbuffer = nxt;
                continue;
            }
            SlabBackTerms bt = slab_back_terms(s, dc, p.dt, T, D, eps, lane);
            // pass 2: the hits again -- from the remembered list when it held them all, else by a second query
            auto emit = [&](int j, const GaussGrad& g) { emit_global(L, dl, j, g, blockIdx.x); };
            if (nhit <= kHitList) {
                __syncwarp();
                slab_gradients(L, L.m, r, p, tbuffer, tau, dl, bt.beta, bt.gamma, ws, sh.prim_of[warp], lane,
                               [&](auto&& leaf) {
                                   for (int base = 0; base < nhit; base += kFan) {
                                       const bool valid = base + lane < nhit;
                                       const int j = valid ? hits[base + lane] : 0;
                                       LeafTest t = test_gaussian(L, r, j, valid, p.tmin, p.tmax, tl, false, false);
                                       if (!leaf(t, j)) return;
                                   }
                               }, emit);
            } else {
                slab_gradients(L, L.m, r, p, tbuffer, tau, dl, bt.beta, bt.gamma, ws, sh.prim_of[warp], lane, enumerate, emit);
            }
            D = __fadd_rn(D, -bt.d_total);
            T = slab_exit_T(bt.tr, eps);
            tbuffer = __fadd_rn(tbuffer, p.slab);
        }
    }
}

}  // namespace

cudaError_t launch_march_forward_per_ray(const MarchLaunch& m, cudaStream_t s);
cudaError_t launch_march_backward_per_ray(const MarchLaunch& m, cudaStream_t s);

static bool use_lists(const MarchLaunch& m) {
    return !(m.m.flags & (RGX_FLAG_BRUTE_FORCE | RGX_FLAG_PER_RAY_SEARCH)) && m.lists.ent_id != nullptr && m.g.n > 0;
}

// Lanes per ray.  Two where the image gives every warp the device can hold a patch of sixteen rays (at sixteen warps on each of 148 SMs that
// is 37,888 rays; the line is at 200x200); with fewer rays, smaller patches: more warps, and fewer Gaussians per patch, the longest patch being all there is to wait for.
// Forward + backward in ms with 2 / 4 / 8 lanes per ray, 100 k object: 64x64 1.01 / 0.54 / 0.36, 128x128 0.65 / 0.45 / 0.36, 150x150
// 0.77 / 0.51 / 0.49, 180x180 0.75 / 0.52 / 0.60, 256x256 0.74 / 0.74 / 0.97, 300x300 0.92 / 1.06 / 1.48; 1 M unbounded: 128x128 0.41 / 0.28 / 0.24,
// 150x150 0.43 / 0.30 / 0.30, 200x200 0.44 / 0.38 / 0.43, 256x256 0.50 / 0.50 / 0.64.  Four lanes would do a little better up to 240x240 (object 0.66 against
// 0.76 at 230x230, unbounded 0.44 against 0.45), but every line moves the order in which a ray's terms are added up, and single gradient entries of
// dense views with it by 1.7e-2 of the tensor's root mean square.  The choice depends on the image alone, so that every march of
// a view -- whole or a row range, recording or not -- adds up a ray's colour in the same order.
static int patch_lanes(const MarchLaunch& m) {
    const long long rays = (long long)m.cam.width * m.cam.height;
    return rays <= 128 * 128 ? 8 : rays <= 200 * 200 ? 4 : 2;
}

// CTAs of a patch kernel: as many as fit the device at once (they fetch patches until there are none left).
template <int P>
static int patch_ctas(const MarchLaunch& m, int ctas_per_sm) {
    const long long want = (long long)m.lists.tiles_x * m.lists.tiles_y * (m.lists.tile * m.lists.tile / Patch<P>::kRays),
                    fit = (long long)m.sm_count * ctas_per_sm;
    return (int)(want < fit ? want : fit);
}

template <int P, bool COUNT, bool SAVE, int HZ>
static void launch_patches(const MarchLaunch& m, cudaStream_t s) {
    note_launch(), march_forward_patches_kernel<P, COUNT, SAVE, HZ><<<patch_ctas<P>(m, forward_ctas<COUNT>()), kPatchWarps * 32, 0, s>>>(m);
}

template <int P>
static void launch_forward_lanes(const MarchLaunch& m, cudaStream_t s) {
    const bool count = (m.m.flags & RGX_FLAG_COUNT_WORK) != 0, save = m.tape != nullptr;
    if (m.hz_phase == 3) {
        if (save) launch_patches<P, false, true, 2>(m, s);
        else launch_patches<P, false, false, 2>(m, s);
    } else if (m.hz_phase != 0) launch_patches<P, false, false, 1>(m, s);
    else if (count && save) launch_patches<P, true, true, 0>(m, s);
    else if (count) launch_patches<P, true, false, 0>(m, s);
    else if (save) launch_patches<P, false, true, 0>(m, s);
    else launch_patches<P, false, false, 0>(m, s);
}

cudaError_t launch_march_forward(const MarchLaunch& m, cudaStream_t s) {
    if (!use_lists(m)) return launch_march_forward_per_ray(m, s);
    if (m.lists.tiles_x * m.lists.tiles_y <= 0) return cudaSuccess;
    switch (patch_lanes(m)) {
        case 2: launch_forward_lanes<2>(m, s); break;
        case 4: launch_forward_lanes<4>(m, s); break;
        default: launch_forward_lanes<8>(m, s);
    }
    return cudaGetLastError();
}

cudaError_t launch_march_backward_search(const MarchLaunch& m, cudaStream_t s) {
    if (!use_lists(m)) return launch_march_backward_per_ray(m, s);
    const int grid = m.lists.tiles_x * m.lists.tiles_y;
    if (grid <= 0) return cudaSuccess;
    note_launch(), march_backward_lists_kernel<<<grid, kThreads, 0, s>>>(m);   // a CTA whose tile was recorded completely returns at once
    return cudaGetLastError();
}

template <int P>
static cudaError_t launch_replay(const MarchLaunch& m, cudaStream_t s) {
    note_launch(), march_backward_patches_kernel<P><<<patch_ctas<P>(m, kReplayCtas), kPatchWarps * 32, 0, s>>>(m);
    return cudaGetLastError();
}

cudaError_t launch_march_backward_replay(const MarchLaunch& m, cudaStream_t s) {
    if (!use_lists(m) || !m.tape) return cudaSuccess;
    if (m.lists.tiles_x * m.lists.tiles_y <= 0) return cudaSuccess;
    switch (patch_lanes(m)) {
        case 2: return launch_replay<2>(m, s);
        case 4: return launch_replay<4>(m, s);
        default: return launch_replay<8>(m, s);
    }
}

}  // namespace rgx
