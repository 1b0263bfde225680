// Per-view tile lists.
//
// All rays of a view leave from one point, so which Gaussians a ray can meet is
// decided by where the Gaussian projects on the image.  Once per view every
// Gaussian is projected to a rectangle of tiles (bin_tile_size) and paired with each
// tile it touches; the pairs are dealt to their tiles and sorted there by the nearest
// distance from the eye, and every tile ends up with a front-to-back list of
// candidate Gaussians with, per entry, the range of distances its box spans.  A ray
// then never searches the hierarchy: it slides along its tile's list.
//
// Takes the place of what OptiX traversal does for the reference at every
// optixTrace (cuda_train/forward/gaussians_aabb.cu:234-313); the list is a superset
// of every hit set, the test that decides a hit stays the per-ray one.
#include "rgx_internal.cuh"
#include "device_math.cuh"
#include <cub/device/device_radix_sort.cuh>
#include <cub/block/block_scan.cuh>
#include <algorithm>
#include <cmath>
#include <cstring>

namespace rgx {

namespace {

constexpr unsigned kFullMask = 0xffffffffu;

// Camera coordinates (x right, y down, z forward, in units of the ray parametrisation a = x/z, b = y/z).
__device__ __forceinline__ void to_camera(const Projector& p, float x, float y, float z, float& xc, float& yc, float& zc) {
    float qx = x - p.eye[0], qy = y - p.eye[1], qz = z - p.eye[2];
    xc = qx * p.du[0] + qy * p.du[1] + qz * p.du[2];
    yc = qx * p.dv[0] + qy * p.dv[1] + qz * p.dv[2];
    zc = qx * p.dw[0] + qy * p.dw[1] + qz * p.dw[2];
}

// A direction in camera coordinates.
__device__ __forceinline__ float3 turn_to_camera(const Projector& p, float x, float y, float z) {
    return make_float3(fmaf(x, p.du[0], fmaf(y, p.du[1], z * p.du[2])), fmaf(x, p.dv[0], fmaf(y, p.dv[1], z * p.dv[2])),
                       fmaf(x, p.dw[0], fmaf(y, p.dw[1], z * p.dw[2])));
}
// The eight corners c +- e0 +- e1 +- e2 of a box in camera coordinates: from its middle and half edges, where eight corners turned
// one by one took three times the arithmetic (bin_near_hist_kernel, 1 M Gaussians 63 -> 56 us).
__device__ __forceinline__ void box_corners(float3 c, float3 e0, float3 e1, float3 e2, float* xc, float* yc, float* zc) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float3 a = i & 2 ? c + e2 : c - e2, b = i & 1 ? a + e1 : a - e1;
        xc[2 * i] = b.x - e0.x; yc[2 * i] = b.y - e0.y; zc[2 * i] = b.z - e0.z;
        xc[2 * i + 1] = b.x + e0.x; yc[2 * i + 1] = b.y + e0.y; zc[2 * i + 1] = b.z + e0.z;
    }
}

// Pixel bounds of eight camera-space corners.  Returns 0 if every corner is behind
// the eye (no ray, which only goes forward, can reach the box), 1 if every corner is
// safely in front (bounds are the bounds of the projected corners), 2 otherwise.
__device__ __forceinline__ int project_corners(const Projector& p, const float* xc, const float* yc, const float* zc,
                                               float& lox, float& hix, float& loy, float& hiy) {
    bool all_front = true, all_behind = true;
    lox = loy = INFINITY; hix = hiy = -INFINITY;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        float len = fabsf(xc[c]) + fabsf(yc[c]) + fabsf(zc[c]);
        bool front = zc[c] > 1e-4f * len && zc[c] > 1e-12f;
        all_front = all_front && front;
        all_behind = all_behind && !(zc[c] > 0.f);
        const float inv = front ? rcp_approx(zc[c]) : NAN;           // the margins about the rectangle cover its rounding; min and max pass by a NaN
        const float a = xc[c] * inv, b = yc[c] * inv;
        lox = fminf(lox, a); hix = fmaxf(hix, a);
        loy = fminf(loy, b); hiy = fmaxf(hiy, b);
    }
    // (of use to the caller where all corners are in front)
    const float x0 = fmaf(lox, p.sx, p.ox), x1 = fmaf(hix, p.sx, p.ox), y0 = fmaf(loy, p.sy, p.oy), y1 = fmaf(hiy, p.sy, p.oy);
    lox = fminf(x0, x1); hix = fmaxf(x0, x1); loy = fminf(y0, y1); hiy = fmaxf(y0, y1);
    return all_behind ? 0 : (all_front ? 1 : 2);
}

// A convex body that straddles the eye plane has no bounded projection.  Its tile
// columns are found from the planes through the eye instead: column [a_lo, a_hi] (in
// x/z) can only be touched if some corner lies on the inner side of each of its two
// bounding planes x - a z = 0, that is unless x_i - a_lo z_i < 0 for every corner or
// x_i - a_hi z_i > 0 for every corner.  Each of the two holds for a in an open interval
// whose ends are ratios x_i / z_i, so the eight corners are looked at once and a column
// costs two comparisons.  Conservative (a tolerance on every corner), exact per plane.
// Same for rows.  Returns the first and last pixel of the touched columns.
__device__ __forceinline__ void straddle_tiles(const float* xc, const float* zc, float scale, float offset, int n_tiles,
                                               int tile, int n_pix, float& lo_pix, float& hi_pix) {
    const float inv_scale = 1.0f / scale;
    const float a_first = (-0.02f - offset) * inv_scale, a_last = ((float)(n_pix - 1) + 0.02f - offset) * inv_scale;
    const float amax = 2.0f * fmaxf(fabsf(a_first), fabsf(a_last));
    float gl = -INFINITY, gh = INFINITY, hl = -INFINITY, hh = INFINITY;   // all below: a in (gl, gh); all above: a in (hl, hh)
    bool okg = true, okh = true;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float tol = 1e-5f * (fabsf(xc[i]) + amax * fabsf(zc[i]));
        const float up = xc[i] + tol, dn = xc[i] - tol;
        if (zc[i] > 1e-20f) {
            gl = fmaxf(gl, up / zc[i]);
            hh = fminf(hh, dn / zc[i]);
        } else if (zc[i] < -1e-20f) {
            gh = fminf(gh, up / zc[i]);
            hl = fmaxf(hl, dn / zc[i]);
        } else {
            okg = okg && up < 0.f;
            okh = okh && dn > 0.f;
        }
    }
    auto touched = [&](int c, float& p0, float& p1) {
        p0 = (float)(c * tile);
        p1 = (float)min(c * tile + tile - 1, n_pix - 1);
        const float a_lo = (p0 - 0.02f - offset) * inv_scale, a_hi = (p1 + 0.02f - offset) * inv_scale;
        const bool all_below = okg && a_lo > gl && a_lo < gh;
        const bool all_above = okh && a_hi > hl && a_hi < hh;
        return !(all_below || all_above);
    };
    lo_pix = INFINITY; hi_pix = -INFINITY;
    int c0 = 0;
    float p0, p1;
    for (; c0 < n_tiles; ++c0)
        if (touched(c0, p0, p1)) { lo_pix = p0; hi_pix = p1; break; }
    for (int c = n_tiles - 1; c > c0; --c)
        if (touched(c, p0, p1)) { hi_pix = p1; break; }
}

__device__ __forceinline__ float3 pixel_dir(const rgx_camera& c, float px, float py) {
    float a = 2.0f * ((px + 0.5f) / (float)c.width - c.pp[0]) * c.tan_half_fov[0];
    float bq = 2.0f * ((py + 0.5f) / (float)c.height - c.pp[1]) * c.tan_half_fov[1];
    float3 d = make_float3(a * c.u[0] + bq * c.v[0] + c.w[0], a * c.u[1] + bq * c.v[1] + c.w[1],
                           a * c.u[2] + bq * c.v[2] + c.w[2]);
    float inv = 1.0f / sqrtf(dot3(d, d));
    return d * inv;
}

// Per tile: direction of the ray through the tile centre and the largest chord |d - d_c| to a
// ray of the tile (the rays of a tile lie inside the pyramid of its four corner rays).
__global__ void bin_tile_dirs_kernel(BinLaunch b, int ntiles) {
    after_previous();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntiles) return;
    int tx = t % b.tiles_x, ty = t / b.tiles_x + b.ty_first;
    float x0 = (float)(tx * b.tile), x1 = (float)min(tx * b.tile + b.tile - 1, b.cam.width - 1);
    float y0 = (float)(ty * b.tile), y1 = (float)min(ty * b.tile + b.tile - 1, b.cam.height - 1);
    float3 dc = pixel_dir(b.cam, 0.5f * (x0 + x1), 0.5f * (y0 + y1));
    float chord = 0.f;
    for (int c = 0; c < 4; ++c) {
        float3 d = pixel_dir(b.cam, (c & 1) ? x1 : x0, (c & 2) ? y1 : y0) - dc;
        chord = fmaxf(chord, sqrtf(dot3(d, d)));
    }
    const float w = chord * 1.001f + 1e-7f;
    b.tile_dir[t] = make_float4(dc.x, dc.y, dc.z, w);
    if (b.pick) atomicMax(&b.pick->chord_bits, __float_as_uint(w));      // positive floats order like their bits
}

// Per-Gaussian data needed to bound its meeting with a tile.
struct PairGeom {
    float2 bx, by, bz;
    float4 g0, g1, g2;
    float far_box;      // largest distance from the eye to the box
    float rho_scale;    // operator norm of the whitening map: 1 / (k s_min), with slack for non-unit quaternions
    float away, slack;  // see pair_range
};

// Range of ray parameters at which some ray of the tile can be inside the Gaussian's box and
// inside its truncation ellipsoid; false if no ray of the tile can.  Every ray of the tile is, at
// parameter t, within t * chord of the central ray's point, so the central ray is tested against
// the box and the ellipsoid grown by that much.
// A ray whose closest approach lies behind the eye misses, even from inside (ellipsoid_stretch in march_common.cuh): for M the whitening
// map and Oe = M (eye - centre), if -Oe . M d < 0.  `away` = |M^T Oe|, so for a ray of the tile that is at most the central ray's plus
// chord * away; `slack` covers what rounding makes of it here and in the march (make_pair_geom).  Such pairs are those of Gaussians that hold the eye and lie
// behind it: a third of the entries that the march of 30 k large Gaussians about the camera tested, a seventh of 1 M
// (forward of the former at 399x301 0.278 -> 0.229 ms, of the latter at 628x414 0.907 -> 0.851, four views of 3 M 14.47 -> 14.02).
__device__ __forceinline__ bool pair_range(const float* eye, float4 td, const PairGeom& g, float& tn, float& tf) {
    const float infl = g.far_box * td.w * 1.0001f + 1e-6f;
    // ellipsoid |M (x - p)| <= 1 grown to radius rho in the whitened frame; first, since it turns away the more: a needle's
    // rectangle is full of tiles beside it
    const float rho = 1.0f + infl * g.rho_scale;
    const float3 O = make_float3(eye[0] - g.g0.x, eye[1] - g.g0.y, eye[2] - g.g0.z);
    const float3 Oe = make_float3(g.g0.w * O.x + g.g1.x * O.y + g.g1.y * O.z, g.g1.z * O.x + g.g1.w * O.y + g.g2.x * O.z,
                                  g.g2.y * O.x + g.g2.z * O.y + g.g2.w * O.z);
    const float3 de = make_float3(g.g0.w * td.x + g.g1.x * td.y + g.g1.y * td.z, g.g1.z * td.x + g.g1.w * td.y + g.g2.x * td.z,
                                  g.g2.y * td.x + g.g2.z * td.y + g.g2.w * td.z);
    const float qa = dot3(de, de), qb = -dot3(Oe, de), qc = dot3(Oe, Oe) - rho * rho;
    if (fmaf(td.w, g.away, qb) < -g.slack) return false;       // behind the eye for every ray of the tile
    const float disc = qb * qb - qa * qc;
    const float mag = qb * qb + fabsf(qa * qc);
    if (disc < -1e-5f * mag) return false;
    tn = 0.f; tf = INFINITY;
    const float o[3] = {eye[0], eye[1], eye[2]}, d[3] = {td.x, td.y, td.z};
    const float lo[3] = {g.bx.x - infl, g.by.x - infl, g.bz.x - infl}, hi[3] = {g.bx.y + infl, g.by.y + infl, g.bz.y + infl};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (fabsf(d[a]) < 1e-12f) {
            if (o[a] < lo[a] || o[a] > hi[a]) return false;
        } else {
            const float inv = __fdividef(1.0f, d[a]);      // the margins below cover its rounding
            float t0 = (lo[a] - o[a]) * inv, t1 = (hi[a] - o[a]) * inv;
            tn = fmaxf(tn, fminf(t0, t1));
            tf = fminf(tf, fmaxf(t0, t1));
        }
    }
    if (tn > tf * (1.0f + 1e-5f) + 1e-6f) return false;
    if (qa > 1e-30f) {
        const float sq = sqrtf(fmaxf(disc, 0.f) + 1e-5f * mag);
        const float inv_qa = __fdividef(1.0f, qa);
        const float r1 = (qb - sq) * inv_qa, r2 = (qb + sq) * inv_qa;
        tn = fmaxf(tn, r1);
        tf = fminf(tf, r2);
    }
    tn = fmaxf(tn * (1.0f - 1e-5f) - 1e-6f, 0.f);
    tf = tf * (1.0f + 1e-5f) + 1e-6f;
    return tn <= tf;
}

// How a (tile, Gaussian) pair is packed into its 64-bit sort key, most significant first:
// tile | near distance (sign dropped, low mantissa bits dropped) | sorted slot of the Gaussian.
// Every key is distinct, so the sorted order does not depend on the order of emission.
// The near distance takes near_bits = 5 exponent bits + 7 to 14 mantissa bits: a window of 32 binades, 2^-16 .. 2^16
// (what lies below rounds down to zero, what lies above to the largest code), good to 0.8 % or better -- a few per
// cent of a slab's length.  The key is then as short as a whole number of 8-bit passes of the radix sort allows
// with at least 12 bits for the distance: 48 bits (six passes, not seven) for 3 M Gaussians on 4,108 tiles.
struct KeyLayout {
    int tile_bits, near_bits, id_bits;
};
constexpr int kNearExpBits = 5;
constexpr int kNearExpWindowBase = 111;     // biased exponent of 2^-16

__host__ __device__ inline KeyLayout key_layout(int ntiles, int n_pad) {
    KeyLayout k;
    k.tile_bits = 1;
    while ((1 << k.tile_bits) < ntiles) ++k.tile_bits;
    k.id_bits = 1;
    while ((1ll << k.id_bits) < (long long)n_pad) ++k.id_bits;
    const int fixed = k.tile_bits + k.id_bits;
    k.near_bits = ((fixed + 12 + 7) / 8) * 8 - fixed;            // 12 .. 19
    return k;
}

// The near distance as the list stores it: rounded down to what the key keeps, so that the
// order of the keys is exactly the order of the stored distances.
__host__ __device__ inline unsigned near_quantised(float tn, const KeyLayout& kl) {
#ifdef __CUDA_ARCH__
    const unsigned bits = __float_as_uint(tn);
#else
    unsigned bits;
    std::memcpy(&bits, &tn, sizeof(bits));
#endif
    const int mant = kl.near_bits - kNearExpBits;
    const int e = (int)((bits << 1) >> 24) - kNearExpWindowBase;
    if (e < 0) return 0u;
    if (e > 31) return (1u << kl.near_bits) - 1u;
    return ((unsigned)e << mant) | ((bits >> (23 - mant)) & ((1u << mant) - 1u));
}
__host__ __device__ inline float near_stored(unsigned q, const KeyLayout& kl) {
    const int mant = kl.near_bits - kNearExpBits;
    const unsigned bits = q == 0u ? 0u : ((((q >> mant) + (unsigned)kNearExpWindowBase) << 23) | ((q & ((1u << mant) - 1u)) << (23 - mant)));
#ifdef __CUDA_ARCH__
    return __uint_as_float(bits);
#else
    float f;
    std::memcpy(&f, &bits, sizeof(f));
    return f;
#endif
}

// Largest distance from the eye to a point of the box, rounded up (pair_range grows the box in proportion to it).
__device__ __forceinline__ float box_far_distance(const float* eye, float2 bx, float2 by, float2 bz) {
    const float fx = fmaxf(fabsf(bx.x - eye[0]), fabsf(bx.y - eye[0])), fy = fmaxf(fabsf(by.x - eye[1]), fabsf(by.y - eye[1])),
                fz = fmaxf(fabsf(bz.x - eye[2]), fabsf(bz.y - eye[2]));
    return sqrtf(fx * fx + fy * fy + fz * fz) * (1.0f + 1e-5f) + 1e-6f;
}

// What pair_range needs to know of a Gaussian, from its box, whitening map, scales, quaternion and hk.
__device__ __forceinline__ PairGeom make_pair_geom(const float* eye, float2 bx, float2 by, float2 bz, float4 g0, float4 g1,
                                                   float4 g2, float4 sd, float4 q, float kk) {
    PairGeom g;
    g.bx = bx; g.by = by; g.bz = bz;
    g.g0 = g0; g.g1 = g1; g.g2 = g2;
    g.far_box = box_far_distance(eye, bx, by, bz);
    float smin = fminf(sd.x, fminf(sd.y, sd.z));
    float qn = q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
    g.rho_scale = 1.02f * fmaxf(1.0f, qn) / (kk * smin);
    const float3 O = make_float3(eye[0] - g0.x, eye[1] - g0.y, eye[2] - g0.z);
    const float3 r0 = make_float3(g0.w, g1.x, g1.y), r1 = make_float3(g1.z, g1.w, g2.x), r2 = make_float3(g2.y, g2.z, g2.w);
    const float3 Oe = make_float3(dot3(r0, O), dot3(r1, O), dot3(r2, O)), v = r0 * Oe.x + r1 * Oe.y + r2 * Oe.z;
    g.away = sqrtf(dot3(v, v));
    // Oe is good to 3.5 rounding errors of |M| |O|, which is more than |Oe| by up to the ratio of the Gaussian's axes, M d to as many of
    // |M|, the product to three more of |Oe| |M|; here and in the march: 4.2e-7 |M|^2 |O| and 7.8e-7 |Oe| |M| together
    const float M2 = dot3(r0, r0) + dot3(r1, r1) + dot3(r2, r2);
    g.slack = 1e-5f * sqrtf(dot3(Oe, Oe) * M2) + 1e-6f * M2 * sqrtf(dot3(O, O));
    return g;
}

__device__ __forceinline__ unsigned long long pair_key(const KeyLayout& kl, unsigned tile, float tn, unsigned slot) {
    return ((unsigned long long)tile << (kl.near_bits + kl.id_bits)) |
           ((unsigned long long)near_quantised(tn, kl) << kl.id_bits) | (unsigned long long)slot;
}

constexpr int kEmitThreads = 256;

// Rectangle of tiles that Gaussian j can touch: the rectangle of its box cut by the rectangle of the oriented box
// of its truncation ellipsoid.  Returns the number of tiles (0: none, rect untouched).
__device__ __forceinline__ int gaussian_rect(const BinLaunch& b, const Projector& p, int j, float2 bx, float2 by, float2 bz,
                                             uint2& rect) {
    const int W = b.cam.width, H = b.cam.height;
    const int tiles_x_all = (W + b.tile - 1) / b.tile, tiles_y_all = (H + b.tile - 1) / b.tile;
    {
        // most Gaussians lie outside the view: the sphere about the box against the four side planes
        const float cx = 0.5f * (bx.x + bx.y) - p.eye[0], cy = 0.5f * (by.x + by.y) - p.eye[1], cz = 0.5f * (bz.x + bz.y) - p.eye[2];
        const float hx = 0.5f * (bx.y - bx.x), hy = 0.5f * (by.y - by.x), hz = 0.5f * (bz.y - bz.x);
        const float r = sqrtf(hx * hx + hy * hy + hz * hz) * (1.0f + 1e-4f), far = sqrtf(cx * cx + cy * cy + cz * cz);
        if (r == INFINITY) {            // an infinite scale: its box has no middle to place corners about, and may touch every tile
            rect = make_uint2((unsigned)(b.tiles_x - 1) << 16, (unsigned)(b.tiles_y - 1) << 16);
            return b.tiles_x * b.tiles_y;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (p.plane[q][0] * cx + p.plane[q][1] * cy + p.plane[q][2] * cz < -(r + 1e-5f * far + 1e-7f) * p.plane[q][3]) return 0;
    }
    float xc[8], yc[8], zc[8];
    float3 mid;
    to_camera(p, 0.5f * (bx.x + bx.y), 0.5f * (by.x + by.y), 0.5f * (bz.x + bz.y), mid.x, mid.y, mid.z);
    box_corners(mid, turn_to_camera(p, 0.5f * (bx.y - bx.x), 0.f, 0.f), turn_to_camera(p, 0.f, 0.5f * (by.y - by.x), 0.f),
                turn_to_camera(p, 0.f, 0.f, 0.5f * (bz.y - bz.x)), xc, yc, zc);
    float lox, hix, loy, hiy;
    int kind = project_corners(p, xc, yc, zc, lox, hix, loy, hiy);
    if (kind == 0) return 0;
    if (kind == 2) {
        straddle_tiles(xc, zc, p.sx, p.ox, tiles_x_all, b.tile, W, lox, hix);
        straddle_tiles(yc, zc, p.sy, p.oy, tiles_y_all, b.tile, H, loy, hiy);
    }
    {
        // oriented box of the ellipsoid {x : |S^-1 R^T (x - p)| <= k}: centre +- k s_a col_a
        const float4 sd = b.sdens[j], q = b.quat[j], g0 = b.g0[j];
        const float k = sqrtf(2.0f * 0.6931471805599453f * b.hk[j]) * 1.0001f;
        float3 U, V, Wc;
        quat_to_columns(q, U, V, Wc);
        float3 e0 = U * (k * sd.x), e1 = V * (k * sd.y), e2 = Wc * (k * sd.z);
        to_camera(p, g0.x, g0.y, g0.z, mid.x, mid.y, mid.z);
        box_corners(mid, turn_to_camera(p, e0.x, e0.y, e0.z), turn_to_camera(p, e1.x, e1.y, e1.z), turn_to_camera(p, e2.x, e2.y, e2.z), xc, yc, zc);
        float olx, ohx, oly, ohy;
        int okind = project_corners(p, xc, yc, zc, olx, ohx, oly, ohy);
        if (okind == 0) return 0;
        if (okind == 2) {
            straddle_tiles(xc, zc, p.sx, p.ox, tiles_x_all, b.tile, W, olx, ohx);
            straddle_tiles(yc, zc, p.sy, p.oy, tiles_y_all, b.tile, H, oly, ohy);
        }
        lox = fmaxf(lox, olx); hix = fminf(hix, ohx); loy = fmaxf(loy, oly); hiy = fminf(hiy, ohy);
    }
    // rays sit at integer pixel coordinates; keep a small safety margin for rounding
    const float m = 0.02f;
    float fx0 = ceilf(lox - m - 1e-5f * fabsf(lox)), fx1 = floorf(hix + m + 1e-5f * fabsf(hix));
    float fy0 = ceilf(loy - m - 1e-5f * fabsf(loy)), fy1 = floorf(hiy + m + 1e-5f * fabsf(hiy));
    fx0 = fmaxf(fx0, 0.f); fx1 = fminf(fx1, (float)W - 1.f);
    fy0 = fmaxf(fy0, (float)b.row_begin); fy1 = fminf(fy1, (float)b.row_end - 1.f);
    if (!(fx0 <= fx1 && fy0 <= fy1)) return 0;
    const unsigned tx0 = (unsigned)fx0 / b.tile, tx1 = (unsigned)fx1 / b.tile;
    const unsigned ty0 = (unsigned)fy0 / b.tile - b.ty_first, ty1 = (unsigned)fy1 / b.tile - b.ty_first;
    rect = make_uint2(tx0 | (tx1 << 16), ty0 | (ty1 << 16));
    return (int)((tx1 - tx0 + 1) * (ty1 - ty0 + 1));
}

constexpr unsigned kWideTiles = 128;     // rectangles of more tiles are listed apart
__device__ __forceinline__ unsigned rect_tiles(uint2 r) { return ((r.x >> 16) - (r.x & 0xffffu) + 1u) * ((r.y >> 16) - (r.y & 0xffffu) + 1u); }
constexpr int kHistBits = 11;      // leading bits of the quantised near distance: its exponent bits and 3 to 6 of the mantissa
constexpr unsigned kNoRect = 0xffffffffu;

__device__ __forceinline__ unsigned hist_bucket(float tn, const KeyLayout& kl) {
    return near_quantised(tn, kl) >> (kl.near_bits - kHistBits);
}

// ---------------------------------------------------------------- culled emission
//
// Rays that end early -- those of a training view, of a dense scene -- look at the beginning of their tile's list
// only.  Such a view's lists need only hold the pairs that begin before a horizon (about near_target of them), and
// the pairs beyond need not even be emitted.  A recording forward lists the rays that reach the horizon after all,
// and march_forward_listed_rays_kernel finishes them by a search of the hierarchy; a forward that records nothing puts
// those rays aside and takes them up again with the complete lists of their tiles (b.tile_flag) -- lists in two depths
// (march_lists.cu).  The horizon is picked before the emission, on the device, from what is cheap to know of a Gaussian:
// the rectangle of tiles it can touch (an upper bound of its pairs) and a lower bound of the distance at which any
// of its pairs begins.  bin_near_hist_kernel: those two per Gaussian, and their histogram; bin_pick_horizon_kernel:
// the bucket at which the running sum reaches the target; the emission kernels then skip Gaussians and pairs that
// lie in later buckets and note, per tile, that something was skipped (tile_more; for a skipped Gaussian all tiles
// of its rectangle, added up from rectangle corners by bin_tile_more_kernel).

__global__ void __launch_bounds__(kEmitThreads) bin_near_hist_kernel(BinLaunch b) {
    after_previous();
    __shared__ unsigned int local[1 << kHistBits];
    for (int i = threadIdx.x; i < (1 << kHistBits); i += kEmitThreads) local[i] = 0u;
    __syncthreads();
    const int j = blockIdx.x * kEmitThreads + threadIdx.x;
    uint2 rect = make_uint2(kNoRect, 0u);
    unsigned code = 0u;
    if (j < b.n) {
        const float2 bx = b.bx[j], by = b.by[j], bz = b.bz[j];
        if (bx.x <= bx.y) {
            const Projector& p = b.proj;
            const KeyLayout kl = key_layout(b.tiles_x * ((b.cam.height + b.tile - 1) / b.tile), b.n_pad);
            uint2 r;
            const int count = gaussian_rect(b, p, j, bx, by, bz, r);
            if (count > 0) {
                // No pair of this Gaussian begins before `gn`: a pair's near distance is where the tile's central ray
                // enters the box grown by far_box * chord (pair_range), a point no nearer to the eye than the box less
                // sqrt(3) times that; the margins are ten times those pair_range takes off.
                const float* e = b.cam.eye;
                const float dx = fmaxf(fmaxf(bx.x - e[0], e[0] - bx.y), 0.f), dy = fmaxf(fmaxf(by.x - e[1], e[1] - by.y), 0.f),
                            dz = fmaxf(fmaxf(bz.x - e[2], e[2] - bz.y), 0.f);
                const float infl = box_far_distance(e, bx, by, bz) * __uint_as_float(b.pick->chord_bits) * 1.0001f + 1e-6f;
                const float gn = fmaxf((sqrtf(dx * dx + dy * dy + dz * dz) - 1.7321f * infl) * (1.0f - 1e-4f) - 1e-4f, 0.f);
                code = hist_bucket(gn, kl);
                rect = r;
                atomicAdd(&local[code], (unsigned)count);
            }
        }
    }
    if (j < b.n_pad) { b.g_rect[j] = rect; b.g_code[j] = code; }
    __syncthreads();
    for (int i = threadIdx.x; i < (1 << kHistBits); i += kEmitThreads)
        if (local[i]) atomicAdd(&b.near_hist[i], (unsigned long long)local[i]);
}

// The cut: the last non-empty bucket up to which the estimated pairs stay within the target (the first non-empty
// one if none does).  Everything is kept (cut = kAllBuckets) when the view has fewer than near_min_total estimated
// pairs or the cut would keep all of them (half of them or more, with near_half).
__global__ void __launch_bounds__(1024) bin_pick_horizon_kernel(BinLaunch b) {
    after_previous();
    using Scan = cub::BlockScan<unsigned long long, 1024>;
    __shared__ typename Scan::TempStorage scan_tmp;
    __shared__ int s_cut, s_first;
    const int t = threadIdx.x;
    const unsigned long long h0 = b.near_hist[2 * t], h1 = b.near_hist[2 * t + 1];
    unsigned long long incl, total;
    if (t == 0) { s_cut = -1; s_first = 1 << kHistBits; }
    __syncthreads();
    Scan(scan_tmp).InclusiveSum(h0 + h1, incl, total);
    const unsigned long long p0 = incl - h1, p1 = incl;
    if (h0) { atomicMin(&s_first, 2 * t); if (p0 <= b.near_target) atomicMax(&s_cut, 2 * t); }
    if (h1) { atomicMin(&s_first, 2 * t + 1); if (p1 <= b.near_target) atomicMax(&s_cut, 2 * t + 1); }
    __syncthreads();
    const int cut = s_cut >= 0 ? s_cut : s_first;
    if (t == 0) b.pick->est_total = total;
    if (cut >= (1 << kHistBits)) { if (t == 0) { b.pick->cut = kAllBuckets; b.pick->est_kept = total; } return; }
    if (t == (cut >> 1)) {
        const unsigned long long kept = (cut & 1) ? p1 : p0;
        const bool partial = total >= b.near_min_total && (b.near_half ? kept * 2 < total : kept < total) &&
                             cut + 1 < (1 << kHistBits);
        b.pick->cut = partial ? (unsigned)cut : kAllBuckets;
        b.pick->est_kept = partial ? kept : total;
    }
}

// Sorts the Gaussians into those before the cut (their slots gathered in kept_slot, so that the emission works on
// full blocks of them) and those beyond it (the corners of their rectangles go into tile_diff).  Few blocks, each with the
// corners of all its Gaussians in shared memory and one atomic per 1024 of them for the list: one atomic per warp and four
// per Gaussian, all on the same few thousand addresses, took 131 us for 1 M Gaussians and 604 us for 7 M (now 9 and 47).
constexpr int kDiffShared = 11900;
constexpr int kCompactThreads = 1024;
__global__ void __launch_bounds__(kCompactThreads) bin_compact_kernel(BinLaunch b) {
    after_previous();
    __shared__ int s_diff[kDiffShared];
    __shared__ unsigned s_count[2][kCompactThreads / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned cut = b.pick->cut;
    const int Wd = b.tiles_x + 1, cells = Wd * (b.tiles_y + 1);
    const bool local = cells <= kDiffShared;
    int* diff = local ? s_diff : b.tile_diff;
    for (int i = t; local && i < cells; i += kCompactThreads) s_diff[i] = 0;
    __syncthreads();
    for (int base = blockIdx.x * kCompactThreads; base < b.n; base += gridDim.x * kCompactThreads) {
        const int j = base + t;
        bool keep = false, wide = false;
        if (j < b.n) {
            const uint2 rect = b.g_rect[j];
            if (rect.x != kNoRect) {
                if (b.g_code[j] > cut) {            // every pair of this Gaussian begins beyond the horizon
                    const unsigned tx0 = rect.x & 0xffffu, tx1 = rect.x >> 16, ty0 = rect.y & 0xffffu, ty1 = rect.y >> 16;
                    atomicAdd(&diff[ty0 * Wd + tx0], 1);
                    atomicAdd(&diff[ty0 * Wd + tx1 + 1], -1);
                    atomicAdd(&diff[(ty1 + 1) * Wd + tx0], -1);
                    atomicAdd(&diff[(ty1 + 1) * Wd + tx1 + 1], 1);
                } else {
                    wide = rect_tiles(rect) > kWideTiles;
                    keep = !wide;
                }
            }
        }
        const unsigned m = __ballot_sync(kFullMask, keep), mw = __ballot_sync(kFullMask, wide);
        if (lane == 0) { s_count[0][warp] = (unsigned)__popc(m); s_count[1][warp] = (unsigned)__popc(mw); }
        __syncthreads();
        if (warp < 2) {
            const unsigned c = s_count[warp][lane];
            unsigned incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const unsigned u = __shfl_up_sync(kFullMask, incl, o); if (lane >= o) incl += u; }
            unsigned at = 0;
            if (lane == 31 && incl) at = (unsigned)atomicAdd(b.total_dev + (warp == 0 ? 1 : 3), (unsigned long long)incl);
            s_count[warp][lane] = __shfl_sync(kFullMask, at, 31) + incl - c;
        }
        __syncthreads();
        if (keep) b.kept_slot[s_count[0][warp] + __popc(m & ((1u << lane) - 1u))] = j;
        if (wide) b.kept_slot[b.n_pad - 1 - (int)(s_count[1][warp] + __popc(mw & ((1u << lane) - 1u)))] = j;
        __syncthreads();
    }
    for (int i = t; local && i < cells; i += kCompactThreads)
        if (s_diff[i]) atomicAdd(&b.tile_diff[i], s_diff[i]);
}

// tile_diff holds +1 / -1 at the corners of the rectangles of the skipped Gaussians; its two-dimensional running
// sum is the number of skipped rectangles over each tile.
__global__ void __launch_bounds__(1024) bin_tile_more_kernel(BinLaunch b) {
    after_previous();
    __shared__ int s_diff[kDiffShared];
    const int W = b.tiles_x + 1, H = b.tiles_y + 1;
    int* d = b.tile_diff;
    if (W * H <= kDiffShared) {
        for (int i = threadIdx.x; i < W * H; i += blockDim.x) s_diff[i] = b.tile_diff[i];
        d = s_diff;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < H; r += blockDim.x) {
        int run = 0;
        for (int c = 0; c < W; ++c) { run += d[r * W + c]; d[r * W + c] = run; }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < b.tiles_x; c += blockDim.x) {
        int run = 0;
        for (int r = 0; r < b.tiles_y; ++r) {
            run += d[r * W + c];
            if (run > 0) b.tile_more[r * b.tiles_x + c] = 1;
        }
    }
}

// Complete emission, first step: every Gaussian's rectangle of tiles; those that have one are listed (big_slot,
// big_rect, those of many tiles from the back) for bin_emit_pairs_kernel.  (A culled emission has the rectangles from
// bin_near_hist_kernel and the list from bin_compact_kernel.)
__global__ void __launch_bounds__(kEmitThreads) bin_list_kernel(BinLaunch b) {
    after_previous();
    const int j = blockIdx.x * kEmitThreads + threadIdx.x, lane = threadIdx.x & 31;
    uint2 rect = make_uint2(kNoRect, 0u);
    bool keep = false;
    if (j < b.n) {
        const float2 bx = b.bx[j], by = b.by[j], bz = b.bz[j];
        if (bx.x <= bx.y) {
            const Projector& p = b.proj;
            keep = gaussian_rect(b, p, j, bx, by, bz, rect) > 0;
        }
    }
    const bool wide = keep && rect_tiles(rect) > kWideTiles;
    auto append = [&](bool mine, int counter) {
        const unsigned m = __ballot_sync(kFullMask, mine);
        if (!m) return;
        unsigned long long at = 0;
        if (lane == __ffs(m) - 1) at = atomicAdd(b.total_dev + counter, (unsigned long long)__popc(m));
        at = __shfl_sync(kFullMask, at, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1u));
        if (mine) {
            const size_t slot = counter == 3 ? (size_t)b.n_pad - 1 - (size_t)at : (size_t)at;
            b.big_slot[slot] = j;
            b.big_rect[slot] = rect;
        }
    };
    append(keep && !wide, 1);
    append(wide, 3);
}

// The pairs of the listed Gaussians.  Warps take the Gaussians a few at a time (one, where there are few for each), 32 tiles
// of a rectangle per step:
// the tile's central ray against the box and the ellipsoid, both grown by the tile's angular radius (pair_range),
// keeps the pairs in which some ray of the tile can meet the Gaussian.  Every warp gathers its pairs in a buffer
// of its own in shared memory and appends them with one atomic per 256; pairs past the capacity are counted but
// not written (the host then grows the arrays and runs the emission again).
// An earlier version walked the candidates of 256 Gaussians block-wide, one candidate per thread whatever
// Gaussian it belonged to, and left only Gaussians of more than 48 tiles to this kernel; the search for the
// candidate's Gaussian and a block-wide barrier per round cost more than the idle lanes of small rectangles do here
// (3 M-Gaussian step by that threshold: 96: 375.9 ms, 48: 371.9, 24: 364.9, 12: 363.7, 4: 362.4, 0: 361.7).
// CULL: the list is bin_compact_kernel's; single pairs that begin beyond the cut are dropped and their tile marked.
constexpr int kBigWarps = 8;
constexpr int kBigBuf = 256;
constexpr int kBigBatch = 8;

template <bool CULL>
__global__ void __launch_bounds__(kBigWarps * 32) bin_emit_pairs_kernel(BinLaunch b) {
    after_previous();
    const unsigned cut = CULL ? b.pick->cut : kAllBuckets;
    __shared__ unsigned long long s_keys[kBigWarps][kBigBuf];
    __shared__ float s_fars[kBigWarps][kBigBuf];
    __shared__ PairGeom s_geom[kBigWarps][kBigBatch];
    __shared__ uint2 s_rect[kBigWarps][kBigBatch];
    __shared__ int s_slot[kBigWarps][kBigBatch];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned long long* keys = s_keys[warp];
    float* fars = s_fars[warp];
    const unsigned long long nlisted = b.total_dev[1], nwide = b.total_dev[3];
    bool wide = true;                        // those of many tiles first, one at a time
    const KeyLayout kl = key_layout(b.tiles_x * ((b.cam.height + b.tile - 1) / b.tile), b.n_pad);
    int nbuf = 0;
    auto flush = [&]() {
        unsigned long long base = 0;
        if (lane == 0 && nbuf > 0) base = atomicAdd(b.total_dev, (unsigned long long)nbuf);
        base = __shfl_sync(kFullMask, base, 0);
        __syncwarp();
        for (int i = lane; i < nbuf; i += 32) {
            const unsigned long long k = base + (unsigned long long)i;
            const unsigned rank = atomicAdd(&b.tile_pcnt[(int)(keys[i] >> (kl.near_bits + kl.id_bits))], 1);
            if (k < b.pair_cap) { b.keys_in[k] = keys[i]; b.vals_in[k] = __float_as_uint(fars[i]); b.ranks[k] = rank; }
        }
        nbuf = 0;
        __syncwarp();
    };
    const unsigned long long warps = (unsigned long long)gridDim.x * kBigWarps;
    const int batch = (int)min(max(nlisted / (8ull * warps), 1ull), (unsigned long long)kBigBatch);
    int have = 0, next = 0;
    unsigned long long idx = 0;
    while (true) {
        if (next == have) {
            // the next few Gaussians, a lane for each: one atomic for them, and their loads in flight together
            if (wide) {
                if (lane == 0) idx = atomicAdd(b.total_dev + 4, 1ull);
                idx = __shfl_sync(kFullMask, idx, 0);
                wide = idx < nwide;
                idx = (unsigned long long)b.n_pad - 1ull - idx;
                have = 1;
            }
            if (!wide) {
                if (lane == 0) idx = atomicAdd(b.total_dev + 2, (unsigned long long)batch);
                idx = __shfl_sync(kFullMask, idx, 0);
                if (idx >= nlisted) break;
                have = (int)min((unsigned long long)batch, nlisted - idx);
            }
            next = 0;
            __syncwarp();
            if (lane < have) {
                const int j = CULL ? b.kept_slot[idx + lane] : b.big_slot[idx + lane];
                s_slot[warp][lane] = j;
                s_rect[warp][lane] = CULL ? b.g_rect[j] : b.big_rect[idx + lane];
                const float kk = sqrtf(2.0f * 0.6931471805599453f * b.hk[j]);
                s_geom[warp][lane] = make_pair_geom(b.cam.eye, b.bx[j], b.by[j], b.bz[j], b.g0[j], b.g1[j], b.g2[j], b.sdens[j], b.quat[j], kk);
            }
            __syncwarp();
        }
        const int j = s_slot[warp][next];
        const uint2 rect = s_rect[warp][next];
        const PairGeom g = s_geom[warp][next];
        ++next;
        const unsigned tx0 = rect.x & 0xffffu, tx1 = rect.x >> 16, ty0 = rect.y & 0xffffu, ty1 = rect.y >> 16;
        const unsigned w = tx1 - tx0 + 1, count = w * (ty1 - ty0 + 1);
        const float inv_w = 1.0f / (float)w;
        for (unsigned it0 = 0; it0 < count; it0 += 32) {
            const unsigned item = it0 + lane;
            bool keep = false;
            unsigned long long key = 0;
            float tf = 0.f;
            if (item < count) {
                const unsigned row = count < (1u << 22) ? __float2uint_rz(((float)item + 0.5f) * inv_w) : item / w;    // item / w either way
                const unsigned t = (ty0 + row) * (unsigned)b.tiles_x + tx0 + item - row * w;
                float tn = 0.f;
                keep = (!b.tile_flag || b.tile_flag[t] != 0) && pair_range(b.cam.eye, b.tile_dir[t], g, tn, tf);
                if (CULL && keep && hist_bucket(tn, kl) > cut) { keep = false; b.tile_more[t] = 1; }
                if (keep) key = pair_key(kl, t, tn, (unsigned)j);
            }
            const unsigned m = __ballot_sync(kFullMask, keep);
            if (nbuf + __popc(m) > kBigBuf) flush();
            if (keep) { const int at = nbuf + __popc(m & ((1u << lane) - 1u)); keys[at] = key; fars[at] = tf; }
            nbuf += __popc(m);
        }
    }
    flush();
}

// ---------------------------------------------------------------- lists that fit shared memory
//
// The emission has counted every tile's pairs and numbered each pair among them.  From that, one block lays the lists out
// (bin_layout_kernel: begin of each tile's pairs and of its padded list, the order of the tiles), the pairs are put in their tile's
// place (bin_place_kernel), and a block per tile sorts them and writes the list (bin_sort_tiles_kernel).  Three launches and two
// passes over the pairs in place of a radix sort of all of them by 48 bits (six passes and a histogram), the ranges, counts,
// scan, sort of the tiles, padding, scatter and summaries that follow it: some twenty launches.  Lists per view: 3 M-Gaussian
// window 0.63 -> 0.35 ms, 1 M at 640x360 0.51 -> 0.39, 30 k at 400x400 0.24 -> 0.17, 4 k at 64x64 0.18 -> 0.09 (launches and the
// host's wait bound the last two).  Lists of more than kSortLong pairs do not fit a block (12 bytes a pair in 227 KB); a view that
// has one takes the radix sort.

// (begin of tile t's pairs in tile_first, of its padded list in tile_pbegin, tiles by falling number of pairs in tile_order)
constexpr int kLayoutThreads = 1024;
__global__ void __launch_bounds__(kLayoutThreads) bin_layout_kernel(BinLaunch b, int ntiles) {
    after_previous();
    using Scan = cub::BlockScan<int2, kLayoutThreads>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int s_bucket[256];
    __shared__ int s_longest, s_many;
    const int t = threadIdx.x;
    if (t == 0) { s_longest = 0; s_many = 0; }
    if (t < 256) s_bucket[t] = 0;
    __syncthreads();
    int2 carry = make_int2(0, 0);
    int longest = 0, many = 0;
    for (int base = 0; base <= ntiles; base += kLayoutThreads) {
        const int i = base + t, n = i < ntiles ? b.tile_pcnt[i] : 0;
        int2 at, sum;
        Scan(tmp).ExclusiveScan(make_int2(n, (n + 31) & ~31), at, make_int2(0, 0), [](int2 x, int2 y) { return make_int2(x.x + y.x, x.y + y.y); }, sum);
        if (i <= ntiles) { b.tile_first[i] = carry.x + at.x; b.tile_pbegin[i] = carry.y + at.y; }
        if (i < ntiles) b.tile_cnt[i] = n;
        carry = make_int2(carry.x + sum.x, carry.y + sum.y);
        longest = max(longest, n);
        many += n > kSortShort ? 1 : 0;
        __syncthreads();
    }
    longest = __reduce_max_sync(kFullMask, longest);
    many = __reduce_add_sync(kFullMask, many);
    if ((t & 31) == 0) { atomicMax(&s_longest, longest); if (many) atomicAdd(&s_many, many); }
    __syncthreads();
    longest = s_longest;
    if (t == 0) {
        // to the host without a copy behind this kernel: the host waits for it, and a copy takes ten microseconds to get going
        BinResult r = *b.result;
        r.longest = (unsigned)longest;
        r.long_tiles = (unsigned)s_many;
        *b.result_host = r;
    }
    // Buckets by length, the longest first; bucket boundaries put every list of more than kSortShort pairs before all others.
    auto bucket = [&](int n) {
        if (n > kSortShort) return 127 - (int)((long long)(n - kSortShort) * 127 / max(longest - kSortShort, 1));
        return 255 - n * 127 / kSortShort;
    };
    for (int i = t; i < ntiles; i += kLayoutThreads) atomicAdd(&s_bucket[bucket(b.tile_pcnt[i])], 1);
    __syncthreads();
    if (t < 32) {                                                        // exclusive scan of 256 counts by one warp
        int run = 0;
        for (int k = 0; k < 256; k += 32) {
            int v = s_bucket[k + t], incl = v;
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(kFullMask, incl, o); if (t >= o) incl += u; }
            s_bucket[k + t] = run + incl - v;
            run += __shfl_sync(kFullMask, incl, 31);
        }
    }
    __syncthreads();
    for (int i = t; i < ntiles; i += kLayoutThreads) b.tile_order[atomicAdd(&s_bucket[bucket(b.tile_pcnt[i])], 1)] = i;
}

__global__ void __launch_bounds__(256) bin_place_kernel(BinLaunch b, int total, int tile_shift) {
    after_previous();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= total) return;
    const uint64_t key = b.keys_in[k];
    const int dest = b.tile_first[(int)(key >> tile_shift)] + (int)b.ranks[k];
    b.keys_out[dest] = key;
    b.vals_out[dest] = b.vals_in[k];
}

// A block sorts the pairs of one tile by (near, slot) -- distinct keys, so the order does not depend on that of emission -- and writes
// its list, padded to blocks of 32 with empty ranges, and the block summaries.  The pairs are dealt into kSortBuckets buckets by
// near distance, about one pair each, and ranked inside their bucket by comparison; where many share a distance (an eye inside
// many Gaussians) a bucket would be too long for that, and the block sorts with a bitonic network.  1024 threads for the lists of
// more than kSortShort pairs, of which an SM holds few blocks; 256 for the others, eight blocks an SM.
constexpr int kSortCrowd = 96;
__host__ __device__ constexpr size_t sort_smem(int cap) { return (size_t)cap * (8 + 4) + (size_t)(cap / 32) * 4; }
template <int kSortThreads, int kSortBuckets>
__global__ void __launch_bounds__(kSortThreads) bin_sort_tiles_kernel(BinLaunch b, KeyLayout kl, int first_unit, int cap) {
    after_previous();
    extern __shared__ __align__(16) unsigned char sort_mem[];
    uint64_t* key = reinterpret_cast<uint64_t*>(sort_mem);               // [cap] near | slot
    unsigned* at = reinterpret_cast<unsigned*>(key + cap);               // [cap] pair numbers by bucket, or in order
    unsigned* far_max = at + cap;                                        // [cap / 32]
    __shared__ unsigned s_start[kSortBuckets];
    __shared__ unsigned s_lo, s_hi, s_most, s_warp[kSortThreads / 32];
    const int t = threadIdx.x, lane = t & 31;
    const int tile = b.tile_order[first_unit + blockIdx.x];
    const int n = b.tile_cnt[tile];
    if (n == 0) return;
    const int seg = b.tile_first[tile], out = b.tile_pbegin[tile];
    const uint64_t mask = (1ull << (kl.near_bits + kl.id_bits)) - 1ull;
    for (int i = t; i < kSortBuckets; i += kSortThreads) s_start[i] = 0u;
    for (int i = t; i < (n + 31) / 32; i += kSortThreads) far_max[i] = 0u;
    if (t == 0) { s_lo = ~0u; s_hi = 0u; s_most = 0u; }
    __syncthreads();
    unsigned lo = ~0u, hi = 0u;
    for (int i = t; i < n; i += kSortThreads) {
        const uint64_t k = b.keys_out[seg + i] & mask;
        key[i] = k;
        const unsigned q = (unsigned)(k >> kl.id_bits);
        lo = min(lo, q); hi = max(hi, q);
    }
    lo = __reduce_min_sync(kFullMask, lo); hi = __reduce_max_sync(kFullMask, hi);
    if (lane == 0) { atomicMin(&s_lo, lo); atomicMax(&s_hi, hi); }
    __syncthreads();
    lo = s_lo;
    const float scale = (float)kSortBuckets / (float)(s_hi - lo + 1u);
    auto bucket = [&](uint64_t k) { return min((int)((float)((unsigned)(k >> kl.id_bits) - lo) * scale), kSortBuckets - 1); };   // monotone in the distance
    for (int i = t; i < n; i += kSortThreads) atomicAdd(&s_start[bucket(key[i])], 1u);
    __syncthreads();
    // exclusive scan of the buckets, eight per thread
    constexpr int kPer = kSortBuckets / kSortThreads;
    unsigned c[kPer], sum = 0u, most = 0u;
#pragma unroll
    for (int k = 0; k < kPer; ++k) { c[k] = s_start[t * kPer + k]; sum += c[k]; most = max(most, c[k]); }
    unsigned incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const unsigned u = __shfl_up_sync(kFullMask, incl, o); if (lane >= o) incl += u; }
    if (lane == 31) s_warp[t >> 5] = incl;
    most = __reduce_max_sync(kFullMask, most);
    if (lane == 0) atomicMax(&s_most, most);
    __syncthreads();
    unsigned run = incl - sum;
    for (int w = 0; w < (t >> 5); ++w) run += s_warp[w];
#pragma unroll
    for (int k = 0; k < kPer; ++k) { s_start[t * kPer + k] = run; run += c[k]; }
    __syncthreads();
    const bool crowded = s_most > (unsigned)kSortCrowd;
    if (crowded) {
        int size = 1;
        while (size < n) size <<= 1;
        for (int i = t; i < size; i += kSortThreads) at[i] = (unsigned)i;                  // numbers past the end compare as largest
        __syncthreads();
        auto value = [&](unsigned i) { return i < (unsigned)n ? key[i] : ~0ull; };
        for (int k = 2; k <= size; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int p = t; p < size / 2; p += kSortThreads) {
                    const int x = ((p & ~(j - 1)) << 1) | (p & (j - 1)), y = x | j;
                    const unsigned ax = at[x], ay = at[y];
                    if ((value(ax) > value(ay)) == ((x & k) == 0)) { at[x] = ay; at[y] = ax; }
                }
                __syncthreads();
            }
    } else {
        for (int i = t; i < n; i += kSortThreads) at[atomicAdd(&s_start[bucket(key[i])], 1u)] = (unsigned)i;    // s_start: now the ends
        __syncthreads();
    }
    for (int p = t; p < n; p += kSortThreads) {
        const unsigned i = at[p];
        const uint64_t k = key[i];
        int rank = p;
        if (!crowded) {
            const int w = bucket(k), begin = w ? (int)s_start[w - 1] : 0, end = (int)s_start[w];
            rank = begin;
            for (int q = begin; q < end; ++q) rank += key[at[q]] < k ? 1 : 0;
        }
        const float near = near_stored((unsigned)(k >> kl.id_bits), kl);
        const unsigned far = b.vals_out[seg + i];
        b.ent_id[out + rank] = (int)(k & ((1ull << kl.id_bits) - 1ull));
        b.ent_range[out + rank] = make_float2(near, __uint_as_float(far));
        atomicMax(&far_max[rank >> 5], far);                                               // distances: positive, ordered like their bits
        if ((rank & 31) == 0) b.blk[(out + rank) >> 5].x = near;
    }
    for (int i = n + t; i < ((n + 31) & ~31); i += kSortThreads) {
        b.ent_id[out + i] = 0;
        b.ent_range[out + i] = make_float2(INFINITY, -INFINITY);
    }
    __syncthreads();
    for (int i = t; i < (n + 31) / 32; i += kSortThreads) b.blk[(out >> 5) + i].y = __uint_as_float(far_max[i]);
}

// ---------------------------------------------------------------- lists of any length: after the radix sort
__global__ void bin_tile_iota_kernel(BinLaunch b, int ntiles) {
    after_previous();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ntiles) b.tile_iota[t] = t;
}

__global__ void __launch_bounds__(256) bin_fill_kernel(BinLaunch b, size_t n_entries) {
    after_previous();
    size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_entries) return;
    b.ent_id[k] = 0;
    b.ent_range[k] = make_float2(INFINITY, -INFINITY);
}

__global__ void __launch_bounds__(256) bin_scatter_kernel(BinLaunch b, int total, KeyLayout kl) {
    after_previous();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= total) return;
    const uint64_t key = b.keys_out[k];
    const int t = (int)(key >> (kl.near_bits + kl.id_bits));
    const size_t dest = (size_t)b.tile_pbegin[t] + (size_t)(k - b.tile_first[t]);
    b.ent_id[dest] = (int)(key & ((1ull << kl.id_bits) - 1ull));
    const unsigned q = (unsigned)((key >> kl.id_bits) & ((1ull << kl.near_bits) - 1ull));
    b.ent_range[dest] = make_float2(near_stored(q, kl), __uint_as_float(b.vals_out[k]));
}

// One warp per block of 32 entries: nearest near distance and farthest far distance.
__global__ void __launch_bounds__(256) bin_blocks_kernel(BinLaunch b, size_t n_blocks) {
    after_previous();
    size_t blk = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (blk >= n_blocks) return;
    float2 r = b.ent_range[blk * 32 + lane];
    float lo = r.x, hi = r.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(kFullMask, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(kFullMask, hi, o));
    }
    if (lane == 0) b.blk[blk] = make_float2(lo, hi);
}

}  // namespace

size_t binning_cub_temp_bytes(size_t pair_cap, int ntiles) {
    size_t a = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, a, (const uint64_t*)nullptr, (uint64_t*)nullptr, (const uint32_t*)nullptr,
                                    (uint32_t*)nullptr, (int64_t)pair_cap, 0, 64, (cudaStream_t)0);
    size_t o = 0;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, o, (const int*)nullptr, (int*)nullptr, (const int*)nullptr,
                                              (int*)nullptr, ntiles, 0, 32, (cudaStream_t)0);
    return o > a ? o : a;
}

// The view's projection, the same for every Gaussian: made once on the host.
Projector make_projector(const BinLaunch& b) {
    Projector p;
    for (int k = 0; k < 3; ++k) { p.eye[k] = b.cam.eye[k]; p.du[k] = b.dual[0][k]; p.dv[k] = b.dual[1][k]; p.dw[k] = b.dual[2][k]; }
    p.sx = (float)b.cam.width / (2.0f * b.cam.tan_half_fov[0]);
    p.sy = (float)b.cam.height / (2.0f * b.cam.tan_half_fov[1]);
    p.ox = b.cam.pp[0] * (float)b.cam.width - 0.5f;
    p.oy = b.cam.pp[1] * (float)b.cam.height - 0.5f;
    // a point eye + t (a u + b v + w), t > 0, of a ray of the rows at hand has a within [a0, a1] and b within [b0, b1]
    // (one pixel of margin), that is x_c - a0 z_c >= 0, a1 z_c - x_c >= 0 and the same for rows
    const float a0 = (-1.0f - p.ox) / p.sx, a1 = ((float)b.cam.width - p.ox) / p.sx;
    const float b0 = ((float)b.row_begin - 1.0f - p.oy) / p.sy, b1 = ((float)b.row_end - p.oy) / p.sy;
    for (int k = 0; k < 3; ++k) {
        p.plane[0][k] = p.du[k] - a0 * p.dw[k];
        p.plane[1][k] = a1 * p.dw[k] - p.du[k];
        p.plane[2][k] = p.dv[k] - b0 * p.dw[k];
        p.plane[3][k] = b1 * p.dw[k] - p.dv[k];
    }
    for (int q = 0; q < 4; ++q)
        p.plane[q][3] = std::sqrt(p.plane[q][0] * p.plane[q][0] + p.plane[q][1] * p.plane[q][1] + p.plane[q][2] * p.plane[q][2]);
    return p;
}

// Phase 1: all (tile, Gaussian) pairs -- with b.pick those that begin before the horizon picked on the way --,
// unsorted, and their number in b.total_dev (which keeps counting past b.pair_cap; the caller reads it back and
// repeats the phase with more room if needed).
cudaError_t launch_bin_emit(const BinLaunch& b, cudaStream_t s) {
    const int tb = 256;
    const int ntiles = b.tiles_x * b.tiles_y;
    cudaError_t e;
    if ((e = cudaMemsetAsync(b.zero, 0, b.zero_bytes, s)) != cudaSuccess) return e;
    const int blocks = (b.n_pad + kEmitThreads - 1) / kEmitThreads;
    if (b.pick) {
        // only the pairs that begin before a horizon, which is picked on the way (see bin_near_hist_kernel)
        const KeyLayout kl = key_layout(b.tiles_x * ((b.cam.height + b.tile - 1) / b.tile), b.n_pad);
        if (kl.near_bits < kHistBits) return cudaErrorInvalidValue;
        launch_after(bin_tile_dirs_kernel, (ntiles + tb - 1) / tb, tb, 0, s, b, ntiles);
        launch_after(bin_near_hist_kernel, blocks, kEmitThreads, 0, s, b);
        launch_after(bin_pick_horizon_kernel, 1, 1024, 0, s, b);
        launch_after(bin_compact_kernel, std::min((b.n + kCompactThreads - 1) / kCompactThreads, 2 * b.sm_count), kCompactThreads, 0, s, b);
        launch_after(bin_emit_pairs_kernel<true>, b.big_grid, kBigWarps * 32, 0, s, b);
        launch_after(bin_tile_more_kernel, 1, 1024, 0, s, b);
        launch_after(bin_layout_kernel, 1, kLayoutThreads, 0, s, b, ntiles);
        return cudaGetLastError();
    }
    launch_after(bin_tile_dirs_kernel, (ntiles + tb - 1) / tb, tb, 0, s, b, ntiles);
    launch_after(bin_list_kernel, blocks, kEmitThreads, 0, s, b);
    launch_after(bin_emit_pairs_kernel<false>, b.big_grid, kBigWarps * 32, 0, s, b);
    launch_after(bin_layout_kernel, 1, kLayoutThreads, 0, s, b, ntiles);
    return cudaGetLastError();
}

// Phase 2: the pairs of every tile in order, padded layout, block summaries.  r: what the emission left for the host.
cudaError_t launch_bin_fill(const BinLaunch& b, int total, const BinResult& r, cudaStream_t s) {
    const int tb = 256;
    const int ntiles = b.tiles_x * b.tiles_y;
    if (total == 0) return cudaSuccess;                    // every list is empty: the counts say so
    // the layout is that of the whole image whatever the row range, so that a row range sees the same order
    const KeyLayout kl = key_layout(b.tiles_x * ((b.cam.height + b.tile - 1) / b.tile), b.n_pad);
    if (r.longest <= (unsigned)kSortLong) {
        launch_after(bin_place_kernel, (total + tb - 1) / tb, tb, 0, s, b, total, kl.near_bits + kl.id_bits);
        int cap = kSortShort;
        while (cap < (int)r.longest) cap <<= 1;
        if (r.long_tiles) {                                // tile_order has these first
            cudaError_t e = cudaFuncSetAttribute(bin_sort_tiles_kernel<1024, 4096>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_smem(kSortLong));
            if (e != cudaSuccess) return e;
            launch_after((bin_sort_tiles_kernel<1024, 4096>), r.long_tiles, 1024, sort_smem(cap), s, b, kl, 0, cap);
        }
        if ((int)r.long_tiles < ntiles)
            launch_after((bin_sort_tiles_kernel<256, 2048>), ntiles - (int)r.long_tiles, 256, sort_smem(kSortShort), s, b, kl, (int)r.long_tiles, kSortShort);
        return cudaGetLastError();
    }
    cudaError_t e;
    size_t temp = b.cub_bytes;
    e = cub::DeviceRadixSort::SortPairs(b.cub_temp, temp, b.keys_in, b.keys_out, b.vals_in, b.vals_out, (int64_t)total, 0,
                                        kl.tile_bits + kl.near_bits + kl.id_bits, s);
    if (e != cudaSuccess) return e;
    // CTAs take the tiles with the longest lists first: the march ends with short tiles, not with one long one
    launch_after(bin_tile_iota_kernel, (ntiles + tb - 1) / tb, tb, 0, s, b, ntiles);
    temp = b.cub_bytes;
    if ((e = cub::DeviceRadixSort::SortPairsDescending(b.cub_temp, temp, b.tile_cnt, b.tile_cnt_sorted, b.tile_iota, b.tile_order,
                                                       ntiles, 0, 32, s)) != cudaSuccess) return e;
    const size_t n_entries = (((size_t)total + 32u * (size_t)ntiles + 31) / 32) * 32;   // upper bound of the padded layout
    launch_after(bin_fill_kernel, (unsigned)((n_entries + tb - 1) / tb), tb, 0, s, b, n_entries);
    launch_after(bin_scatter_kernel, (total + tb - 1) / tb, tb, 0, s, b, total, kl);
    const size_t n_blocks = (n_entries + 31) / 32;
    launch_after(bin_blocks_kernel, (unsigned)((n_blocks + 7) / 8), 256, 0, s, b, n_blocks);
    return cudaGetLastError();
}

// Upper end of histogram bucket `bucket` as a distance: every pair in buckets <= bucket begins before it.
float bin_hist_bucket_end(const BinLaunch& b, int bucket) {
    const KeyLayout kl = key_layout(b.tiles_x * ((b.cam.height + b.tile - 1) / b.tile), b.n_pad);
    // bucket = the leading kHistBits bits of the quantised distance; the next bucket's smallest code bounds this one
    if (bucket + 1 >= (1 << kHistBits)) return INFINITY;
    return near_stored((unsigned)(bucket + 1) << (kl.near_bits - kHistBits), kl);
}

}  // namespace rgx
