// splat.cu — headless particle splatting: SurfaceReconstruction's two
// particle passes (src/SurfaceReconstruction.cpp:176-231) as CUDA kernels
// writing device buffers instead of GL framebuffers.
//
//  depth      shaders/particledepth/{vertex,fragment}.glsl: each particle is a
//             view-aligned quad of half-size 0.1 (two triangles, PointSprite's
//             indices 0,2,1 / 2,0,3, src/PointSprite.cpp:33-55); a fragment
//             inside the unit disc of its texture coordinate writes the
//             depth of the sphere surface, clip z / clip w, clamped to
//             [0, 1]; the depth test keeps the smallest (cleared to 1).
//  thickness  shaders/thickness/{vertex,fragment}.glsl with noise off: every
//             fragment inside the disc adds 1 (additive blending, no depth
//             test; cleared to 0).
//
// Rasterisation follows the GL rules the reference relies on: the viewport
// transform xw = (W/2) xd + W/2, pixel centres at (i + 1/2, j + 1/2), row 0
// at the bottom, a pixel centre on a shared edge owned by exactly one
// triangle (top-left rule in window coordinates with y up), attributes
// interpolated perspective-correctly, and primitives clipped to the near and
// far planes (-w <= z <= w).  Every floating-point step is one explicitly
// rounded operation in a fixed order, so the CPU oracle reproduces the
// output bit for bit; both outputs are order-independent (a minimum and an
// exact count), so thread scheduling cannot change them.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/pbf.h"
#include "internal.h"
#include "sim.h"

namespace pbf {
namespace {

__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }

struct View {
    float V[16], P[16];  // column-major: m[4 * column + row]
};

// mat4 * vec4 as GLSL evaluates it: column 0 * x + column 1 * y + column 2 * z
// + column 3 * w, summed left to right, one rounding per operation.
__device__ __forceinline__ float4 mul4(const float* m, float4 v) {
    float4 r;
    r.x = fa(fa(fa(fm(m[0], v.x), fm(m[4], v.y)), fm(m[8], v.z)), fm(m[12], v.w));
    r.y = fa(fa(fa(fm(m[1], v.x), fm(m[5], v.y)), fm(m[9], v.z)), fm(m[13], v.w));
    r.z = fa(fa(fa(fm(m[2], v.x), fm(m[6], v.y)), fm(m[10], v.z)), fm(m[14], v.w));
    r.w = fa(fa(fa(fm(m[3], v.x), fm(m[7], v.y)), fm(m[11], v.z)), fm(m[15], v.w));
    return r;
}

// Edge function of (a -> b) at p, in window coordinates.
__device__ __forceinline__ float edge(float ax, float ay, float bx, float by, float px, float py) {
    return fs(fm(fs(bx, ax), fs(py, ay)), fm(fs(by, ay), fs(px, ax)));
}

// Does a pixel centre exactly on edge (a -> b) of a counter-clockwise
// triangle (y up) belong to it?  Top edges (horizontal, traversed towards -x)
// and left edges (traversed towards -y) do.
__device__ __forceinline__ bool owns_edge(float ax, float ay, float bx, float by) {
    return (ay == by && bx < ax) || by < ay;
}

__device__ __forceinline__ bool inside(float e, bool own) { return e > 0.0f || (e == 0.0f && own); }

// A projected particle: the quad's corners k = 0..3 at (-1, 1), (1, 1),
// (1, -1), (-1, -1) in window coordinates with clip w and z, the two view-space
// x and y of the corners and their z, the pixel box, a lower bound of the depths
// its fragments can write and a bound on the error of their estimates.
struct Sprite {
    float x[4], y[4], w[4], cz[4];
    float xm, xp, ym, yp, z;
    float dlow, margin;
    int x0, x1, y0, y1;
    bool clip;  // straddles the near or far plane
};

// One of the quad's triangles (PointSprite indices 0,2,1 and 2,0,3), made
// counter-clockwise in window coordinates.
struct Tri {
    float ax, ay, bx, by, cx, cy, area;
    float ka, kb, kc;       // about 1 / (area w) of a, b, c
    bool own0, own1, own2;  // of the edges opposite a, b, c
    bool swapped;           // b and c exchanged
    bool ok;
};

__device__ __forceinline__ Tri make_tri(const Sprite& q, int i0, int i1, int i2) {
    Tri t;
    t.area = edge(q.x[i0], q.y[i0], q.x[i1], q.y[i1], q.x[i2], q.y[i2]);
    t.ok = !(t.area == 0.0f || t.area != t.area);
    t.swapped = t.area < 0.0f;
    if (t.swapped) t.area = -t.area;
    t.ax = q.x[i0];
    t.ay = q.y[i0];
    t.bx = t.swapped ? q.x[i2] : q.x[i1];
    t.by = t.swapped ? q.y[i2] : q.y[i1];
    t.cx = t.swapped ? q.x[i1] : q.x[i2];
    t.cy = t.swapped ? q.y[i1] : q.y[i2];
    const float ia = __fdividef(1.0f, t.area);
    const float k1 = __fdividef(ia, q.w[i1]), k2 = __fdividef(ia, q.w[i2]);
    t.ka = __fdividef(ia, q.w[i0]);
    t.kb = t.swapped ? k2 : k1;
    t.kc = t.swapped ? k1 : k2;
    t.own0 = owns_edge(t.bx, t.by, t.cx, t.cy);
    t.own1 = owns_edge(t.cx, t.cy, t.ax, t.ay);
    t.own2 = owns_edge(t.ax, t.ay, t.bx, t.by);
    return t;
}

__device__ __forceinline__ bool covers(const Tri& t, float px, float py, float3& e) {
    e.x = edge(t.bx, t.by, t.cx, t.cy, px, py);
    e.y = edge(t.cx, t.cy, t.ax, t.ay, px, py);
    e.z = edge(t.ax, t.ay, t.bx, t.by, px, py);
    return t.ok && inside(e.x, t.own0) && inside(e.y, t.own1) && inside(e.z, t.own2);
}

// Lower bound of the depths of a sprite's fragments, and of how far an estimate
// of one (fragment) can lie above the value.  A fragment's position is in the
// box of the corners' positions widened by 0.1 towards the eye
// (perspective-correct weights are not negative), and z / w has its extremes at
// corners of a box with w > 0.  The margins cover the rounding of the
// interpolation (1e-5 of the coordinates, and 0.1 sqrt(1e-5) in z where the
// sphere's edge turns away) and of the transform and division (64 units in the
// last place of the terms).
__device__ __forceinline__ void depth_bounds(Sprite& q, const View& view) {
    const float dd = 1e-5f * (fabsf(q.xm) + fabsf(q.ym) + fabsf(q.z) + 1.0f);
    const float lo[3] = {q.xm - 0.1f - dd, q.ym - 0.1f - dd, q.z - dd};
    const float hi[3] = {q.xp + 0.1f + dd, q.yp + 0.1f + dd, q.z + 0.1f + dd};
    float d = 3.0e38f, big = 1.0f, wmin = 3.0e38f, terms = 0.0f;
    q.dlow = -3.0e38f;
    q.margin = 3.0e38f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float x = k & 1 ? hi[0] : lo[0], y = k & 2 ? hi[1] : lo[1], z = k & 4 ? hi[2] : lo[2];
        const float z0 = view.P[2] * x, z1 = view.P[6] * y, z2 = view.P[10] * z;
        const float w0 = view.P[3] * x, w1 = view.P[7] * y, w2 = view.P[11] * z;
        const float cz = z0 + z1 + z2 + view.P[14], cw = w0 + w1 + w2 + view.P[15];
        const float za = fabsf(z0) + fabsf(z1) + fabsf(z2) + fabsf(view.P[14]);
        const float wa = fabsf(w0) + fabsf(w1) + fabsf(w2) + fabsf(view.P[15]);
        if (!(cw > 1e-4f * wa)) return;  // w may come near 0: no bound
        const float r = __fdividef(cz, cw);
        big = fmaxf(big, fabsf(r));
        terms = fmaxf(terms, za + fabsf(r) * wa);
        wmin = fminf(wmin, cw);
        d = fminf(d, r);
    }
    const float iw = __fdividef(1.0f, wmin);
    const float rounding = 4e-6f * terms * iw;
    const float dz = dd + 3.2e-4f;
    q.dlow = d - rounding;
    q.margin = rounding + iw * ((fabsf(view.P[2]) + big * fabsf(view.P[3])) * dd +
                                (fabsf(view.P[6]) + big * fabsf(view.P[7])) * dd +
                                (fabsf(view.P[10]) + big * fabsf(view.P[11])) * dz);
}

// Projects a particle; false when it is not drawn.
template <int PASS>
__device__ __forceinline__ bool make_sprite(const float4 p4, const View& view, uint32_t W,
                                            uint32_t H, Sprite& q) {
    // vertex shader: world position 0.2 p + 0.2 (-64, 1, -64) (vertex.glsl:41/42)
    const float4 c = make_float4(fa(fm(0.2f, p4.x), fm(0.2f, -64.0f)), fa(fm(0.2f, p4.y), fm(0.2f, 1.0f)),
                                 fa(fm(0.2f, p4.z), fm(0.2f, -64.0f)), 1.0f);
    const float4 m = mul4(view.V, c);
    // the corner offset's w: depth adds vec4(0.1 v, 0, 1), thickness adds
    // vec4(v, 0, 1) * 0.1 (the reference's w quirks, kept)
    const float ow = PASS == PBF_SPLAT_DEPTH ? 1.0f : 0.1f;
    const float hw = fm(0.5f, (float)W), hh = fm(0.5f, (float)H);
    q.xm = fa(m.x, fm(0.1f, -1.0f));
    q.xp = fa(m.x, fm(0.1f, 1.0f));
    q.ym = fa(m.y, fm(0.1f, -1.0f));
    q.yp = fa(m.y, fm(0.1f, 1.0f));
    q.z = fa(m.z, 0.0f);
    int near_out = 0, far_out = 0;
    float xmin = 3.0e38f, xmax = -3.0e38f, ymin = 3.0e38f, ymax = -3.0e38f;
    bool front = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 ps = make_float4(k == 0 || k == 3 ? q.xm : q.xp, k < 2 ? q.yp : q.ym, q.z,
                                      fa(m.w, ow));
        const float4 cl = mul4(view.P, ps);
        front = front && cl.w > 0.0f;  // a corner at or behind the eye: not drawn
        near_out += cl.z < -cl.w;
        far_out += cl.z > cl.w;
        q.x[k] = fa(fm(hw, fd(cl.x, cl.w)), hw);
        q.y[k] = fa(fm(hh, fd(cl.y, cl.w)), hh);
        q.w[k] = cl.w;
        q.cz[k] = cl.z;
        xmin = fminf(xmin, q.x[k]);
        xmax = fmaxf(xmax, q.x[k]);
        ymin = fminf(ymin, q.y[k]);
        ymax = fmaxf(ymax, q.y[k]);
    }
    if (!front || near_out == 4 || far_out == 4) return false;
    q.clip = near_out > 0 || far_out > 0;
    // pixel centres i + 0.5 inside [xmin, xmax]
    const float fx0 = ceilf(xmin - 0.5f), fx1 = floorf(xmax - 0.5f);
    const float fy0 = ceilf(ymin - 0.5f), fy1 = floorf(ymax - 0.5f);
    if (!(fx0 <= fx1) || !(fy0 <= fy1)) return false;
    if (fx1 < 0.0f || fy1 < 0.0f || fx0 >= (float)W || fy0 >= (float)H) return false;
    q.x0 = (int)fmaxf(fx0, 0.0f);
    q.x1 = (int)fminf(fx1, (float)W - 1.0f);
    q.y0 = (int)fmaxf(fy0, 0.0f);
    q.y1 = (int)fminf(fy1, (float)H - 1.0f);
    if (PASS == PBF_SPLAT_DEPTH) depth_bounds(q, view);
    return true;
}

// The fragment of a sprite at pixel (tx, ty): whether it lies on the disc
// (thickness) or, into `d`, its depth when that is below `seen`, the value read
// at the pixel.  The triangle that owns the pixel centre is found first and the
// attributes interpolated once, in it.
template <int PASS>
__device__ __forceinline__ bool fragment(const Sprite& q, const Tri& t0, const Tri& t1,
                                         const View& view, int tx, int ty, float seen, float& d) {
    const float px = (float)tx + 0.5f, py = (float)ty + 0.5f;
    float3 e, e1;
    const bool in0 = covers(t0, px, py, e), in1 = covers(t1, px, py, e1);
    if (!in0 && !in1) return false;  // (a pixel centre belongs to at most one)
    // corners a, b, c of the triangle: 0, 2, 1 or 2, 0, 3, the last two swapped
    // where the triangle was clockwise
    const bool sw = in0 ? t0.swapped : t1.swapped;
    if (!in0) e = e1;
    const float sx = in0 ? 1.0f : -1.0f;
    // the disc and the depth from unrounded weights first: within about 4e-6 of
    // the fragment's, so that only fragments on the disc's edge, and in the
    // depth pass those that may be in front, need the rounded ones
    bool edge_case = true;
    if (!q.clip) {
        const float m0 = e.x * (in0 ? t0.ka : t1.ka), m1 = e.y * (in0 ? t0.kb : t1.kb),
                    m2 = e.z * (in0 ? t0.kc : t1.kc);
        const float ms = m0 + m1 + m2, mu = sx * (m1 + m2 - m0),
                    mv = sx * (sw ? m0 + m1 - m2 : m0 - m1 + m2);
        const float over = mu * mu + mv * mv - ms * ms;  // (r - 1) ms^2
        edge_case = !(fabsf(over) > 1e-4f * (ms * ms));
        if (!edge_case && over > 0.0f) return false;
        if (PASS == PBF_SPLAT_THICKNESS && !edge_case) return true;
        if (PASS == PBF_SPLAT_DEPTH) {
            const float rs = __fdividef(1.0f, ms), eu = mu * rs, ev = mv * rs;
            const float ex = (in0 ? q.xm : q.xp) + (m1 + m2) * rs * (sx * (q.xp - q.xm)) - 0.1f * eu;
            const float ey = (in0 ? q.yp : q.ym) + (sw ? m2 : m1) * rs * (sx * (q.ym - q.yp)) - 0.1f * ev;
            const float ez = q.z + 0.1f * __fsqrt_rn(fmaxf(1.0f - eu * eu - ev * ev, 0.0f));
            const float ed = __fdividef(
                view.P[2] * ex + view.P[6] * ey + view.P[10] * ez + view.P[14],
                view.P[3] * ex + view.P[7] * ey + view.P[11] * ez + view.P[15]);
            if (ed - q.margin > seen) return false;
        }
    }
    const float area = in0 ? t0.area : t1.area;
    const float aw = in0 ? q.w[0] : q.w[2];
    const float u1w = in0 ? q.w[2] : q.w[0], u2w = in0 ? q.w[1] : q.w[3];
    const float bw = sw ? u2w : u1w, cw = sw ? u1w : u2w;
    // perspective-correct barycentric weights
    const float l0 = fd(fd(e.x, area), aw), l1 = fd(fd(e.y, area), bw), l2 = fd(fd(e.z, area), cw);
    const float ls = fa(fa(l0, l1), l2);
    auto interp = [&](float A, float B, float C) {
        return fd(fa(fa(fm(l0, A), fm(l1, B)), fm(l2, C)), ls);
    };
    // (B, C) of an attribute whose unswapped corners hold u1, u2
    auto at = [&](float A, float u1, float u2) {
        return interp(A, sw ? u2 : u1, sw ? u1 : u2);
    };
    if (q.clip) {
        const float zc = at(in0 ? q.cz[0] : q.cz[2], in0 ? q.cz[2] : q.cz[0],
                            in0 ? q.cz[1] : q.cz[3]);
        const float wc = at(aw, u1w, u2w);
        if (zc < -wc || zc > wc) return false;
    }
    // texture coordinates: corners 0, 2, 1 hold (-1, 1), (1, -1), (1, 1) and
    // corners 2, 0, 3 hold (1, -1), (-1, 1), (-1, -1)
    const float u = at(-sx, sx, sx), v = at(sx, -sx, sx);
    // fragment shader: r = dot(t, t); discard outside the disc
    const float r = fa(fm(u, u), fm(v, v));
    if (r > 1.0f) return false;
    if (PASS == PBF_SPLAT_THICKNESS) return true;
    // normal = (t, -sqrt(1 - r)); fPos = fPosition - 0.1 normal;
    // depth = (P fPos).z / (P fPos).w  (particledepth/fragment.glsl:40-46)
    const float nz = -__fsqrt_rn(fs(1.0f, r));
    const float x0 = in0 ? q.xm : q.xp, x1 = in0 ? q.xp : q.xm;
    const float y0 = in0 ? q.yp : q.ym, y1 = in0 ? q.ym : q.yp;
    const float4 fp = make_float4(fs(at(x0, x1, x1), fm(0.1f, u)), fs(at(y0, y1, y0), fm(0.1f, v)),
                                  fs(interp(q.z, q.z, q.z), fm(0.1f, nz)), 1.0f);
    const float4 cp = mul4(view.P, fp);
    d = fd(cp.z, cp.w);
    if (d != d) return false;  // NaN fragments are dropped
    d = d < 0.0f ? 0.0f : (d > 1.0f ? 1.0f : d);
    return d < seen;
}

// Depth pass.  A warp takes kGroup sprites, a share of its lanes each.  Where none
// of them has more than kSmallPixels pixels in its box every share fills its own
// sprite, otherwise the whole warp fills them one after the other, 8 x 4 pixels at
// a time.
//
// What bounds it: instruction issue and the latency of the pixel reads.  A
// fragment's depth takes 12 rounded divisions, and a million sprites at 1920 x
// 1080 lie about 50 deep, so nearly all of that work would go to fragments that
// change nothing.  Depths at a pixel only fall: a tile behind the values already
// there (read kTiles tiles at a time; an older, larger value at worst) is
// dropped before any interpolation, and a fragment by its estimated depth.
// That pays when the front sprites come first (sprite_order); back to front,
// the million took 3,190 us.  Filled by the whole warp, a sprite of a few pixels
// waits for its pixel reads and its triangles all the same, one sprite after the
// other.  Measured, us, whole call (35 of them the launches, the fill and the
// wait): a thread per sprite without the depth bound / all sprites by the warp /
// as now:
//   1,000,000 sprites at spacing 0.5 on 320 x 240 134 / 245 / 129, on 1280 x 720
//     - / 345 / 250, on 1920 x 1080 - / 515 / 453; 65,600 on 320 x 240 45 / 56 / 45,
//     on 1280 x 720 - / 77 / 71.
// kSmallPixels: 8, 32 and 128 for the million on 1280 x 720 300 / 301 / 250, on 640 x
// 480 257 / 200 / 173; no case was slower with 128.  Four sprites per warp give a
// scene of some ten thousand enough warps, eight spend less on projecting them:
// 65,600 sprites on 1920 x 1080 96 and 109, on 320 x 240 52 and 47; 262,144 on 1280 x
// 720 129 and 119, 1,000,000 on 1920 x 1080 475 and 454.  The lines are kManySprites
// and, on images below kSmallImage pixels, kManyOnSmallImage.
constexpr int kTiles = 2;

// The order in which the groups of sprites are taken, from 16 sprites spread
// over the array.  Particles are numbered along a lattice, so one end of the
// array is often nearer to the eye: where the mean depths of the samples' two
// halves differ by more than a quarter of their range, from that end.  Otherwise
// in steps that spread over the whole array, so that depths already there are a
// fair sample of the sprites and an order from back to front costs no more than
// a random one.
struct Order {
    uint32_t groups, step, flip;
    __device__ __forceinline__ uint32_t at(uint32_t g) const {
        const uint32_t k = (uint32_t)(((uint64_t)g * step) % groups);
        return flip ? groups - 1u - k : k;
    }
};
__device__ __forceinline__ Order sprite_order(const float4* __restrict__ pos, uint32_t n,
                                              uint32_t group, const View& view) {
    const uint32_t lane = threadIdx.x & 31u;
    // lane l < 16: view-space z of sample l, up to a common factor and offset
    const float4 p = __ldg(pos + (uint32_t)(((uint64_t)n * (2u * (lane & 15u) + 1u)) >> 5));
    const float z = view.V[2] * p.x + view.V[6] * p.y + view.V[10] * p.z;
    float lo = z, hi = z, sum = z;  // over the samples of this half (8 lanes)
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, d));
        hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, d));
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
    }
    const float first = __shfl_sync(0xFFFFFFFFu, sum, 0), last = __shfl_sync(0xFFFFFFFFu, sum, 8);
    lo = fminf(__shfl_sync(0xFFFFFFFFu, lo, 0), __shfl_sync(0xFFFFFFFFu, lo, 8));
    hi = fmaxf(__shfl_sync(0xFFFFFFFFu, hi, 0), __shfl_sync(0xFFFFFFFFu, hi, 8));
    const float diff = (last - first) * 0.125f;  // the eye looks along -z
    const bool directed = fabsf(diff) > 0.25f * (hi - lo);
    Order o;
    o.groups = (n + group - 1) / group;
    // 7919 is a prime: its multiples visit every group unless it divides their number
    o.step = directed || o.groups % 7919u == 0u ? 1u : 7919u;
    o.flip = directed && diff > 0.0f;
    return o;
}

constexpr uint32_t kManySprites = 262144;
constexpr uint32_t kSmallImage = 500000, kManyOnSmallImage = 16384;
constexpr int kSmallPixels = 128;
template <uint32_t kGroup>
__global__ void __launch_bounds__(128, 8)
k_splat_depth(const float4* __restrict__ pos, uint32_t n, View view, uint32_t W, uint32_t H,
              float* __restrict__ out) {
    __shared__ Sprite shared[4][kGroup];
    const uint32_t lane = threadIdx.x & 31u;
    Sprite* const mine = shared[threadIdx.x >> 5];
    const Order order = sprite_order(pos, n, kGroup, view);
    const uint32_t group = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (group >= order.groups) return;
    // every lane of a sprite's share projects it (as fast as one of them would)
    constexpr uint32_t kShare = 32 / kGroup;
    const uint32_t slot = lane / kShare, part = lane & (kShare - 1u);
    const uint32_t k = order.at(group) * kGroup + slot;
    bool drawn = false;
    int pixels = 0;
    if (k < n) {
        Sprite q;
        drawn = make_sprite<PBF_SPLAT_DEPTH>(pos[k], view, W, H, q);
        if (drawn) {
            pixels = (q.x1 - q.x0 + 1) * (q.y1 - q.y0 + 1);
            if (part == 0u) mine[slot] = q;
        }
    }
    __syncwarp();
    if (!__any_sync(0xFFFFFFFFu, pixels > kSmallPixels)) {
        if (!drawn) return;
        const Sprite& s = mine[slot];
        const int cols = s.x1 - s.x0 + 1;
        Tri t0, t1;
        bool made = false;
        for (int p = (int)part; p < pixels; p += (int)kShare) {
            const int row = p / cols, tx = s.x0 + p - row * cols, ty = s.y0 + row;
            float* const at = out + (size_t)ty * W + tx;
            const float seen = __ldcg(at);
            if (seen < s.dlow) continue;
            if (!made) {
                t0 = make_tri(s, 0, 2, 1);
                t1 = make_tri(s, 2, 0, 3);
                made = true;
            }
            float d;
            if (fragment<PBF_SPLAT_DEPTH>(s, t0, t1, view, tx, ty, seen, d))
                atomicMin(reinterpret_cast<unsigned int*>(at), __float_as_uint(d));
        }
        return;
    }
    uint32_t todo = __ballot_sync(0xFFFFFFFFu, drawn && part == 0u);
    const int dx = (int)(lane & 7u), dy = (int)(lane >> 3);
    while (todo) {
        const int src = __ffs((int)todo) - 1;
        todo &= todo - 1;
        const Sprite& s = mine[src / (int)kShare];
        Tri t0, t1;  // made for the first tile that may be in front
        bool made = false;
        const int cols = (s.x1 - s.x0 + 8) >> 3, tiles = cols * ((s.y1 - s.y0 + 4) >> 2);
        for (int base = 0; base < tiles; base += kTiles) {
            float seen[kTiles];
            int row = base / cols, col = base - row * cols;
#pragma unroll
            for (int t = 0; t < kTiles; ++t) {
                const int tx = s.x0 + 8 * col + dx, ty = s.y0 + 4 * row + dy;
                seen[t] = -1.0f;  // outside the box: below every bound
                if (base + t < tiles && tx <= s.x1 && ty <= s.y1)
                    seen[t] = __ldcg(out + (size_t)ty * W + tx);
                if (++col == cols) {
                    col = 0;
                    ++row;
                }
            }
            bool front = false;
#pragma unroll
            for (int t = 0; t < kTiles; ++t) front = front || (seen[t] >= 0.0f && !(seen[t] < s.dlow));
            if (!__any_sync(0xFFFFFFFFu, front)) continue;
            if (!made) {
                t0 = make_tri(s, 0, 2, 1);
                t1 = make_tri(s, 2, 0, 3);
                made = true;
            }
            row = base / cols, col = base - row * cols;
#pragma unroll
            for (int t = 0; t < kTiles; ++t) {
                const int tx = s.x0 + 8 * col + dx, ty = s.y0 + 4 * row + dy;
                float d;
                if (seen[t] >= 0.0f && !(seen[t] < s.dlow) &&
                    fragment<PBF_SPLAT_DEPTH>(s, t0, t1, view, tx, ty, seen[t], d))
                    atomicMin(reinterpret_cast<unsigned int*>(out) + (size_t)ty * W + tx,
                              __float_as_uint(d));
                if (++col == cols) {
                    col = 0;
                    ++row;
                }
            }
        }
    }
}

// Thickness pass, first half: `diff` (zeroed) receives +1 where a sprite's
// pixels start in a row and -1 after they end; k_splat_count sums the rows.  A
// thread fills its own sprite, except sprites of more than kOwnPixels pixels,
// which the warp fills one after the other, 8 x 4 pixels at a time: a few
// sprites close to the eye do not hold up their warp.
//
// What bounds it: the atomics.  A sprite 7 pixels across covers 40 pixels in 7
// rows, and the image's atomic additions then run at about the L2's rate; two
// per row are a third of them, and the sums are whole numbers either way.  The
// rounded weights (8 divisions a fragment) are needed at the disc's edge only.
// Measured, us, both halves: 65,536 sprites at 512 x 512 25 -> 17;
// 1,046,272 at 960 x 540 386 -> 234.
// Few sprites, and sprites on a small image, are added pixel by pixel (!kRows: below
// kFewSprites, or below kMoreSprites on images below kFewPixels): there the second
// half costs more than its atomics save.  Whole call, us, pixels / rows: 4,096 sprites
// on 320 x 240 37 / 44, on 640 x 480 46 / 46, on 960 x 540 50 / 48; 65,600 on 320 x
// 240 41 / 44, on 480 x 360 47 / 45; 262,144 on 256 x 256 57 / 56; 400 on 1920 x 1080
// 38 / 45.
constexpr int kOwnPixels = 256;
constexpr uint32_t kFewSprites = 1024, kMoreSprites = 131072, kFewPixels = 200000;
template <bool kRows>
__global__ void __launch_bounds__(128)
k_splat_thickness(const float4* __restrict__ pos, uint32_t n, View view, uint32_t W, uint32_t H,
                  float* __restrict__ out) {
    int* const diff = reinterpret_cast<int*>(out);
    __shared__ Sprite shared[128];
    const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    Sprite q;
    const bool drawn = id < n && make_sprite<PBF_SPLAT_THICKNESS>(pos[id], view, W, H, q);
    const bool large = drawn && (q.x1 - q.x0 + 1) * (q.y1 - q.y0 + 1) > kOwnPixels;
    float unused;
    if (large) shared[threadIdx.x] = q;
    if (drawn && !large) {
        const Tri t0 = make_tri(q, 0, 2, 1), t1 = make_tri(q, 2, 0, 3);
        for (int ty = q.y0; ty <= q.y1; ++ty) {
            int* const row = diff + (size_t)ty * W;
            bool on = false;
            for (int tx = q.x0; tx <= q.x1; ++tx) {
                const bool in = fragment<PBF_SPLAT_THICKNESS>(q, t0, t1, view, tx, ty, 0.0f, unused);
                if (!kRows) {
                    if (in) atomicAdd(out + (size_t)ty * W + tx, 1.0f);
                    continue;
                }
                if (in != on) atomicAdd(row + tx, in ? 1 : -1);
                on = in;
            }
            if (kRows && on && q.x1 + 1 < (int)W) atomicAdd(row + q.x1 + 1, -1);
        }
    }
    __syncwarp();
    uint32_t todo = __ballot_sync(0xFFFFFFFFu, large);
    const int dx = (int)(lane & 7u), dy = (int)(lane >> 3);
    while (todo) {
        const int src = __ffs((int)todo) - 1;
        todo &= todo - 1;
        const Sprite& s = shared[(threadIdx.x & ~31u) + src];
        const Tri t0 = make_tri(s, 0, 2, 1), t1 = make_tri(s, 2, 0, 3);
        for (int ty = s.y0 + dy; ty - dy <= s.y1; ty += 4)
            for (int tx = s.x0 + dx; tx - dx <= s.x1; tx += 8) {
                const bool in = tx <= s.x1 && ty <= s.y1 &&
                                fragment<PBF_SPLAT_THICKNESS>(s, t0, t1, view, tx, ty, 0.0f, unused);
                if (!kRows) {
                    if (in) atomicAdd(out + (size_t)ty * W + tx, 1.0f);
                    continue;
                }
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, in);
                int* const at = diff + (size_t)ty * W + tx;
                if (in && (dx == 0 || !(m >> (lane - 1u) & 1u))) atomicAdd(at, 1);
                if (in && (dx == 7 || !(m >> (lane + 1u) & 1u)) && tx + 1 < (int)W)
                    atomicAdd(at + 1, -1);
            }
    }
}

// Thickness pass, second half: running sums along each row, in place, as the
// float counts that adding 1 at a time gives (it stops at 2^24).  A block per
// row, kCountBlock pixels of it at a time, four per thread.  What bounds it: the
// latency of one step of a row, so rows take one or two steps (a warp per row,
// 128 pixels at a time, took 15 at 1920 pixels: 10 us of the call where a few
// sprites are drawn).
constexpr int kCountThreads = 256, kCountBlock = 4 * kCountThreads;
__global__ void __launch_bounds__(kCountThreads) k_splat_count(float* __restrict__ out, uint32_t W) {
    __shared__ int warps[kCountThreads / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float* const o = out + (size_t)blockIdx.x * W;
    int carry = 0;
    for (uint32_t x0 = 0; x0 < W; x0 += kCountBlock) {
        int v[4];
        const uint32_t x = x0 + 4 * threadIdx.x;
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = x + k < W ? __float_as_int(o[x + k]) : 0;
        v[1] += v[0];
        v[2] += v[1];
        v[3] += v[2];
        int before = v[3];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, before, d);
            if ((int)lane >= d) before += y;
        }
        if (lane == 31u) warps[warp] = before;
        __syncthreads();
        int total = 0;
        before += carry - v[3];
#pragma unroll
        for (uint32_t w = 0; w < kCountThreads / 32; ++w) {
            if (w < warp) before += warps[w];
            total += warps[w];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (x + k < W) o[x + k] = (float)min(before + v[k], 1 << 24);
        carry += total;
        __syncthreads();
    }
}

__global__ void k_fill(float* __restrict__ out, size_t count, float value) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) out[i] = value;
}

}  // namespace
}  // namespace pbf

extern "C" pbf_status pbf_splat(int pass, const float* positions, uint32_t n, const pbf_view* view,
                                uint32_t width, uint32_t height, float* out, void* stream) {
    pbf::NvtxRange nvtx_("pbf_splat");
    using namespace pbf;
    if (pass != PBF_SPLAT_DEPTH && pass != PBF_SPLAT_THICKNESS)
        return fail(nullptr, PBF_ERR_INVALID_ARGUMENT, "pass must be PBF_SPLAT_DEPTH or PBF_SPLAT_THICKNESS");
    if (!view || !out || (n > 0 && !positions))
        return fail(nullptr, PBF_ERR_INVALID_ARGUMENT, "NULL argument");
    if (width == 0 || height == 0 || width > 16384 || height > 16384)
        return fail(nullptr, PBF_ERR_INVALID_ARGUMENT, "width and height must be in [1, 16384]");
    cudaStream_t st = (cudaStream_t)stream;
    View v;
    for (int k = 0; k < 16; ++k) {
        v.V[k] = view->viewmat[k];
        v.P[k] = view->projmat[k];
    }
    const size_t count = (size_t)width * height;
    k_fill<<<(unsigned)((count + 255) / 256), 256, 0, st>>>(out, count,
                                                            pass == PBF_SPLAT_DEPTH ? 1.0f : 0.0f);
    if (n > 0) {
        const float4* p = (const float4*)positions;
        if (pass == PBF_SPLAT_DEPTH) {
            const bool many = n >= kManySprites ||
                              (n >= kManyOnSmallImage && count < kSmallImage);
            if (!many)
                k_splat_depth<4><<<(n + 15) / 16, 128, 0, st>>>(p, n, v, width, height, out);
            else
                k_splat_depth<8><<<(n + 31) / 32, 128, 0, st>>>(p, n, v, width, height, out);
        } else {
            const unsigned g = (n + 127) / 128;
            if (n < kFewSprites || (n < kMoreSprites && count < kFewPixels)) {
                k_splat_thickness<false><<<g, 128, 0, st>>>(p, n, v, width, height, out);
            } else {
                k_splat_thickness<true><<<g, 128, 0, st>>>(p, n, v, width, height, out);
                k_splat_count<<<height, kCountThreads, 0, st>>>(out, width);
            }
        }
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "pbf_splat");
    return PBF_OK;
}
