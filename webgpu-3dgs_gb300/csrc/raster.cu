// raster.cu - stage 6 of the rebin: tiled front-to-back alpha blending.
//
// Same per-pixel arithmetic and termination rules as
// src/shaders/compute/rasterize_tiles.wgsl:44-110: pixel centre = pixel + 0.5;
// per splat: circular cull at radius_px, power = -0.5 * d^T conic d, skip power
// > 0, alpha = min(0.99, opacity * exp(power)), skip alpha < 1/255, C += T *
// alpha * rgb, T *= 1 - alpha, stop the pixel once T < 1e-4 (checked after
// blending); the output is rgba16float (C, 1 - T), premultiplied, no
// background.  Each tile's cost is recorded: the number of splats iterated
// before its last pixel terminated.
//
// Three variants:
//  * plain (any tile): one CTA per tile, one thread per pixel, the sorted
//    splats staged in batches of RasterArgs::batch by double-buffered cp.async,
//    left as soon as every pixel has terminated (the reference keeps looping);
//  * culled (an area that divides by 32): the same, and each warp owns a block of
//    8x4 pixels, or where the sides do not divide so 32 pixels in row order, and
//    tests every staged splat once against its pixels' box;
//  * warps (sides that divide by 8, all usual tiles): independent warps over
//    regions of 2x2 blocks of 8x8 pixels, two pixels a lane (see there).
// A splat is converted once per CTA or warp into its raster form (r^2, the
// quadratic form's coefficients, the visibility bound), so a (pixel, splat) pair
// costs one ex2 and a branch-free handful of FP32 operations (a skipped splat
// blends with alpha = 0, which leaves the pixel bit-unchanged).  It is skipped
// for a block or a region only when no pixel centre of it can pass the
// per-pixel tests: outside the radius circle, or the minimum of d^T conic d over
// it keeps alpha below 1/255, with margins that cover f32 rounding and the fast
// division of the edge minimisers.  Pixels therefore blend exactly the same
// splats in the same order.
//
// The variants share the per-pixel arithmetic (in the last as paired FP32
// instructions, each half rounded like the scalar one), so their images are
// bit-identical.  For splats whose quadratic form can cancel badly the radius
// test and power = -0.5 d^T conic d follow the reference's f32 expression order
// exactly (no contraction; SplatStage below); the others, the exponent (ex2 in
// the log2 domain) and the blend (fused multiply-adds) differ from the reference
// only in rounding, which the 2/255 image tolerance covers.
//
// Bound: instruction issue (67 to 74% busy, ALU 46 to 53%, 20 warps an SM; DRAM
// under 10%).  One strip of a tile per CTA -> independent warps over regions, cull
// per region, blocks handed on: 8 views of 3M splats 3935 -> 2518 us, 12 mixed
// views 5580 -> 3784, one 3M frame 425 -> 344, 100k 74 -> 61.
#include <algorithm>
#include <map>
#include <mutex>

#include "gs3d_internal.cuh"

namespace gs3d {
namespace {

// A staged splat in one of two forms of the quadratic form q(d) = b.x dx^2 +
// b.y dx dy + b.z dy^2 (c.w says which):
//   fast  (c.w = 0): b = log2(e)/2 (conic.x, 2 conic.y, conic.z), q = Q =
//         -power log2(e), evaluated with FMAs;
//   exact (c.w = 1): b = (conic.x, 2 conic.y, conic.z), q = s = d^T conic d
//         = -2 power, evaluated in the reference's operation order without
//         contraction (every sum a scalar __fadd_rn: a paired FP32 multiply
//         feeding a paired add is contracted into a paired FMA).
// Splats take the exact form when the terms of q can reach 2^12 inside the
// radius, (|conic.x| + 2 |conic.y| + |conic.z|) r^2 > 2^12: there the terms
// cancel (elongated splats seen far from their mean), and the rounding order
// decides the result.  So do conics that are not positive definite (by rounding of
// a huge covariance): theirs is the q < 0 test.  Below that bound the fast form's q differs from the
// reference's by about 2^-11 at most, so each alpha differs by a relative
// 1e-3 and a pixel, whose blend weights alpha_i T_i sum to at most 1, by
// about that much.  b.w = vis, in q's units; its two lowest bits hold the
// splat's kind (prepare).
struct SplatStage {  // first 48 bytes of a ProjectedSplat, prepared in place (prepare())
  float4 a;  // mean_px.x, mean_px.y, radius_px^2, opacity
  float4 b;  // q coefficients (see above), vis
  float4 c;  // color.xyz, form
};

constexpr float kHalfLog2e = 0.72134752044448170f;
constexpr float kExactFormBound = 4096.0f;
// How a splat's alpha is evaluated: fast form whose op exp(power) stays below
// the 0.99 clamp; fast form with the clamp; exact form (which clamps).
constexpr uint32_t kSimple = 0u, kClamped = 1u, kExact = 2u;
// vis of splats culled by their circle alone, 3.0e38.  Its two low bits are clear:
// prepare leaves the kind there, and every kind has to stay at or above it.
constexpr float kCircleOnly = 0x1.c363c8p+127f;
static_assert((__builtin_bit_cast(uint32_t, kCircleOnly) & 3u) == 0u, "room for the kind");

struct Pixel {
  float cr, cg, cb, T;
};

// ex2.approx: 2^x on the SFU.
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Converts the staged ProjectedSplat prefix (mean, depth, radius | conic,
// opacity | color, valid) into the raster form.  vis = the largest Q at which
// alpha can still reach 1/255, with a 1% margin, in the units of the splat's
// form (-1: never visible; kCircleOnly or more: use the circle only: a conic
// with a non-positive diagonal, or anything not finite, whose NaN alphas pass as
// 0.99 whatever the opacity).
//
// vis also carries the rounding of the quadratic form, so that the cull stays
// conservative for any conic, needles included (condition numbers of 10^3
// and more, splats with axes more than 30:1 apart).  With u = 2^-24 and
// t(d) = |A| dx^2 + 2 |B dx dy| + |C| dy^2, the per-pixel form in either
// operation order and the cull's own evaluation each lie within about 4 u t
// of the exact form, and rect_may_hit's approximate stationary points raise it
// by far less (2^-42 t).  A pixel that passes its tests lies in the circle, and
// the cull's points within `ext` of one (ext bounds the diagonal of a warp's
// pixel block), so t <= (|A| + 2 |B| + |C|) (r + ext)^2; 16 u times that is
// added, twice the sum of both.  Needles kept for every block of their circle
// (as before the bound) are 4.8 times the blocks that hold a visible pixel on
// a 4K close-up of heavy-tailed scales, 1.3 times on the 3M-splat orbit views:
// raster 6.34 -> 1.61 ms there (3M splats, 32x32 tiles), 3.94 -> 3.31 ms for
// 8 orbit views (64x32), 0.425 -> 0.362 ms for one view at 16x16.
__device__ __forceinline__ void prepare(SplatStage& s, float ext) {
  const float4 a = s.a, b = s.b;
  const float A = b.x, B = b.y, C = b.z, op = b.w;
  const float sum = fabsf(A) + 2.0f * fabsf(B) + fabsf(C);
  // the form's terms anywhere near the circle, NaN or infinite where the mean, the
  // radius, the conic or the opacity is (an infinite one gives NaN where exp
  // underflows); lim is NaN there
  const float reach = a.w + ext, near = fmaf(0.0f, a.x + a.y + op, sum * reach * reach);
  const float lim = fmaf(0.0f, near, op * 255.0f);
  const float r2 = a.w * a.w;
  const float terms = sum * r2;
  // the second bound gives q >= t / 800, far above its rounding; a splat whose
  // covariance did not lose it to rounding has B^2 < 0.992 A C where the first holds
  // (a condition number below 455)
  const bool fast = terms <= kExactFormBound && A > 0.0f && B * B <= 0.995f * A * C;
  float vis;
  if (lim < 0.999f) {
    vis = -1.0f;  // alpha = opacity * exp(power) <= opacity < 1/255 everywhere
  } else {
    vis = __log2f(lim) * 1.01f + 1e-3f + (kHalfLog2e * 9.5367431640625e-07f) * near;
    // false for NaNs too
    if (!(lim > 1.0f && A > 0.0f && C > 0.0f && vis < 1.0e38f)) vis = kCircleOnly;
  }
  s.a = make_float4(a.x, a.y, r2, op);
  if (fast) {
    // no clamp where ex2 of a value <= 0 (to 2 ulp) times op stays below it
    const bool simple = lim <= 0.9899f * 255.0f;
    vis = __uint_as_float((__float_as_uint(vis) & ~3u) | (simple ? kSimple : kClamped));
    s.b = make_float4(kHalfLog2e * A, 2.0f * kHalfLog2e * B, kHalfLog2e * C, vis);
    s.c.w = 0.0f;
  } else {  // also non-finite terms
    vis = fminf(vis * (1.0f / kHalfLog2e), kCircleOnly);
    s.b = make_float4(A, 2.0f * B, C, __uint_as_float((__float_as_uint(vis) & ~3u) | kExact));
    s.c.w = 1.0f;
  }
}

// Bounds the diagonal of the pixel-centre box of any warp of the culled
// variants: 8x8 or 8x4 blocks (9.9), else rows of the tile.
__device__ __forceinline__ float warp_box_reach(const RasterArgs& a, bool blocks) {
  return blocks ? 12.0f : (float)(a.tile_w + a.tile_h);
}

// rasterize_tiles.wgsl:81-98 for one (pixel, splat) pair: the splat's alpha
// at the pixel centre and whether it passes the per-pixel tests (not outside
// the radius, power not > 0, alpha not < 1/255: a NaN passes, as in the
// reference).  A skipped splat blends with alpha = 0 (blend_alpha), which
// leaves C and T bit-unchanged.
__device__ __forceinline__ float splat_alpha(float pfx, float pfy, const SplatStage& s,
                                             bool exact, bool& ok) {
  const float4 a = s.a, b = s.b;
  const float dx = pfx - a.x;
  const float dy = pfy - a.y;
  if (!exact) {
    // fast form: q < 0 cannot occur (no power > 0 test needed): these splats'
    // conics are positive definite by a margin (prepare), so q, computed to
    // a relative 1e-3, and the reference's s keep the sign of the form at every
    // pixel centre, which lies 6e-8 pixels or more from the mean unless exactly
    // on it
    const float d2 = fmaf(dx, dx, dy * dy);
    const float q = fmaf(b.x * dx, dx, fmaf(b.y * dx, dy, b.z * dy * dy));  // -power log2(e)
    const float alpha = fminf(0.99f, a.w * ex2_approx(-q));
    ok = !(d2 > a.z) && !(alpha < 1.0f / 255.0f);
    return alpha;
  }
  // the reference's order: d^2 = dx dx + dy dy, s = (c0 dx) dx + (2 c1 dx) dy + (c2 dy) dy
  const float d2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
  const float q = __fadd_rn(
      __fadd_rn(__fmul_rn(__fmul_rn(b.x, dx), dx), __fmul_rn(__fmul_rn(b.y, dx), dy)),
      __fmul_rn(__fmul_rn(b.z, dy), dy));
  const float alpha = fminf(0.99f, a.w * ex2_approx(__fmul_rn(q, -kHalfLog2e)));  // exp(-s/2)
  ok = !(d2 > a.z) && !(q < 0.0f) && !(alpha < 1.0f / 255.0f);
  return alpha;
}

// Blends alpha (0 when !ok, which leaves C and T bit-unchanged); returns
// true when the pixel terminates here.
__device__ __forceinline__ bool blend_alpha(Pixel& p, const float4 c, float alpha, bool ok) {
  const float al = ok ? alpha : 0.0f;
  const float ta = p.T * al;
  p.cr = fmaf(ta, c.x, p.cr);
  p.cg = fmaf(ta, c.y, p.cg);
  p.cb = fmaf(ta, c.z, p.cb);
  p.T = p.T * (1.0f - al);
  return ok && p.T < 1.0e-4f;
}

// The plain variant's splat; true when the pixel terminates.
__device__ __forceinline__ bool blend_one(float pfx, float pfy, const SplatStage& s, Pixel& p) {
  // outside the radius (d^2 as splat_alpha forms it): alpha would be 0
  const float dx = pfx - s.a.x, dy = pfy - s.a.y;
  const float d2 = s.c.w == 0.0f ? fmaf(dx, dx, dy * dy)
                                 : __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
  if (d2 > s.a.z) return false;
  bool ok;
  const float alpha = splat_alpha(pfx, pfy, s, s.c.w != 0.0f, ok);
  return blend_alpha(p, s.c, alpha, ok);
}

// Two pixels of one column in the halves of a float2.  Every component is computed
// by the scalar operation of splat_alpha / blend_alpha, in the same order and
// rounding (the paired FP32 instructions of sm_100 round each half like their
// scalar forms), so each pixel is bit-identical to the one-pixel forms.
__device__ __forceinline__ float2 bcast(float x) { return make_float2(x, x); }

// splat_alpha of a simple splat, 0 where it is skipped: the same operations without
// the clamp, which cannot act.
__device__ __forceinline__ float simple_alpha(float pfx, float pfy, const SplatStage& s) {
  const float4 a = s.a, b = s.b;
  const float dx = pfx - a.x;
  const float dy = pfy - a.y;
  const float d2 = fmaf(dx, dx, dy * dy);
  const float q = fmaf(b.x * dx, dx, fmaf(b.y * dx, dy, b.z * dy * dy));
  const float alpha = a.w * ex2_approx(-q);
  return !(d2 > a.z) && !(alpha < 1.0f / 255.0f) ? alpha : 0.0f;
}
__device__ __forceinline__ float2 simple_alpha(float pfx, float2 pfy, const SplatStage& s) {
  const float4 a = s.a, b = s.b;
  const float dx = pfx - a.x;
  const float2 dy = __fadd2_rn(pfy, bcast(-a.y));
  const float2 d2 = __ffma2_rn(bcast(dx), bcast(dx), __fmul2_rn(dy, dy));
  const float2 q =
      __ffma2_rn(bcast(b.x * dx), bcast(dx),
                 __ffma2_rn(bcast(b.y * dx), dy, __fmul2_rn(__fmul2_rn(bcast(b.z), dy), dy)));
  const float2 alpha = __fmul2_rn(bcast(a.w), make_float2(ex2_approx(-q.x), ex2_approx(-q.y)));
  return make_float2(!(d2.x > a.z) && !(alpha.x < 1.0f / 255.0f) ? alpha.x : 0.0f,
                     !(d2.y > a.z) && !(alpha.y < 1.0f / 255.0f) ? alpha.y : 0.0f);
}
// The same for an exact-form splat.
__device__ __forceinline__ float exact_alpha(float pfx, float pfy, const SplatStage& s) {
  bool ok;
  const float alpha = splat_alpha(pfx, pfy, s, true, ok);
  return ok ? alpha : 0.0f;
}
// (the products are paired, every sum a scalar __fadd_rn, never merged into an FMA)
__device__ __forceinline__ float2 exact_alpha(float pfx, float2 pfy, const SplatStage& s) {
  const float4 a = s.a, b = s.b;
  const float dx = pfx - a.x;
  const float2 dy = __fadd2_rn(pfy, bcast(-a.y));
  const float dxx = __fmul_rn(dx, dx);
  const float t1 = __fmul_rn(__fmul_rn(b.x, dx), dx);
  const float2 dyy = __fmul2_rn(dy, dy);
  const float2 t2 = __fmul2_rn(bcast(__fmul_rn(b.y, dx)), dy);
  const float2 t3 = __fmul2_rn(__fmul2_rn(bcast(b.z), dy), dy);
  const float2 d2 = make_float2(__fadd_rn(dxx, dyy.x), __fadd_rn(dxx, dyy.y));
  const float2 q =
      make_float2(__fadd_rn(__fadd_rn(t1, t2.x), t3.x), __fadd_rn(__fadd_rn(t1, t2.y), t3.y));
  const float2 ev = __fmul2_rn(q, bcast(-kHalfLog2e));
  const float2 am = __fmul2_rn(bcast(a.w), make_float2(ex2_approx(ev.x), ex2_approx(ev.y)));
  const float2 alpha = make_float2(fminf(0.99f, am.x), fminf(0.99f, am.y));
  return make_float2(
      !(d2.x > a.z) && !(q.x < 0.0f) && !(alpha.x < 1.0f / 255.0f) ? alpha.x : 0.0f,
      !(d2.y > a.z) && !(q.y < 0.0f) && !(alpha.y < 1.0f / 255.0f) ? alpha.y : 0.0f);
}
// The same for a splat of either form: both are evaluated and one is taken, so
// that four of a step overlap (a branch per splat costs more than the few
// operations that the forms do not share).  The q < 0 and clamp tests cannot
// act on a fast-form splat that has none.
__device__ __forceinline__ float any_alpha(float pfx, float pfy, const SplatStage& s, bool exact) {
  const float4 a = s.a, b = s.b;
  const float dx = pfx - a.x;
  const float dy = pfy - a.y;
  const float u = __fmul_rn(b.x, dx), v = __fmul_rn(b.y, dx);
  const float w = __fmul_rn(__fmul_rn(b.z, dy), dy);
  const float dyy = __fmul_rn(dy, dy);
  const float qe = __fadd_rn(__fadd_rn(__fmul_rn(u, dx), __fmul_rn(v, dy)), w);
  const float qf = fmaf(u, dx, fmaf(v, dy, w));
  const float d2 = exact ? __fadd_rn(__fmul_rn(dx, dx), dyy) : fmaf(dx, dx, dyy);
  const float q = exact ? qe : qf;
  const float alpha = fminf(0.99f, a.w * ex2_approx(__fmul_rn(q, exact ? -kHalfLog2e : -1.0f)));
  return !(d2 > a.z) && !(q < 0.0f) && !(alpha < 1.0f / 255.0f) ? alpha : 0.0f;
}
__device__ __forceinline__ float2 any_alpha(float pfx, float2 pfy, const SplatStage& s,
                                            bool exact) {
  const float4 a = s.a, b = s.b;
  const float dx = pfx - a.x;
  const float2 dy = __fadd2_rn(pfy, bcast(-a.y));
  const float u = __fmul_rn(b.x, dx), v = __fmul_rn(b.y, dx);
  const float2 w = __fmul2_rn(__fmul2_rn(bcast(b.z), dy), dy);
  const float2 dyy = __fmul2_rn(dy, dy);
  // exact: every sum a scalar __fadd_rn (never merged into an FMA)
  const float t1 = __fmul_rn(u, dx), dxx = __fmul_rn(dx, dx);
  const float2 t2 = __fmul2_rn(bcast(v), dy);
  // fast
  const float2 qf = __ffma2_rn(bcast(u), bcast(dx), __ffma2_rn(bcast(v), dy, w));
  const float2 df = __ffma2_rn(bcast(dx), bcast(dx), dyy);
  const float2 q = make_float2(exact ? __fadd_rn(__fadd_rn(t1, t2.x), w.x) : qf.x,
                               exact ? __fadd_rn(__fadd_rn(t1, t2.y), w.y) : qf.y);
  const float2 d2 =
      make_float2(exact ? __fadd_rn(dxx, dyy.x) : df.x, exact ? __fadd_rn(dxx, dyy.y) : df.y);
  const float2 ev = __fmul2_rn(q, bcast(exact ? -kHalfLog2e : -1.0f));
  const float2 am = __fmul2_rn(bcast(a.w), make_float2(ex2_approx(ev.x), ex2_approx(ev.y)));
  const float2 alpha = make_float2(fminf(0.99f, am.x), fminf(0.99f, am.y));
  return make_float2(
      !(d2.x > a.z) && !(q.x < 0.0f) && !(alpha.x < 1.0f / 255.0f) ? alpha.x : 0.0f,
      !(d2.y > a.z) && !(q.y < 0.0f) && !(alpha.y < 1.0f / 255.0f) ? alpha.y : 0.0f);
}

// The blend state of a lane's pixels: one (Px1) or two of a column (Px2).
// T is 0 once a pixel has terminated (out-of-view pixels start so), and a
// splat then adds exactly nothing to it; `fin` holds the T it ended with.
constexpr float kEndT = 1.0e-4f;
struct Px1 {
  float y, cr = 0.f, cg = 0.f, cb = 0.f, T = 1.f, fin = 0.f;
  using V = float;
  static constexpr int kN = 1;
  __device__ static V mul(V a, V b) { return a * b; }
  __device__ static V fma(V a, float c, V b) { return fmaf(a, c, b); }
  __device__ static V keep(V al) { return 1.0f - al; }
  __device__ static float& at(V& v, int) { return v; }
};
struct Px2 {
  float2 y, cr = {0.f, 0.f}, cg = {0.f, 0.f}, cb = {0.f, 0.f}, T = {1.f, 1.f}, fin = {0.f, 0.f};
  using V = float2;
  static constexpr int kN = 2;
  __device__ static V mul(V a, V b) { return __fmul2_rn(a, b); }
  __device__ static V fma(V a, float c, V b) { return __ffma2_rn(a, bcast(c), b); }
  __device__ static V keep(V al) { return __ffma2_rn(al, bcast(-1.0f), bcast(1.0f)); }
  __device__ static float& at(V& v, int i) { return i ? v.y : v.x; }
};
template <typename PX>
__device__ __forceinline__ bool px_live(PX& p) {
  bool live = false;
#pragma unroll
  for (int i = 0; i < PX::kN; ++i) live = live || PX::at(p.T, i) > 0.0f;
  return live;
}
template <typename PX>
__device__ __forceinline__ float px_final(PX& p, int i) {
  return PX::at(p.T, i) > 0.0f ? PX::at(p.T, i) : PX::at(p.fin, i);
}

__device__ __forceinline__ void store_pixel(uint2* image, uint32_t W, uint32_t px, uint32_t py,
                                            const Pixel& p) {
  const __half2 rg = __floats2half2_rn(p.cr, p.cg);
  const __half2 ba = __floats2half2_rn(p.cb, 1.0f - p.T);
  image[(size_t)py * W + px] =
      make_uint2(*reinterpret_cast<const uint32_t*>(&rg), *reinterpret_cast<const uint32_t*>(&ba));
}

// Stages sorted splats [first, min(first + batch, end)) into dst; thread t
// copies entries t, t + nt, ... (one commit group per thread and batch).
__device__ __forceinline__ void stage_batch(const gs3d_projected_splat* __restrict__ proj,
                                            const uint32_t* __restrict__ values, uint32_t first,
                                            uint32_t end, uint32_t batch, uint32_t nt,
                                            SplatStage* dst) {
  for (uint32_t k = threadIdx.x; k < batch; k += nt) {
    const uint32_t idx = first + k;
    if (idx >= end) break;
    const uint32_t id = __ldg(values + idx);
    const float4* src = reinterpret_cast<const float4*>(proj + id);
    cp_async16(&dst[k].a, src + 0);
    cp_async16(&dst[k].b, src + 1);
    cp_async16(&dst[k].c, src + 2);
  }
  cp_async_commit();
}

// x clamped to [lo, hi]; NaN where a bound is (fminf and fmaxf drop it).
__device__ __forceinline__ float clamp_nan(float x, float lo, float hi) {
  asm("max.NaN.f32 %0, %0, %1;\n min.NaN.f32 %0, %0, %2;" : "+f"(x) : "f"(lo), "f"(hi));
  return x;
}

// Can the splat reach alpha >= 1/255 inside the rectangle of pixel centres
// [x0,x1] x [y0,y1]?  Minimum of the splat's q over the rectangle
// (scale-invariant, so either form works), compared with vis; plus the radius
// circle.  Any point d of a rectangle without the mean sees the mean through
// the edge nearest to it in x or in y, and q(t d) = t^2 q(d): so where q <= vis
// somewhere, it is on one of those two edges, also for a form that rounding
// made indefinite.  Along an edge q is convex (the conic's diagonal is
// positive), so its minimum there is at the clamped stationary point.
// Conservative by the margins folded into vis (prepare) and the circle.  NaN
// means (one coordinate or both), radii, conics or opacities are never culled (the
// per-pixel tests decide, as in the reference): no comparison with a NaN culls.
__device__ __forceinline__ bool rect_may_hit(const float4 a, const float4 b, float2 xr,
                                             float2 yr) {
  // the box corners relative to the mean (x - m computed as x + (-m))
  const float2 xd = __fadd2_rn(xr, bcast(-a.x)), yd = __fadd2_rn(yr, bcast(-a.y));
  const float x0 = xd.x, x1 = xd.y, y0 = yd.x, y1 = yd.y;
  const float ex = clamp_nan(0.0f, x0, x1), ey = clamp_nan(0.0f, y0, y1);
  const float vis = b.w;
  if (ex * ex + ey * ey > a.z * 1.0001f + 1e-3f || vis < 0.0f) return false;
  const float qa = b.x, qb = b.y, qc = b.z;
  // stationary points of the edges x = ex and y = ey, by the fast reciprocal
  // division: an error d in the point raises q there by qa d^2 (qc d^2) over
  // the edge minimum, far inside the margins folded into vis
  const float vy = fminf(fmaxf(__fdividef(-0.5f * qb, qc) * ex, y0), y1);
  const float hx = fminf(fmaxf(__fdividef(-0.5f * qb, qa) * ey, x0), x1);
  const float2 x = make_float2(ex, hx), y = make_float2(vy, ey);
  const float2 q = __ffma2_rn(__fmul2_rn(bcast(qa), x), x,
                              __ffma2_rn(__fmul2_rn(bcast(qb), x), y,
                                         __fmul2_rn(__fmul2_rn(bcast(qc), y), y)));
  // the mean inside (ex = ey = 0): q is 0 at both, or the circle decides
  return fminf(q.x, q.y) <= vis || (ex == 0.0f && ey == 0.0f) || vis >= kCircleOnly;
}

// ---- the culled variants' inner loops ------------------------------------------
// A warp works on one segment of a staged batch at a time: it tests the
// segment's splats against its pixel block, 32 a step, and queues the ones that
// may hit in order in its list; then it blends the list four splats a step.
// The four alphas do not depend on one another, only T's four multiplications
// form a chain, and the cut-off is looked at once a step: T never grows, so a
// pixel above the cut-off after the fourth splat has not ended before.  In a
// step that ends a pixel, the products of the chain from its end on are
// dropped.
constexpr int kGroup = 4, kFineGroup = 8;      // splats blended a step
constexpr uint32_t kSegment = 256;             // splats culled before they are blended
constexpr uint32_t kListPitch = kSegment + 8;  // list entries per warp (padded steps)
constexpr uint32_t kKindShift = 14;            // list entry: staged index | kind << 14
constexpr uint32_t kIndexMask = (1u << kKindShift) - 1u;

// Queues the splats [k0, k1) of `cur` that may hit the box; returns how many,
// padded with `none` (an invisible staged splat) to whole steps.
__device__ __forceinline__ uint32_t cull_segment(const SplatStage* cur, uint32_t k0, uint32_t k1,
                                                 uint32_t none, float2 xr, float2 yr,
                                                 uint16_t* list) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t n = 0;
#pragma unroll 1
  for (uint32_t k = k0; k < k1; k += 32) {
    const uint32_t j = k + lane;
    const uint32_t i = j < k1 ? j : none;
    const float4 a = cur[i].a, b = cur[i].b;
    const bool hit = rect_may_hit(a, b, xr, yr);
    const uint32_t mask = __ballot_sync(0xffffffffu, hit);
    if (hit)
      list[n + __popc(mask & lanemask_lt())] =
          (uint16_t)(i | (__float_as_uint(b.w) << kKindShift));
    n += __popc(mask);
  }
  if (lane < kGroup) list[n + lane] = (uint16_t)none;
  __syncwarp();
  return n;
}

// Blends the n queued splats into the lane's pixels; false once every pixel
// of the warp has terminated, with used = 1 + the position in the tile's list
// (position(staged index)) of the splat that ended the lane's last pixel,
// where it ended in the last step (the warp's largest is among those).
template <int G, typename PX, typename POS>
__device__ __forceinline__ bool blend_list(const SplatStage* cur, const uint16_t* list,
                                           uint32_t n, float pfx, PX& p, POS position,
                                           uint32_t& used) {
  using V = typename PX::V;
  constexpr bool kAhead = G > kGroup;  // one warp's chain: the next step's entries early
  uint32_t ahead[G / 2];               // two a word
  if (kAhead) {
#pragma unroll
    for (int h = 0; h < G / 2; ++h) ahead[h] = reinterpret_cast<const uint32_t*>(list)[h];
  }
  for (uint32_t i = 0; i < n; i += G) {
    uint32_t e[G / 2];
#pragma unroll
    for (int h = 0; h < G / 2; ++h) {
      if (kAhead) {
        e[h] = ahead[h];
        ahead[h] = reinterpret_cast<const uint32_t*>(list + i + G)[h];
      } else {
        e[h] = reinterpret_cast<const uint32_t*>(list + i)[h];
      }
    }
    uint32_t id[G], any = 0u, all = ~0u;
#pragma unroll
    for (int h = 0; h < G / 2; ++h) {
      id[2 * h] = e[h] & kIndexMask;
      id[2 * h + 1] = (e[h] >> 16) & kIndexMask;
      any |= e[h];
      all &= e[h];
    }
    constexpr uint32_t kKinds = (3u << kKindShift) | (3u << (16 + kKindShift));
    constexpr uint32_t kAllExact = (kExact << kKindShift) | (kExact << (16 + kKindShift));
    V al[G];
    if ((any & kKinds) == 0u) {
#pragma unroll
      for (int h = 0; h < G; ++h) al[h] = simple_alpha(pfx, p.y, cur[id[h]]);
    } else if ((all & kKinds) == kAllExact) {
#pragma unroll
      for (int h = 0; h < G; ++h) al[h] = exact_alpha(pfx, p.y, cur[id[h]]);
    } else {
#pragma unroll
      for (int h = 0; h < G; ++h)
        al[h] = any_alpha(pfx, p.y, cur[id[h]],
                          ((e[h / 2] >> (16 * (h & 1))) & (kExact << kKindShift)) != 0u);
    }
    V t[G + 1];  // T before each splat and after the last
    t[0] = p.T;
#pragma unroll
    for (int h = 0; h < G; ++h) t[h + 1] = PX::mul(t[h], PX::keep(al[h]));
    V ta[G];
#pragma unroll
    for (int h = 0; h < G; ++h) ta[h] = PX::mul(t[h], al[h]);
    bool ends = false;
#pragma unroll
    for (int k = 0; k < PX::kN; ++k)
      ends = ends || (PX::at(t[G], k) < kEndT && PX::at(t[0], k) > 0.0f);
    p.T = t[G];
    const bool any_ends = __any_sync(0xffffffffu, ends);
    if (any_ends) {
#pragma unroll
      for (int k = 0; k < PX::kN; ++k) {
        float tn = PX::at(t[1], k);
#pragma unroll
        for (int h = 1; h < G; ++h) {
          const bool before = PX::at(t[h], k) >= kEndT;
          PX::at(ta[h], k) = before ? PX::at(ta[h], k) : 0.0f;
          tn = before ? PX::at(t[h + 1], k) : tn;
        }
        const bool end = tn < kEndT;
        if (end && PX::at(t[0], k) > 0.0f) PX::at(p.fin, k) = tn;
        PX::at(p.T, k) = end ? 0.0f : tn;
      }
    }
#pragma unroll
    for (int h = 0; h < G; ++h) {
      const float4 c = cur[id[h]].c;
      p.cr = PX::fma(ta[h], c.x, p.cr);
      p.cg = PX::fma(ta[h], c.y, p.cg);
      p.cb = PX::fma(ta[h], c.z, p.cb);
    }
    if (any_ends && !__any_sync(0xffffffffu, px_live(p))) {
#pragma unroll
      for (int k = 0; k < PX::kN; ++k)
#pragma unroll
        for (int h = 0; h < G; ++h)
          if (PX::at(t[h], k) >= kEndT && PX::at(t[h + 1], k) < kEndT)
            used = max(used, position(id[h]) + 1);
      return false;
    }
  }
  return true;
}

// The staged splats [0, cnt) of one batch, by one warp.
template <typename PX>
__device__ __forceinline__ void warp_batch(const SplatStage* cur, uint32_t cnt, uint32_t none,
                                           float2 xr, float2 yr, uint16_t* list, float pfx, PX& p,
                                           uint32_t base, uint32_t& used) {
  if (!__any_sync(0xffffffffu, px_live(p))) return;
  for (uint32_t k0 = 0; k0 < cnt; k0 += kSegment) {
    const uint32_t n = cull_segment(cur, k0, min(cnt, k0 + kSegment), none, xr, yr, list);
    if (!blend_list<kGroup>(cur, list, n, pfx, p, [&](uint32_t i) { return base + i; }, used)) break;
    __syncwarp();  // the list is rewritten
  }
  if (px_live(p)) used = base + cnt;
}

struct TileGeom {
  uint32_t tile;      // global tile id
  uint32_t ox, oy;    // pixel origin of the tile in its view
  uint32_t W, H;      // view size
  uint2* image;       // the view's image
};

__device__ __forceinline__ TileGeom tile_geom(const RasterArgs& a, uint32_t t) {
  const uint32_t v =
      find_view(a.n_views, t, [&](uint32_t k) { return __ldg(&a.views[k].f.tile_base); });
  const ViewDesc& vd = a.views[v];
  const uint32_t lt = t - __ldg(&vd.f.tile_base);
  const uint32_t tx_count = __ldg(&vd.f.tile_count[0]);
  TileGeom g;
  g.tile = t;
  g.ox = (lt % tx_count) * a.tile_w;
  g.oy = (lt / tx_count) * a.tile_h;
  g.W = __ldg(&vd.f.viewport[0]);
  g.H = __ldg(&vd.f.viewport[1]);
  g.image = a.image + __ldg(&vd.pixel_base);
  return g;
}

// One thread per pixel, linear pixel order (the reference's layout).
__device__ void raster_tile_plain(const RasterArgs& a, const TileGeom& g, SplatStage* buf0,
                                  SplatStage* buf1, uint32_t* s_cost) {
  const uint32_t nt = a.tile_w * a.tile_h;  // == blockDim.x
  const uint32_t D = a.batch ? a.batch : nt;  // splats per staged batch
  const uint32_t tid = threadIdx.x;
  const uint32_t px = g.ox + tid % a.tile_w;
  const uint32_t py = g.oy + tid / a.tile_w;
  const bool in_bounds = px < g.W && py < g.H;
  const float pfx = (float)px + 0.5f, pfy = (float)py + 0.5f;

  const uint32_t start = __ldg(a.tile_offsets + g.tile);
  const uint32_t end = __ldg(a.tile_offsets + g.tile + 1);
  const uint32_t len = end > start ? end - start : 0u;
  const uint32_t nbatches = (len + D - 1) / D;

  Pixel p{0.f, 0.f, 0.f, 1.0f};
  bool done = !in_bounds;
  uint32_t used = 0;

  if (nbatches > 0) stage_batch(a.proj, a.values, start, end, D, nt, buf0);
  for (uint32_t bi = 0; bi < nbatches; ++bi) {
    SplatStage* cur = (bi & 1) ? buf1 : buf0;
    if (bi + 1 < nbatches) {
      stage_batch(a.proj, a.values, start + (bi + 1) * D, end, D, nt, (bi & 1) ? buf0 : buf1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    const uint32_t cnt = min(D, end - (start + bi * D));
    for (uint32_t k = tid; k < cnt; k += nt) prepare(cur[k], 0.0f);  // own copies are complete
    __syncthreads();
    if (!done) {
      for (uint32_t j = 0; j < cnt; ++j) {
        if (blend_one(pfx, pfy, cur[j], p)) {
          done = true;
          used = bi * D + j + 1;
          break;
        }
      }
      if (!done) used = bi * D + cnt;
    }
    if (__syncthreads_and(done)) {
      cp_async_wait<0>();  // drain the prefetch of the next batch before leaving
      break;
    }
  }
  if (in_bounds) {
    atomicMax(s_cost, used);
    store_pixel(g.image, g.W, px, py, p);
  }
}

// Culled variant: warps own compact pixel blocks and skip splats that no
// pixel of their block can blend.  blockDim.x == tile_w * tile_h, a multiple
// of 32.
__device__ void raster_tile_culled(const RasterArgs& a, const TileGeom& g, SplatStage* buf0,
                                   SplatStage* buf1, uint16_t* lists, uint32_t* s_cost) {
  const uint32_t nt = a.tile_w * a.tile_h, nthr = nt;
  const uint32_t D = a.batch ? a.batch : nt;  // splats per staged batch
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t lx, ly;
  const bool blocks = (a.tile_w % 8 == 0) && ((nthr / a.tile_w) % 4 == 0);
  const float reach = warp_box_reach(a, blocks);
  if (blocks) {  // 8x4 pixel block per warp
    const uint32_t bw = a.tile_w / 8;
    lx = (warp % bw) * 8 + (lane & 7);
    ly = (warp / bw) * 4 + (lane >> 3);
  } else {
    lx = tid % a.tile_w;
    ly = tid / a.tile_w;
  }
  const uint32_t px = g.ox + lx;
  const uint32_t py = g.oy + ly;
  const bool in_bounds = px < g.W && py < g.H;
  const float pfx = (float)px + 0.5f, pfy = (float)py + 0.5f;
  // the warp's pixel-centre bounding box
  float xlo = pfx, xhi = pfx, ylo = pfy, yhi = pfy;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    xlo = fminf(xlo, __shfl_xor_sync(0xffffffffu, xlo, o));
    xhi = fmaxf(xhi, __shfl_xor_sync(0xffffffffu, xhi, o));
    ylo = fminf(ylo, __shfl_xor_sync(0xffffffffu, ylo, o));
    yhi = fmaxf(yhi, __shfl_xor_sync(0xffffffffu, yhi, o));
  }

  const uint32_t start = __ldg(a.tile_offsets + g.tile);
  const uint32_t end = __ldg(a.tile_offsets + g.tile + 1);
  const uint32_t len = end > start ? end - start : 0u;
  const uint32_t nbatches = (len + D - 1) / D;

  Px1 p;
  p.y = pfy;
  if (!in_bounds) p.T = 0.0f;
  uint32_t used = 0;
  const float2 xr = make_float2(xlo, xhi), yr = make_float2(ylo, yhi);
  uint16_t* list = lists + warp * kListPitch;

  if (nbatches > 0) stage_batch(a.proj, a.values, start, end, D, nthr, buf0);
  for (uint32_t bi = 0; bi < nbatches; ++bi) {
    SplatStage* cur = (bi & 1) ? buf1 : buf0;
    if (bi + 1 < nbatches) {
      stage_batch(a.proj, a.values, start + (bi + 1) * D, end, D, nthr, (bi & 1) ? buf0 : buf1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    const uint32_t cnt = min(D, end - (start + bi * D));
    for (uint32_t k = tid; k < cnt; k += nthr) prepare(cur[k], reach);  // own copies are complete
    __syncthreads();
    warp_batch(cur, cnt, D, xr, yr, list, pfx, p, bi * D, used);
    if (__syncthreads_and(!px_live(p))) {
      cp_async_wait<0>();
      break;
    }
  }
  if (in_bounds) {
    atomicMax(s_cost, used);
    store_pixel(g.image, g.W, px, py, Pixel{p.cr, p.cg, p.cb, px_final(p, 0)});
  }
}

// The first 32 bytes of a record in one 256-bit load (records are 64-byte
// aligned).
__device__ __forceinline__ void load_record(const gs3d_projected_splat* p, SplatStage& s) {
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(s.a.x), "=f"(s.a.y), "=f"(s.a.z), "=f"(s.a.w), "=f"(s.b.x), "=f"(s.b.y), "=f"(s.b.z),
        "=f"(s.b.w)
      : "l"(p));
  s.c = __ldg(reinterpret_cast<const float4*>(p) + 2);
}

// ---- the warp variant: tiles whose sides divide by 8 ---------------------------
// A work item is one warp's: a region of up to 2x2 pixel blocks of 8x8 of a
// tile, a lane shading rows y and y + 4 of one column of a block.  Warps share
// nothing, so there are no block barriers (with a tile's splats staged per CTA
// they were 26% of the warps' time, waiting for the block with the most hits)
// and every warp takes its next item from the queue by itself.
//
// A warp walks the tile's splats 32 at a time: each lane fetches a record one
// step ahead, prepares it and tests it against the whole region, and the
// splats that may hit it (in order) are kept in shared memory.  Once they fill
// it, each block of the region queues its hits among them and blends
// (cull_segment, blend_list), its pixels' state parked in shared memory
// meanwhile.  So the tests against blocks and the padded steps run on full
// vectors: in a 64x32 tile most splats miss a given 16x16 region.
//
// Items of one block instead of a region (and of half a block, one pixel a
// lane) trade those gains for a shorter chain: they serve launches with fewer
// regions than resident warps, and the heaviest tiles.
constexpr uint32_t kRegionBlocks = 4;
constexpr uint32_t kItemWarps = 4;  // warps of a CTA (independent of one another)
constexpr uint32_t kKept = 104;     // splats kept before they are blended (a multiple of 8)
struct WarpSmem {
  SplatStage kept[kKept + 1];  // c.w = position in the tile's list; [kKept] hits nothing
  float4 state[kRegionBlocks][2][32];  // a block's pixels, per lane
  uint16_t list[kKept + 16];
  uint32_t n_sent, sent[kRegionBlocks - 1];  // places of blocks to come back for (lane 0)
};

__device__ __forceinline__ void load_px(const float4 (&st)[2][32], uint32_t lane, Px2& p) {
  const float4 a = st[0][lane], b = st[1][lane];  // T < 0: terminated with -T
  p.cr = make_float2(a.x, a.y);
  p.cg = make_float2(a.z, a.w);
  p.cb = make_float2(b.x, b.y);
  p.T = make_float2(fmaxf(b.z, 0.0f), fmaxf(b.w, 0.0f));
  p.fin = make_float2(fmaxf(-b.z, 0.0f), fmaxf(-b.w, 0.0f));
}
__device__ __forceinline__ void store_px(float4 (&st)[2][32], uint32_t lane, const Px2& p) {
  st[0][lane] = make_float4(p.cr.x, p.cr.y, p.cg.x, p.cg.y);
  st[1][lane] = make_float4(p.cb.x, p.cb.y, p.T.x > 0.0f ? p.T.x : -p.fin.x,
                            p.T.y > 0.0f ? p.T.y : -p.fin.y);
}
__device__ __forceinline__ void load_px(const float4 (&st)[2][32], uint32_t lane, Px1& p) {
  const float4 a = st[0][lane];
  p.cr = a.x;
  p.cg = a.y;
  p.cb = a.z;
  p.T = fmaxf(a.w, 0.0f);
  p.fin = fmaxf(-a.w, 0.0f);
}
__device__ __forceinline__ void store_px(float4 (&st)[2][32], uint32_t lane, const Px1& p) {
  st[0][lane] = make_float4(p.cr, p.cg, p.cb, p.T > 0.0f ? p.T : -p.fin);
}

// ---- blocks handed on ------------------------------------------------------------
// How far a region's warp has to walk its list is known only once its pixels
// have terminated, and the queue may run empty while a few warps still have
// thousands of splats before them.  A warp that finds no more items takes a
// place in a line and waits; a warp that sees some waiting hands blocks of its
// region on to them, with their pixels' state and the list position (the
// pixels' arithmetic does not change, so neither do the image and the costs).
// The n-th block handed on goes to the n-th place, so every waiting warp polls a
// word of its own.  Only the warps of the first kHelperCtas CTAs wait: a waiting
// warp keeps its CTA's shared memory from kernels of other streams (3 eager
// 1005x672 views at a time: 442 us alone and 199 us with three contexts in
// turn; with every warp waiting 442 and 299, with none 672 and 248).
//
// A block sent to a place stays its sender's until somebody takes it (compare and
// swap): the warp that waits there, or the sender, which comes back for what it
// has sent when it is done with the rest of its region.  So no block depends on
// anybody's waiting: a place may be sent to before it is taken, a warp that has
// waited wait_polls polls (a second and more) just leaves, and a place that it left
// behind keeps nothing.  (Blocks sent to places already taken only: 16 views of
// 640x360 1089 -> 1147 us.)
constexpr uint32_t kHelperCtas = 64;     // the others leave when the queue is empty
constexpr uint32_t kHandOnLeft = 512;    // list entries left below which nothing is handed on
struct PoolSlot {
  float4 state[2][32];
  uint32_t tile, view_x, view_y, k;
};
enum : uint32_t { PLACE_EMPTY = 0u, PLACE_BLOCK = 1u, PLACE_TAKEN = 2u };
// RasterArgs::pool_ctrl, all zero at launch: blocks sent, places taken, warps
// waiting, warps started and not yet gone, waits that ran out, blocks that their
// senders took back.
struct PoolCtrl {
  uint32_t sent, places, waiting, present, expired, taken_back;
};
__device__ __forceinline__ PoolCtrl* pool_ctrl(const RasterArgs& a) {
  return reinterpret_cast<PoolCtrl*>(a.pool_ctrl);
}
__device__ __forceinline__ uint4 pool_look(const RasterArgs& a) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(a.pool_ctrl)
               : "memory");
  return v;
}
__device__ __forceinline__ void send_block(const RasterArgs& a, const float4 (&st)[2][32],
                                           uint32_t place, uint32_t tile, uint32_t x, uint32_t y,
                                           uint32_t k) {
  const uint32_t lane = threadIdx.x & 31;
  PoolSlot& s = static_cast<PoolSlot*>(a.pool)[place];
  __stcg(&s.state[0][lane], st[0][lane]);
  __stcg(&s.state[1][lane], st[1][lane]);
  if (lane == 0) __stcg(reinterpret_cast<uint4*>(&s.tile), make_uint4(tile, x, y, k));
  __threadfence();
  __syncwarp();
  if (lane == 0) st_relaxed_u32(a.pool_places + place, PLACE_BLOCK);
}
// Lane 0: takes the block at a place that has been sent one; false if somebody has.
__device__ __forceinline__ bool take_block(const RasterArgs& a, uint32_t place) {
  const bool mine = atomicCAS(a.pool_places + place, PLACE_BLOCK, PLACE_TAKEN) == PLACE_BLOCK;
  __threadfence();
  return mine;
}
// Lane 0 of a warp without work: takes a place and waits for a block; its place, or
// ~0u once every warp waits (nobody has a block to send) or the polls run out.
__device__ __forceinline__ uint32_t wait_for_block(const RasterArgs& a) {
  PoolCtrl* c = pool_ctrl(a);
  atomicAdd(&c->waiting, 1u);
  uint32_t place = atomicAdd(&c->places, 1u), polls = 0;
  for (; place < kRasterPlaces && polls < a.wait_polls; ++polls) {
    if (ld_relaxed_u32(a.pool_places + place) != PLACE_EMPTY) {
      atomicSub(&c->waiting, 1u);
      if (take_block(a, place)) return place;
      atomicAdd(&c->waiting, 1u);  // its sender has
      place = atomicAdd(&c->places, 1u);
      continue;
    }
    if ((polls & 3u) == 3u) {
      const uint4 v = pool_look(a);
      if (v.z >= v.w) break;
    }
    __nanosleep(300);
  }
  if (polls == a.wait_polls) atomicAdd(&c->expired, 1u);
  atomicSub(&c->waiting, 1u);
  atomicSub(&c->present, 1u);
  return ~0u;
}

// Shades the nbx x nby blocks at pixel (x0, y0) of the view; returns the
// region's share of the tile's cost.  FINE: one block, whose chain through the
// list is what counts: records are fetched two steps ahead (into the states of
// the blocks that it does not have), a splat that may hit the region is queued
// at once, and few are kept before they are blended.
template <typename PX, bool FINE, bool HAND_ON>
__device__ uint32_t shade_region(const RasterArgs& a, const TileGeom& g, uint32_t x0, uint32_t y0,
                                 uint32_t nbx, uint32_t nby, WarpSmem& w,
                                 uint32_t slot_in = ~0u) {
  constexpr uint32_t kRows = PX::kN == 2 ? 8 : 4;  // of a block
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nb = FINE ? 1u : nbx * nby;
  const float bx0 = (float)x0 + 0.5f, by0 = (float)y0 + 0.5f;
  float2 xr = make_float2(bx0, bx0 + (float)(8 * nbx - 1));
  float2 yr = make_float2(by0, by0 + (float)(kRows * nby - 1));
  auto px_of = [&](uint32_t b) { return x0 + (b % nbx) * 8 + (lane & 7); };
  auto py_of = [&](uint32_t b) { return y0 + (b / nbx) * kRows + (lane >> 3); };

  uint32_t alive = 0;  // blocks with a pixel that has not terminated
  uint32_t owned = (1u << nb) - 1u;
  const uint32_t start = __ldg(a.tile_offsets + g.tile);
  const uint32_t last = __ldg(a.tile_offsets + g.tile + 1);
  const uint32_t end = last > start ? last : start;
  uint32_t begin = start;
  if (HAND_ON && FINE && PX::kN == 2 && slot_in != ~0u) {  // a block handed on
    const PoolSlot& ps = static_cast<PoolSlot*>(a.pool)[slot_in];
    w.state[0][0][lane] = __ldcg(&ps.state[0][lane]);
    w.state[0][1][lane] = __ldcg(&ps.state[1][lane]);
    begin = __ldcg(&ps.k);
    alive = 1u;
  } else {
    for (uint32_t b = 0; b < nb; ++b) {
      PX p;
#pragma unroll
      for (int i = 0; i < PX::kN; ++i)
        if (!(px_of(b) < g.W && py_of(b) + 4 * i < g.H)) PX::at(p.T, i) = 0.0f;
      store_px(w.state[b], lane, p);
      if (__any_sync(0xffffffffu, px_live(p))) alive |= 1u << b;
    }
  }
  uint32_t used = 0, n = 0;

  // blends the n kept splats into every block
  auto flush = [&]() {
    if (FINE && lane < 2 * kFineGroup) w.list[n + lane] = (uint16_t)kKept;  // whole steps
    __syncwarp();
    for (uint32_t b = 0; b < nb; ++b) {
      if (!((alive >> b) & 1u)) continue;
      const float fx = bx0 + (float)((b % nbx) * 8), fy = by0 + (float)((b / nbx) * kRows);
      const uint32_t hits =
          FINE ? n
               : cull_segment(w.kept, 0, n, kKept, make_float2(fx, fx + 7.0f),
                              make_float2(fy, fy + (float)(kRows - 1)), w.list);
      PX p;
      load_px(w.state[b], lane, p);
      const float ly = fy + (float)(lane >> 3);
      PX::at(p.y, 0) = ly;
      if (PX::kN == 2) PX::at(p.y, 1) = ly + 4.0f;
      if (!blend_list<FINE && PX::kN == 1 ? kFineGroup : kGroup>(w.kept, w.list, hits, fx + (float)(lane & 7), p,
                      [&](uint32_t i) { return __float_as_uint(w.kept[i].c.w); }, used))
        alive &= ~(1u << b);
      store_px(w.state[b], lane, p);
      __syncwarp();  // the list is rewritten
    }
    n = 0;
  };
  // keeps the lanes' splats (list positions k + lane) that may hit the region
  auto keep = [&](SplatStage& s, uint32_t k) {
    prepare(s, 24.0f);  // the region's pixel centres lie within 15 sqrt(2)
    const bool hit = k + lane < end && rect_may_hit(s.a, s.b, xr, yr);
    const uint32_t mask = __ballot_sync(0xffffffffu, hit);
    if (hit) {
      const uint32_t i = n + __popc(mask & lanemask_lt());
      s.c.w = __uint_as_float(k - start + lane);
      w.kept[i] = s;
      if (FINE) w.list[i] = (uint16_t)(i | (__float_as_uint(s.b.w) << kKindShift));
    }
    n += __popc(mask);
  };
  uint32_t id = 0;  // of the record to fetch next
  auto fetch_id = [&](uint32_t k) {
    if (k + lane < end) id = __ldg(a.values + k + lane);
  };

  if (FINE) {
    SplatStage* ring = reinterpret_cast<SplatStage*>(&w.state[1][0][0]);  // 2 steps of 32
    auto fetch = [&](uint32_t k, uint32_t slot) {  // a lane reads back only what it fetched
      if (k + lane < end) {
        const float4* src = reinterpret_cast<const float4*>(a.proj + id);
        SplatStage* dst = ring + slot * 32 + lane;
        cp_async16(&dst->a, src);
        cp_async16(&dst->b, src + 1);
        cp_async16(&dst->c, src + 2);
      }
      cp_async_commit();
    };
    fetch_id(begin);
    fetch(begin, 0);
    fetch_id(begin + 32);
    fetch(begin + 32, 1);
    fetch_id(begin + 64);
    uint32_t slot = 0;
    for (uint32_t k = begin; alive; k += 32, slot ^= 1u) {
      const bool more = k < end;
      if (more) {
        cp_async_wait<1>();
        SplatStage s = ring[slot * 32 + lane];
        keep(s, k);
        fetch(k + 64, slot);
        fetch_id(k + 96);
      }
      if (more ? n > kKept - 48 : n > 0) flush();
      if (!more) break;
    }
    cp_async_wait<0>();
  } else {
    SplatStage next{};
    fetch_id(start);
    if (start + lane < end) load_record(a.proj + id, next);
    fetch_id(start + 32);
    for (uint32_t k = start; alive; k += 32) {
      const bool more = k < end;
      if (more) {
        SplatStage s = next;
        if (k + 32 + lane < end) load_record(a.proj + id, next);
        fetch_id(k + 64);
        keep(s, k);
      }
      if (more ? n > kKept - 32 : n > 0) {
        uint4 pool = make_uint4(0u, 0u, 0u, 0u);
        const uint32_t at = k + 32;
        const bool look = HAND_ON && end > at + kHandOnLeft && (alive & (alive - 1u)) != 0u;
        if (look && lane == 0) pool = pool_look(a);
        flush();
        if (look && (alive & (alive - 1u)) != 0u) {
          const int places =
              __shfl_sync(0xffffffffu, (int)min(pool.y, kRasterPlaces) - (int)pool.x, 0);
          for (int i = 0; i < places && (alive & (alive - 1u)) != 0u; ++i) {
            uint32_t place = 0;
            if (lane == 0) place = atomicAdd(&pool_ctrl(a)->sent, 1u);
            place = __shfl_sync(0xffffffffu, place, 0);
            if (place >= kRasterPlaces) break;
            const uint32_t b = 31 - __clz(alive);
            send_block(a, w.state[b], place, g.tile, x0 + (b % nbx) * 8, y0 + (b / nbx) * kRows,
                       at);
            if (lane == 0) w.sent[w.n_sent++] = place;
            alive &= ~(1u << b);
            owned &= ~(1u << b);
          }
          if ((alive & (alive - 1u)) == 0u) {  // one block left: test against it alone
            const uint32_t b = 31 - __clz(alive);
            const float fx = bx0 + (float)((b % nbx) * 8), fy = by0 + (float)((b / nbx) * kRows);
            xr = make_float2(fx, fx + 7.0f);
            yr = make_float2(fy, fy + (float)(kRows - 1));
          }
        }
      }
      if (!more) break;
    }
  }

  for (uint32_t b = 0; b < nb; ++b) {
    if (HAND_ON && !((owned >> b) & 1u)) continue;
    PX p;
    load_px(w.state[b], lane, p);
#pragma unroll
    for (int i = 0; i < PX::kN; ++i) {
      const uint32_t px = px_of(b), py = py_of(b) + 4 * i;
      if (px < g.W && py < g.H)
        store_pixel(g.image, g.W, px, py,
                    Pixel{PX::at(p.cr, i), PX::at(p.cg, i), PX::at(p.cb, i), px_final(p, i)});
    }
  }
  __syncwarp();
  return alive ? end - start : __reduce_max_sync(0xffffffffu, used);
}

// Persistent warps.  Work items: first those of the heavy tiles at the head of
// an order by decreasing expected cost, each half a block; then the regions of
// the other tiles in order, or their blocks where a launch has too few regions
// (a.fine); then blocks handed on.
template <bool HAND_ON>
__global__ void __launch_bounds__(kItemWarps * 32, 5) raster_kernel_warps(RasterArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  WarpSmem& w = reinterpret_cast<WarpSmem*>(smem)[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31;
  after_predecessor(a.heavy);
  if (lane == 0) {
    w.kept[kKept].a = make_float4(0.f, 0.f, -1.f, 0.f);
    w.kept[kKept].b = make_float4(0.f, 0.f, 0.f, -1.f);
    w.kept[kKept].c = make_float4(0.f, 0.f, 0.f, 0.f);
    w.n_sent = 0;
    if (HAND_ON) atomicAdd(&pool_ctrl(a)->present, 1u);
  }
  __syncwarp();
  const uint32_t bw = a.tile_w / 8, blocks = bw * (a.tile_h / 8);
  const uint32_t rw = (bw + 1) / 2, regions = rw * ((a.tile_h / 8 + 1) / 2);
  const uint32_t heavy = a.heavy != nullptr ? min(__ldg(a.heavy), a.num_tiles) : 0u;
  const uint32_t per_tile = a.fine ? blocks : regions;
  const uint64_t heavy_items = (uint64_t)heavy * 2 * blocks;
  const uint64_t items = heavy_items + (uint64_t)(a.num_tiles - heavy) * per_tile;
  bool queued = true;  // the queue may still hold items
  for (;;) {
    unsigned long long item = items;
    uint32_t slot = ~0u;
    if (HAND_ON) {  // a block of the region just shaded that nobody has taken
      if (lane == 0) {
        while (w.n_sent && slot == ~0u) {
          const uint32_t place = w.sent[--w.n_sent];
          if (take_block(a, place)) {
            atomicAdd(&pool_ctrl(a)->taken_back, 1u);
            slot = place;
          }
        }
      }
      slot = __shfl_sync(0xffffffffu, slot, 0);
    }
    if (queued && (!HAND_ON || slot == ~0u)) {
      if (lane == 0) item = atomicAdd(a.queue_counter, 1ull);
      item = __shfl_sync(0xffffffffu, item, 0);
      queued = item < items;
    }
    uint32_t t, x, y, nbx = 1, nby = 1;
    const bool in_heavy = item < heavy_items;
    bool fine = a.fine;
    TileGeom g;
    if (HAND_ON ? item < items : queued) {
      uint32_t sub;
      if (in_heavy) {
        t = (uint32_t)(item / (2 * blocks));
        sub = (uint32_t)(item - (uint64_t)t * (2 * blocks));
      } else {
        const uint64_t j = item - heavy_items;
        t = (uint32_t)(j / per_tile);
        sub = (uint32_t)(j - (uint64_t)t * per_tile);
        t += heavy;
      }
      if (a.order != nullptr) t = __ldg(a.order + t);
      g = tile_geom(a, t);
      if (in_heavy) {
        const uint32_t b = sub >> 1;
        x = g.ox + (b % bw) * 8;
        y = g.oy + (b / bw) * 8 + (sub & 1) * 4;
      } else if (fine) {
        x = g.ox + (sub % bw) * 8;
        y = g.oy + (sub / bw) * 8;
      } else {
        const uint32_t rx = 2 * (sub % rw), ry = 2 * (sub / rw);
        x = g.ox + rx * 8;
        y = g.oy + ry * 8;
        nbx = min(2u, bw - rx);
        nby = min(2u, a.tile_h / 8 - ry);
      }
    } else {
      if (!HAND_ON) break;
      if (slot == ~0u) {
        if (blockIdx.x >= kHelperCtas) {
          if (lane == 0) atomicSub(&pool_ctrl(a)->present, 1u);
          break;
        }
        if (lane == 0) slot = wait_for_block(a);
        slot = __shfl_sync(0xffffffffu, slot, 0);
        if (slot == ~0u) break;
      }
      const uint4 info =
          __ldcg(reinterpret_cast<const uint4*>(&static_cast<PoolSlot*>(a.pool)[slot].tile));
      t = info.x;
      x = info.y;
      y = info.z;
      g = tile_geom(a, t);
      fine = true;
    }
    uint32_t cost;
    if (in_heavy) {
      cost = shade_region<Px1, true, HAND_ON>(a, g, x, y, 1, 1, w);
    } else if (fine) {
      cost = shade_region<Px2, true, HAND_ON>(a, g, x, y, 1, 1, w, slot);
    } else {
      cost = shade_region<Px2, false, HAND_ON>(a, g, x, y, nbx, nby, w);
    }
    if (lane == 0 && a.tile_costs != nullptr && cost)
      atomicMax(a.tile_costs + t, cost);  // zeroed before the launch; max over a tile's items
  }
}

// Persistent CTAs over the queue of tiles; MODE 0: one thread per pixel,
// linear; 1: culled, 8x4 warp blocks.
template <int MODE>
__device__ __forceinline__ void raster_loop(const RasterArgs& a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t D = a.batch ? a.batch : a.tile_w * a.tile_h;
  SplatStage* buf0 = reinterpret_cast<SplatStage*>(smem);
  SplatStage* buf1 = buf0 + D + 1;  // entry D of both: a splat that hits nothing
  uint16_t* lists = reinterpret_cast<uint16_t*>(buf1 + D + 1);
  __shared__ uint32_t s_item, s_cost;
  if (MODE != 0 && threadIdx.x < 2) {
    SplatStage& none = (threadIdx.x ? buf1 : buf0)[D];
    none.a = make_float4(0.f, 0.f, -1.f, 0.f);
    none.b = make_float4(0.f, 0.f, 0.f, -1.f);
    none.c = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  while (true) {
    if (threadIdx.x == 0) {
      s_item = (uint32_t)atomicAdd(a.queue_counter, 1ull);
      s_cost = 0u;
    }
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= a.num_tiles) break;
    const uint32_t t = a.order != nullptr ? __ldg(a.order + item) : item;
    const TileGeom g = tile_geom(a, t);
    if (MODE == 1) {
      raster_tile_culled(a, g, buf0, buf1, lists, &s_cost);
    } else {
      raster_tile_plain(a, g, buf0, buf1, &s_cost);
    }
    __syncthreads();  // s_cost complete; shared buffers free for the next tile
    if (threadIdx.x == 0 && a.tile_costs != nullptr) atomicMax(a.tile_costs + t, s_cost);
  }
}

__global__ void raster_kernel_plain(RasterArgs a) { raster_loop<0>(a); }
__global__ void __launch_bounds__(1024) raster_kernel_culled(RasterArgs a) { raster_loop<1>(a); }

// Variant, block size, staged batch and resident CTAs per SM of the raster
// launch for `a` (the occupancy is computed once per device and shape).
struct RasterConfig {
  int mode;
  uint32_t threads, D;
  size_t smem;
  int per_sm;
  uint32_t regions, blocks;  // work items per tile of the warp variant
  void (*kern)(RasterArgs);
};

// Two staged batches and, for the culled variants, a list per warp.
size_t raster_smem(int mode, uint32_t D, uint32_t threads) {
  if (mode == 2) return kItemWarps * sizeof(WarpSmem);
  return 2 * ((size_t)D + 1) * sizeof(SplatStage) +
         (mode != 0 ? (size_t)(threads / 32) * kListPitch * sizeof(uint16_t) : 0);
}

cudaError_t raster_config(const RasterArgs& a, RasterConfig* cfg) {
  const uint32_t nt = a.tile_w * a.tile_h;
  if (a.batch % 32 != 0 || a.batch > 1024) return cudaErrorInvalidValue;
  const bool culled = nt % 32 == 0;  // whole warps; else pixel by pixel
  // warp items where the tile splits into 8x8 blocks
  const int mode = !culled ? 0 : (a.tile_w % 8 == 0 && a.tile_h % 8 == 0) ? 2 : 1;
  if (mode != 2 && nt > 1024) return cudaErrorInvalidValue;  // one thread a pixel
  const uint32_t D = mode == 2 ? 0u : a.batch ? a.batch : nt;
  const uint32_t threads = mode == 2 ? kItemWarps * 32 : nt;
  const size_t smem = raster_smem(mode, D, threads);
  auto kern = mode == 2 ? raster_kernel_warps<false> : mode == 1 ? raster_kernel_culled
                                                           : raster_kernel_plain;
  // launch configuration per (device, variant, tile area, batch), computed
  // once per process (the shared-memory attribute is a per-device setting)
  static std::mutex mu;
  static std::map<uint64_t, int> cache;
  int dev = 0;
  {
    const cudaError_t e = current_device(&dev);
    if (e != cudaSuccess) return e;
  }
  const uint64_t key = ((uint64_t)dev << 48) | ((uint64_t)mode << 40) |
                       ((uint64_t)threads << 20) | D;
  int per_sm = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) per_sm = it->second;
  }
  if (per_sm == 0) {
    // one attribute per kernel, set to the largest batch's footprint so that
    // configurations cached earlier keep fitting
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)raster_smem(mode, 1024, 1024));
    if (e == cudaSuccess && mode == 2)
      e = cudaFuncSetAttribute(raster_kernel_warps<true>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, (int)threads, smem);
    if (e != cudaSuccess) return e;
    per_sm = std::max(n, 1);
    std::lock_guard<std::mutex> lock(mu);
    cache[key] = per_sm;
  }
  const uint32_t bw = a.tile_w / 8, bh = a.tile_h / 8;
  *cfg = RasterConfig{mode,   threads, D,   smem, per_sm, mode == 2 ? ((bw + 1) / 2) * ((bh + 1) / 2) : 1u,
                      mode == 2 ? bw * bh : 1u, kern};
  return cudaSuccess;
}

// Launches with fewer regions than this many times the resident warps are
// shaded by blocks: they are bound by the longest item's chain (raster of a
// 400k-splat frame with 0.75 regions a warp: 302 -> 143 us, of a 100k-splat one
// with 1.2: 124 -> 64 us; a 3M-splat frame with 2.7: 342 us by regions, 473 by
// blocks).
constexpr float kFineWaves = 1.75f;
// Blocks are handed on in the row-major order, which cannot know the long lists
// beforehand; in an order by predicted costs, which may be wrong about one (eight
// views of opaque and translucent clusters at 1080p in learned order, raster at
// 16x16 tiles 7199 -> 3559 us, 32x32 5023 -> 3656, 64x32 5373 -> 3644; of evenly
// spread ones 2432 -> 2442); and in the order by key counts up to this many regions
// a warp (16 views of 640x360 with 5 regions a warp: raster 975 -> 871 us; with 20
// and more the tail is short and the check costs 2%).
constexpr float kHandOnWaves = 8.0f;

}  // namespace

cudaError_t raster_shape(const RasterArgs& a, int sm_count, uint32_t* items_per_tile,
                         uint32_t* resident) {
  RasterConfig cfg;
  const cudaError_t e = raster_config(a, &cfg);
  if (e != cudaSuccess) return e;
  *items_per_tile = cfg.regions;
  *resident = (uint32_t)sm_count * (uint32_t)cfg.per_sm * (cfg.mode == 2 ? kItemWarps : 1u);
  return cudaSuccess;
}

size_t raster_pool_bytes() { return kRasterPlaces * sizeof(PoolSlot); }

cudaError_t launch_raster(const RasterArgs& args, int sm_count, LaunchStream s) {
  if (args.num_tiles == 0) return cudaSuccess;
  RasterArgs a = args;
  RasterConfig cfg;
  cudaError_t e = raster_config(a, &cfg);
  if (e != cudaSuccess) return e;
  const uint32_t ctas = (uint32_t)sm_count * (uint32_t)cfg.per_sm;
  uint64_t max_ctas = a.num_tiles;
  if (cfg.mode == 2) {
    const float waves = (float)a.num_tiles * (float)cfg.regions / (float)(ctas * kItemWarps);
    a.fine = waves <= kFineWaves;
    if (!a.fine && (a.order == nullptr || a.predicted || waves < kHandOnWaves))
      cfg.kern = raster_kernel_warps<true>;
    max_ctas = ((uint64_t)a.num_tiles * cfg.blocks * 2 + kItemWarps - 1) / kItemWarps;
  } else {
    a.heavy = nullptr;  // split items exist in the warp variant only
  }
  const uint32_t grid = (uint32_t)std::min<uint64_t>(max_ctas, ctas);
  if (cfg.mode == 2) return launch_after(cfg.kern, grid, cfg.threads, cfg.smem, s, a);
  cfg.kern<<<grid, cfg.threads, cfg.smem, s>>>(a);
  return cudaGetLastError();
}

}  // namespace gs3d
