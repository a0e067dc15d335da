// trace_fast.cuh -- the RK step of trace_common.cuh as straight-line code.
//
// The tracers are bound by instruction issue, not by memory: the plain form
// of a jittered RK4 step (rk_step), with its 17 IEEE divisions, 10 square roots
// and the index clamps of the four bilinear samples, executes 815 thread
// instructions (ncu).  Here a step is evaluated without any of them and
// with one test at its end: the step's values are those of rk_step bit for
// bit when every guard below holds, and a lane for which one does not hold
// (a sample next to the grid's edge, a NaN, an overflow, a jittered component
// below 2^-30, one generator state in 10^9) evaluates the step again with
// rk_step.
//
// What makes each shortcut exact:
//
//   unit vectors    u / |u| from one reciprocal square root estimate, square
//                   root and quotients correctly rounded (unit_math.cuh).
//   pixel index     trunc(v) for 0 <= v < 2^23 is v + 2^23 rounded towards
//                   zero; the sum's low bits are the integer, so neither
//                   conversion unit nor clamp is used (the clamps cannot bind
//                   for samples within one pixel of an interior pixel).
//   quantisation    trunc(|v| 2^k) the same way in one fused operation; the
//                   host checks that a step is below 127 units.
//   jitter draws    the generator's reduction without its last conditional
//                   subtraction, which acts on 5 of 2^32 states (guarded).
//   products by a power of two fused with the sum that follows (exact).
//   adaptive dt     DT_MAX, without root and division, when a test with
//                   margin shows the error small enough; else as next_dt.
//
// x and y of a step go through the packed two-float instructions of sm_100a
// (each half rounded as the scalar instruction rounds it), which halve the
// issue slots of the bilinear sums and the step's products.
//
// Measured (B200, both directions, RK4): 815 -> 414 thread instructions per step
// on 4096^2 fan terrain with one trajectory a seed (421 on 1024^2 incised relief,
// 2x2); 2x2, 1.64e10 steps: 505 -> 274 ms; 256^2 hills, RK2: 11.9 -> 6.2 ms.  What is left is
// bound by the float units (80 % of the issue slots' worth of work: packed
// operations take two cycles, the generator's wide products four), so
// variants that trade slots for float work (wide products for the addresses
// or the draws' reduction) measured 2 to 5 % slower, fewer or more resident
// warps (24, 36, 38, 40 against 32 per SM) 0 to 4 % slower.
#pragma once
#include "capi_util.cuh"
#include "trace_common.cuh"
#include "unit_math.cuh"

namespace slm {

typedef u64 F2;  // two floats in a register pair: x low, y high

__device__ __forceinline__ F2 pack2(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ F2 splat2(float v) { return pack2(v, v); }
__device__ __forceinline__ void unpack2(F2 a, float& x, float& y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 add2_rz(F2 a, F2 b) {
    F2 r;
    asm("add.rz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// three-operand minimum, NaN if any operand is
__device__ __forceinline__ float min3_nan(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

constexpr float FAST_MAGIC = 8388608.0f;           // 2^23
constexpr uint32_t FAST_MAGIC_BITS = 0x4B000000u;  // its bit pattern
constexpr float FAST_S_MIN = 0x1p-60f;             // least square of a vector or a jittered component
constexpr uint32_t FAST_C_BITS = 0x21800000u;      // 2^-60, the least component that is not zero
constexpr float FAST_JITTER = 0x1p-8f;             // least magnitude of STEP_JITTERED

constexpr uint32_t LEHMER_M = 0xfffffffbu;

// How a launch forms its steps.  A flow component that is exactly 0 is nothing
// unusual (planes along an axis, and relief in whole metres or centimetres), so
// no form may leave such steps to step_exact: a plane along an axis, RK4, then
// took 401 ms where one oblique to the axes took 134 (rk_step for all: 305).
//
//   STEP_JITTERED  the components after the jitter are tested: at least 2^-30
//                  each.  That covers the flow's own: where one is too small
//                  for an exact quotient (below 2^-103, or its quotient not
//                  normal), its unit component is below 2^-72, and the
//                  jittered one, at least 2^-30, is the jitter alone.
//   STEP_FAINT     a jitter below 2^-8, or none, may leave a component at 0 or
//                  next to it: components before and after it are tested to be
//                  0 or at least 2^-60, which takes one instruction and a half
//                  a stage more (1 % of the time of a launch).
//   STEP_PLAIN     no jitter and no second normalisation; tested as STEP_FAINT.
enum StepForm : int { STEP_GENERAL = 0, STEP_JITTERED = 1, STEP_FAINT = 2, STEP_PLAIN = 3 };

// u / |u| as rk_step forms it: |u| = sqrt(x*x + y*y), both components divided
// by it.  Exact, but for the sign of a zero component (which no later value
// depends on), when s = x*x + y*y >= 2^-60 is finite and each component is
// zero or at least 2^-60: the residuals are then exact and the quotients normal.
__device__ __forceinline__ F2 unit_fast(F2 u, float& xx, float& yy, float& s) {
    unpack2(mul2(u, u), xx, yy);
    s = __fadd_rn(xx, yy);
    const float y0 = rsqrt_estimate(s);
    const float len = root_from(s, y0), r = reciprocal_from(len, y0);
    const F2 r2 = splat2(r), q = mul2(u, r2);
    return fma2(fma2(splat2(-len), q, u), r2, q);
}

// sqrt(x*x + y*y) of a quantised step (multiples of 2^-k, so the sum of
// squares is 0 or above 2^-40; the added 2^-100 is absorbed unless it is 0,
// where it keeps the estimate finite and the root 0)
__device__ __forceinline__ float quantised_length(float s) {
    return root_from(s, rsqrt_estimate(__fadd_rn(s, 0x1p-100f)));
}

// A grid as the fast step uses it.  Part of the launch's parameters in the
// single-grid kernels, one per lane in the batched one.
struct FastGeo {
    uint32_t pitch;     // bytes of a grid row of vectors
    uint32_t koff;      // byte offset of a pixel's vector: pitch * bits(2^23 + xi) + 8 * bits(2^23 + yi) + koff
    uint32_t off_last;  // largest such offset whose four taps lie in the grid
    float cx, cy;       // interior pixels: |xi - cx| <= rx, |yi - cy| <= ry, that is
    float rx, ry;       //   1 <= xi <= nxp - 3 and 1 <= yi <= nyp - 3 (one less on long axes)
    float kerr;         // dt^2 kerr >= |d2 - d1|^2 implies a next dt of DT_MAX
    float gs_rcp;       // IEEE reciprocal of GRID_SCALE
};

// base: the grid's first pixel in its arrays
__host__ __device__ __forceinline__ FastGeo make_fast_geo(uint32_t nxp, uint32_t nyp, float gs, float dt_max,
                                                          float adjusted_max_error, uint32_t base) {
    FastGeo f;
    f.pitch = 8u * nyp;
    f.koff = 8u * base - (f.pitch + 8u) * FAST_MAGIC_BITS;
    f.off_last = 8u * (base + nxp * nyp - nyp - 2u);
    f.cx = 0.5f * (float)(nxp - 2u);
    f.cy = 0.5f * (float)(nyp - 2u);
    // A step's samples lie at most 0.99 pixels from its start (fast_grid) and
    // the coordinates' rounding stays below the other 0.01 up to 2^16: no clamp
    // can bind for a start one pixel (at its upper side two) inside the grid.
    // With the usual padding of 2 that is every pixel of the region; with one
    // pixel less, as beyond 2^16, its last row and column are not, and 3 % of
    // a warp's steps on 256^2 meet one (24 tiles, RK2: 102 ms, now 95).
    f.rx = 0.5f * ((float)nxp - (nxp <= 65536u ? 4.0f : 6.0f));
    f.ry = 0.5f * ((float)nyp - (nyp <= 65536u ? 4.0f : 6.0f));
    f.gs_rcp = 1.0f / gs;
    const float k = adjusted_max_error * gs / dt_max;
    f.kerr = (k > 0x1p-30f && k < 0x1p30f) ? k * k * (1.0f - 0x1p-16f) : -1.0f;  // -1: never by the test
    return f;
}

// Constants of the fast step, formed on the host: the kernels' loops would
// otherwise form them again in every step (they do not fit the registers).
// As pairs, they are operands of the packed instructions.
struct FastConst {
    float2 pp5, pad, magic, one, half, two, mag, draw, draw0, div6_hi, div6_lo;
    float res, inv, minus_magic_inv;
};

static inline FastConst make_fast_const(const slm_params& p) {
    const auto both = [](float v) { return make_float2(v, v); };
    FastConst k;
    k.pp5 = both(p.pad_width_pp5);
    k.pad = both((float)p.pad_width);
    k.magic = both(FAST_MAGIC);
    k.one = both(1.0f);
    k.half = both(0.5f);
    k.two = both(2.0f);
    k.mag = both(p.jitter_magnitude);
    k.draw = both(0x1p-32f);
    k.draw0 = both(-0.5f);
    k.div6_hi = both(0x1.555556p-3f);
    k.div6_lo = both(-0x1.555556p-28f);
    k.res = (float)p.trajectory_resolution;
    k.inv = 1.0f / k.res;  // a power of two
    k.minus_magic_inv = -FAST_MAGIC * k.inv;
    return k;
}

__device__ __forceinline__ F2 as_f2(const float2& v) { return pack2(v.x, v.y); }

// a + m where m is a product of its own rounding.  With add2(mul2(..), a) here
// (contraction is switched off) 8.6 M of the 16.8 M pairs of slm_selftest_packed
// come out as a fused operation's, and the oracle's sums are missed; as m * 1 + a
// with a 1 that is a kernel argument every pair is rounded twice.
__device__ __forceinline__ F2 add2_product(F2 m, F2 a, const FastConst& k) { return fma2(m, as_f2(k.one), a); }

// Whether a grid's steps can be evaluated by step_fast: quantised steps below
// 127 units (so below a pixel, and no conversion wraps), coordinates that
// 2^23 + i holds.  Grids below 8 pixels have no interior worth the test.
__host__ __device__ __forceinline__ bool fast_grid(uint32_t nxp, uint32_t nyp, uint32_t base, float cf,
                                                   float dt_max, uint32_t resolution) {
    const float h = fabsf(cf) * dt_max;
    return nxp >= 8u && nyp >= 8u && nxp <= (1u << 22) && nyp <= (1u << 22) &&
           (u64)nxp * nyp + base <= (1ull << 29) &&  // 32-bit byte offsets
           dt_max > 0.0f && h >= 0x1p-20f && h <= 0.99f && h * (float)resolution <= 126.0f && fabsf(cf) <= 0x1p30f;
}

// The conditions on the parameters all grids of a launch share: a resolution
// that is a power of two, a jitter that keeps quotients normal, a dt rule
// that never lengthens a step.
__host__ __device__ __forceinline__ bool fast_params(const slm_params& p) {
    const uint32_t r = p.trajectory_resolution;
    const float m = fabsf(p.jitter_magnitude);
    return r != 0u && (r & (r - 1u)) == 0u && r <= (1u << 20) && (m == 0.0f || (m >= 0x1p-40f && m <= 0x1p10f)) &&
           p.adjusted_max_error >= 0.0f && p.pad_width < (1u << 20);
}

// The form of a jittered launch whose grids fast_grid admits.
static inline StepForm jittered_form(const slm_params& p) {
    return !fast_params(p) ? STEP_GENERAL : fabsf(p.jitter_magnitude) >= FAST_JITTER ? STEP_JITTERED : STEP_FAINT;
}

// 2^23 + clamped pixel index of a position, per axis (get_array_idx); the
// clamp written so that NaN gives pixel 0, as axis_index
__device__ __forceinline__ F2 pixel_magic_clamped(Vec2 a, float pp5, uint32_t nxp, uint32_t nyp) {
    const float vx = fminf(fmaxf(a.x + pp5, 0.0f), (float)(nxp - 1u));
    const float vy = fminf(fmaxf(a.y + pp5, 0.0f), (float)(nyp - 1u));
    return pack2(__fadd_rz(vx, FAST_MAGIC), __fadd_rz(vy, FAST_MAGIC));
}

__device__ __forceinline__ uint32_t offset_from_magic(F2 t, const FastGeo& f) {
    float tx, ty;
    unpack2(t, tx, ty);
    return f.pitch * __float_as_uint(tx) + (8u * __float_as_uint(ty) + f.koff);
}

// Bilinear flow at a, whose pixel is floor2 (at byte offset `off` of uv);
// unnormalised.
__device__ __forceinline__ F2 taps_fast(F2 a, F2 floor2, uint32_t off, const float2* __restrict__ uv,
                                        const FastGeo& f, const FastConst& k) {
    const F2 w = add2(sub2(a, floor2), as_f2(k.pad));
    const F2 w1 = sub2(as_f2(k.one), w);
    float wr, wu, wl, wd;
    unpack2(w, wr, wu);
    unpack2(w1, wl, wd);
    const char* b = reinterpret_cast<const char*>(uv);
    const F2* p = reinterpret_cast<const F2*>(b + off);
    const F2* q = reinterpret_cast<const F2*>(b + (off + f.pitch));
    const F2 q00 = __ldg(p), q01 = __ldg(p + 1), q10 = __ldg(q), q11 = __ldg(q + 1);
    const F2 wl2 = splat2(wl), wr2 = splat2(wr);
    const F2 lo = add2_product(mul2(q00, wl2), mul2(q10, wr2), k);
    const F2 hi = add2_product(mul2(q01, wl2), mul2(q11, wr2), k);
    return add2_product(mul2(lo, splat2(wd)), mul2(hi, splat2(wu)), k);
}

// one generator step: lehmer_next up to its conditional subtraction
__device__ __forceinline__ uint32_t lehmer_fast(uint32_t s) {
    const u64 p = (u64)s * 279470273u + 279470273u;
    const uint32_t lo = (uint32_t)p, hi = (uint32_t)(p >> 32);
    const uint32_t h5 = hi * 5u;
    const uint32_t y = lo + h5;
    return y < lo ? y + 5u : y;
}

// Guards gathered over one step: the least sum of squares of a flow vector or
// square of a jittered component (NaN if one is), the least pattern of a
// component less 1 (a zero's wraps to the largest), the largest state.
struct FastGuard {
    float smallest;
    uint32_t component;
    uint32_t state;
};

__device__ __forceinline__ void guard_components(FastGuard& gd, F2 v) {
    float x, y;
    unpack2(v, x, y);
    gd.component = __viaddmin_u32(__float_as_uint(fminf(fabsf(x), fabsf(y))), 0xffffffffu, gd.component);
}

// The unit flow vector at a stage's point, jittered; s: the flow's sum of squares.
template <int FORM>
__device__ __forceinline__ F2 stage_fast(F2 a, F2 floor2, uint32_t off, uint32_t& rng, FastGuard& gd, float& s,
                                         const float2* __restrict__ uv, const FastGeo& f, const FastConst& k) {
    float xx, yy, sj;
    const F2 flow = taps_fast(a, floor2, off, uv, f, k);
    F2 u = unit_fast(flow, xx, yy, s);
    if (FORM != STEP_JITTERED) guard_components(gd, flow);
    if (FORM == STEP_PLAIN) return u;
    if (FORM == STEP_JITTERED || k.mag.x != 0.0f) {
        const uint32_t r0 = lehmer_fast(rng), r1 = lehmer_fast(r0);
        rng = r1;
        gd.state = max(gd.state, max(r0, r1));
        // r * 2^-32 - 1/2 in one rounding (the product is exact)
        const F2 r = fma2(pack2(__uint2float_rn(r0), __uint2float_rn(r1)), as_f2(k.draw), as_f2(k.draw0));
        u = add2_product(mul2(r, as_f2(k.mag)), u, k);
    }
    if (FORM == STEP_FAINT) guard_components(gd, u);
    u = unit_fast(u, xx, yy, sj);
    if (FORM == STEP_JITTERED) gd.smallest = min3_nan(gd.smallest, xx, yy);
    else gd.smallest = min3_nan(gd.smallest, sj, sj);
    return u;
}

// the pixel of an intermediate point, without clamps
__device__ __forceinline__ void locate_fast(F2 a, const FastGeo& f, const FastConst& k, F2& floor2, uint32_t& off) {
    const F2 t = add2_rz(add2(a, as_f2(k.pp5)), as_f2(k.magic));
    floor2 = sub2(t, as_f2(k.magic));
    off = min(offset_from_magic(t, f), f.off_last);  // in the grid even when a guard will fail
}

// Quantisation to 1 / TRAJECTORY_RESOLUTION (a power of two), |v| res < 127
__device__ __forceinline__ float quant_fast(float v, const FastConst& k) {
    const float t = __fmaf_rz(fabsf(v), k.res, FAST_MAGIC);
    return copysignf(__fmaf_rn(t, k.inv, k.minus_magic_inv), v);
}

struct FastStep {
    Vec2 d1, d2, next, u1;
    F2 t;          // 2^23 + pixel of next
    uint32_t off;  // byte offset of that pixel's vector; on a grid that fast_grid admits
    uint32_t idx;  // the pixel, on any grid (a byte offset wraps from pixel 2^29 on)
    uint32_t rng;
};

// rk_step for a lane whose guards failed
template <int ORDER, bool JITTER>
__device__ __noinline__ FastStep step_exact(Vec2 a, float dt, uint32_t rng, float cf, const float2* uv, uint32_t base,
                                            const slm_params& p, uint32_t nxp, uint32_t nyp) {
    const Geo g{nxp, nyp, cf, 0.0f, 0.0f, 0.0f};  // the step itself reads neither DT_MAX nor GRID_SCALE
    const Step st = rk_step<ORDER, JITTER>(a, dt, rng, uv + base, p, g);
    return FastStep{st.d1, st.d2, st.next, st.u1, pixel_magic_clamped(st.next, p.pad_width_pp5, nxp, nyp),
                    8u * (base + st.idx), base + st.idx, rng};
}

// One RK step from a0 (pixel t0 - 2^23, at byte offset off0 of the array uv)
// with time step dt; true if every guard held and the values are rk_step's.
// GATED: a lane outside the interior reads nothing (its grid may have none) and
// stays where it is; else it reads its clamped pixel's taps.
template <int ORDER, int FORM, bool GATED>
__device__ __forceinline__ bool step_fast(Vec2 a0, F2 t0, uint32_t off0, float dt, float cf, uint32_t rng,
                                          const float2* __restrict__ uv, const FastGeo& f, const FastConst& k,
                                          FastStep& o) {
    const F2 a = pack2(a0.x, a0.y);
    const F2 cf2 = splat2(cf), dt2 = splat2(dt);
    F2 fl = sub2(t0, as_f2(k.magic));
    float ix, iy;
    unpack2(sub2(fl, pack2(f.cx, f.cy)), ix, iy);
    const bool inside = (fabsf(ix) <= f.rx) & (fabsf(iy) <= f.ry);
    if (GATED && !inside) {
        o.d1 = o.d2 = o.u1 = Vec2{0.0f, 0.0f};
        o.next = a0;
        o.t = t0;
        o.off = off0;
        o.idx = off0 >> 3;
        o.rng = rng;
        return false;
    }
    uint32_t off = min(off0, f.off_last);
    FastGuard gd{FAST_S_MIN, 0xffffffffu, 0u};
    float s1, s2, s3, s4;  // sums of squares of the stages' flow vectors
    const F2 k1 = stage_fast<FORM>(a, fl, off, rng, gd, s1, uv, f, k);
    const F2 h1 = mul2(mul2(k1, cf2), dt2);
    float hx, hy, sx, sy;
    unpack2(h1, hx, hy);
    o.d1.x = quant_fast(hx, k);
    o.d1.y = quant_fast(hy, k);
    if (ORDER == 2) {
        const F2 d1 = pack2(o.d1.x, o.d1.y);
        const F2 b = add2(a, d1);
        locate_fast(b, f, k, fl, off);
        const F2 k2 = stage_fast<FORM>(b, fl, off, rng, gd, s2, uv, f, k);
        gd.smallest = min3_nan(gd.smallest, s1, s2);
        unpack2(mul2(as_f2(k.half), add2_product(mul2(mul2(k2, cf2), dt2), d1, k)), sx, sy);
    } else {
        const F2 b = fma2(as_f2(k.half), h1, a);
        locate_fast(b, f, k, fl, off);
        const F2 h2 = mul2(mul2(stage_fast<FORM>(b, fl, off, rng, gd, s2, uv, f, k), cf2), dt2);
        gd.smallest = min3_nan(gd.smallest, s1, s2);
        const F2 c = fma2(as_f2(k.half), h2, a);
        locate_fast(c, f, k, fl, off);
        const F2 h3 = mul2(mul2(stage_fast<FORM>(c, fl, off, rng, gd, s3, uv, f, k), cf2), dt2);
        const F2 d = add2_product(h3, a, k);
        locate_fast(d, f, k, fl, off);
        const F2 h4 = mul2(mul2(stage_fast<FORM>(d, fl, off, rng, gd, s4, uv, f, k), cf2), dt2);
        gd.smallest = min3_nan(gd.smallest, s3, s4);
        const F2 w = add2_product(h4, fma2(as_f2(k.two), h3, fma2(as_f2(k.two), h2, h1)), k);
        // div6 without its range test: below 2^-120 both quantise to 0
        unpack2(fma2(as_f2(k.div6_hi), w, mul2(as_f2(k.div6_lo), w)), sx, sy);
    }
    o.d2.x = quant_fast(sx, k);
    o.d2.y = quant_fast(sy, k);
    const F2 next = add2(a, pack2(o.d2.x, o.d2.y));
    o.t = add2_rz(add2(next, as_f2(k.pp5)), as_f2(k.magic));
    o.off = offset_from_magic(o.t, f);
    o.idx = o.off >> 3;
    o.rng = rng;
    unpack2(next, o.next.x, o.next.y);
    unpack2(k1, o.u1.x, o.u1.y);
    bool ok = (gd.smallest >= FAST_S_MIN) & inside;
    if (FORM != STEP_JITTERED) ok = ok & (gd.component >= FAST_C_BITS - 1u);
    if (FORM != STEP_PLAIN) ok = ok & (gd.state < LEHMER_M);
    else ok = ok & (fabsf(sx) < 1.0f) & (fabsf(sy) < 1.0f);  // an infinite sum of squares gives NaN here
    return ok;
}

// next_dt from the two quantised steps' difference (ex, ey), its two
// quotients by GRID_SCALE, the root and the last quotient formed as in
// unit_fast (gs_rcp: the IEEE reciprocal of GRID_SCALE; a quotient by it is
// exact by the same theorem).  A time step or an error too small for exact
// residuals takes the IEEE operations.
__device__ __forceinline__ float next_dt_fast(float ex, float ey, float dt, float dt_max, float gs, float gs_rcp,
                                              float adjusted_max_error) {
    const float x = quotient_from(ex, gs, gs_rcp), y = quotient_from(ey, gs, gs_rcp);
    const float s = __fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y));
    const float n = __fmul_rn(adjusted_max_error, dt);
    float cand;
    if (s >= 0x1p-100f && n >= FAST_S_MIN) {
        const float y0 = rsqrt_estimate(s);
        const float err = root_from(s, y0);
        cand = quotient_from(n, err, reciprocal_from(err, y0));
    } else {
        if (ex == 0.0f && ey == 0.0f) return dt_max;
        const float err = vlen(__fdiv_rn(ex, gs), __fdiv_rn(ey, gs));
        if (err == 0.0f) return dt_max;
        cand = __fdiv_rn(n, err);
    }
    return fminf(dt_max, cand);
}

// ------------------------------------------------------------------ plain walks
// The un-jittered step of the trajectory recorder and the mapping walks,
// which are bound by the latency of one step after another: by step_fast
// where the launch admits it, else by rk_step.  Uniform in a launch.
struct WalkGrid {
    FastGeo f;
    FastConst k;
    uint32_t fast;
};

static inline WalkGrid make_walk_grid(const slm_params& p) {
    WalkGrid w;
    w.f = make_fast_geo(p.nx_padded, p.ny_padded, p.grid_scale, p.dt_max, p.adjusted_max_error, 0u);
    w.k = make_fast_const(p);
    w.fast = fast_params(p) &&
             fast_grid(p.nx_padded, p.ny_padded, 0u, p.combo_factor, p.dt_max, p.trajectory_resolution);
    return w;
}

// Walks of a warp when n are spread evenly over the warps that the SMs hold of
// the walk kernels (28 each), `most` at most.  A launch of few walks takes as
// long as the longest of them, and a warp's steps take turns with its lanes'
// different branches.
static inline uint32_t walk_share(uint32_t n, uint32_t most = 32u) {
    const uint32_t warps = (uint32_t)num_sms() * 28u;
    const uint32_t share = n / warps + (n % warps ? 1u : 0u);
    return share < most ? share : most;
}

template <int ORDER>
__device__ __forceinline__ Step plain_step(Vec2 a, float dt, const float2* __restrict__ uv, const slm_params& p,
                                           const WalkGrid& w) {
    FastStep st;
    bool ok = false;
    if (w.fast) {
        const F2 t = pixel_magic_clamped(a, p.pad_width_pp5, p.nx_padded, p.ny_padded);
        ok = step_fast<ORDER, STEP_PLAIN, false>(a, t, offset_from_magic(t, w.f), dt, p.combo_factor, 0u, uv, w.f, w.k, st);
    }
    if (!ok) st = step_exact<ORDER, false>(a, dt, 0u, p.combo_factor, uv, 0u, p, p.nx_padded, p.ny_padded);
    return Step{st.d1, st.d2, st.u1, st.next, st.idx};
}

// |d| of a quantised step
__device__ __forceinline__ float step_length(Vec2 d, const WalkGrid& w) {
    return w.fast ? quantised_length(__fmaf_rn(d.y, d.y, d.x * d.x)) : vlen(d.x, d.y);
}

// the next time step after one of dt whose quantised steps differ by (ex, ey)
__device__ __forceinline__ float walk_dt(float ex, float ey, float dt, const slm_params& p, const WalkGrid& w) {
    if (w.fast) {
        if (dt * dt * w.f.kerr >= __fmaf_rn(ey, ey, ex * ex)) return p.dt_max;
        return next_dt_fast(ex, ey, dt, p.dt_max, p.grid_scale, w.f.gs_rcp, p.adjusted_max_error);
    }
    return next_dt(dt, vlen(__fdiv_rn(ex, p.grid_scale), __fdiv_rn(ey, p.grid_scale)), p);
}

}  // namespace slm
