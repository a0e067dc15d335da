// preprocess.cu -- the conditioned gradient vector field of a DTM region
// (python/streamlines/preprocess.py:531-621) in one tiled kernel.
//
// The reference runs it on the host: two scipy generic_filter passes with
// Python callbacks (find_blockages, :647-699), np.gradient, then numba loops
// over every cell (find_and_fix_loops, :302-349) and over the blockages
// (fix_blockages, :351-387), normalisation, edge padding and the NaN mask.
// Every value of a pixel depends only on the ROI within two pixels of it, so
// one kernel does it all.  A warp walks down a strip of PP_OUT columns, one
// lane a column (two halo columns on either side), with the last rows of the
// ROI, the velocities and the blockage codes in registers and the neighbours'
// by shuffles; looped cells of a row are the bits of a ballot.  Each pixel's
// final uv (with its edge-padding replicas), slope, masks and codes are
// written as the row is reached.
//
// Arithmetic follows the reference operation for operation (IEEE float32,
// --fmad=false):
//   gradient   np.gradient of the float32 ROI, one-sided at the edges, then
//              / pixel_size in float32;
//   hypot      float32 np.hypot: the double sum of the exact squares,
//              square-rooted in double and rounded once to float32;
//   loops      check_has_loop as numba compiles it: velocity sums in float32,
//              its speed in double rounded to float32, divergence and curl in
//              float32 (2-term dot products round once), compared with the
//              double thresholds (a float32 against a float64 parameter);
//   fixes      break_out_of_loop: component / hypotf of the int8 vector;
//              fix_blockages: (dx, dy) / sqrt(2) in double, stored as float32.
//
// The kernel is bound by instruction issue, not by its 29 bytes a pixel.  Two
// thirds of the instructions were the double square roots of the hypots, the
// IEEE divisions, and the index arithmetic and shared-memory loads of a tiled
// form (16 x 32 tiles with halos; 47 loads and 200 integer operations a pixel).
// The hypots and quotients are formed in float32 now (unit_of_fast), with a
// guard that leaves what it cannot decide to the double path; a cell's speed is
// only compared with its threshold, which its square decides but next to it;
// the thresholds are rounded to float32 on the host the way that keeps the
// comparison; and the rows in registers need neither tiles nor indices.
//
// Measured (B200, every output, float32): 4096 x 3001 416 -> 241 us, 2000 x 2001
// 143 -> 96 us, 300 x 311 14.6 -> 13.4 us; 725 -> 438 thread instructions a pixel
// (7 blocks an SM; 5, 6 and 8 measured 12 %, 2 % and 0 % slower).
#include "capi_util.cuh"
#include "unit_math.cuh"
#include <algorithm>
#include <cmath>
#include <limits>

namespace slm {

constexpr int PP_OUT = 28;    // columns a warp writes (lanes 2 .. 29)
constexpr int PP_WARPS = 4;   // warps (adjacent strips) a block

// flow-vector bits (get_flow_vector, preprocess.py:195-226)
enum : uint32_t { FV_W = 1, FV_E = 2, FV_S = 4, FV_N = 8, FV_SW = 16, FV_SE = 32, FV_NW = 64, FV_NE = 128 };

__device__ __forceinline__ int clampi(int i, int n) { return i < 0 ? 0 : (i >= n ? n - 1 : i); }

__device__ __forceinline__ float hypot_f32(float a, float b) {
    if (isinf(a) || isinf(b)) return __int_as_float(0x7f800000);
    const double s = __dadd_rn(__dmul_rn((double)a, (double)a), __dmul_rn((double)b, (double)b));
    return __double2float_rn(__dsqrt_rn(s));
}

// set_speed_field (preprocess.py:118-136)
__device__ __forceinline__ float speed_of(float u, float v) {
    const float s = hypot_f32(u, v);
    return (!isfinite(s) || s == 0.0f) ? 1.0f : s;
}

// speed_of(u, v) and u, v divided by it.
//
// The sum of squares is held as a float and its remainder (the squares' fused
// residuals and the sum's), 2^-46 of it in all; the root's correction r + t is
// then within 2^-43.4 of the square root of the double sum, whose own
// rounding is 2^-53.  Both ends of r + t -+ 2^-42 r rounding to one float
// decide it (rounding the root to double first cannot change that: it moves
// the root less); otherwise, one time in 2^17, and outside the range where
// every residual is exact, the double path runs.  The quotients are
// unit_math.cuh's.  True if the fast path held.
__device__ __forceinline__ bool unit_of_fast(float& u, float& v, float& speed) {
    const float p = __fmul_rn(u, u), q = __fmul_rn(v, v);
    const float pe = __fmaf_rn(u, u, -p), qe = __fmaf_rn(v, v, -q);
    const float big = fmaxf(p, q), small = fminf(p, q);
    const float sh = __fadd_rn(big, small);
    const float sl = __fadd_rn(__fadd_rn(__fsub_rn(big, sh), small), __fadd_rn(pe, qe));
    const float y0 = rsqrt_estimate(sh), r = __fmul_rn(sh, y0);
    const float t = __fmul_rn(__fadd_rn(__fmaf_rn(-r, r, sh), sl), half_of(y0));
    const float margin = __fmul_rn(r, 0x1p-42f);
    const float len = __fadd_rn(r, __fsub_rn(t, margin));
    // a component's square is 0 or at least 2^-120, so it is 0 or at least 2^-60
    const bool ok = len == __fadd_rn(r, __fadd_rn(t, margin)) && sh >= 0x1p-60f && sh <= 0x1p100f &&
                    (p >= 0x1p-120f || u == 0.0f) && (q >= 0x1p-120f || v == 0.0f);
    const float y = reciprocal_from(len, y0);
    const float a = quotient_from(u, len, y), b = quotient_from(v, len, y);
    if (ok) {
        u = a;
        v = b;
        speed = len;
    }
    return ok;
}

// the same by the definition
__device__ __noinline__ float3 unit_of_exact(float u, float v) {
    const float s = speed_of(u, v);
    return make_float3(__fdiv_rn(u, s), __fdiv_rn(v, s), s);
}

// get_flow_vector's priority: SW, SE, NW, NE, W, E, S, N
__device__ __forceinline__ void flow_vector(uint32_t nn, int& dx, int& dy) {
    dx = 0; dy = 0;
    if (nn & FV_SW) { dx = -1; dy = -1; }
    else if (nn & FV_SE) { dx = +1; dy = -1; }
    else if (nn & FV_NW) { dx = -1; dy = +1; }
    else if (nn & FV_NE) { dx = +1; dy = +1; }
    else if (nn & FV_W) { dx = -1; }
    else if (nn & FV_E) { dx = +1; }
    else if (nn & FV_S) { dy = -1; }
    else if (nn & FV_N) { dy = +1; }
}

struct PreOut {
    float2* uv;            // [nxp][nyp]
    float* slope;          // [nxp][nyp] or null
    uint8_t* uv_mask;      // [nxp][nyp] or null
    uint8_t* mask;         // [nxp][nyp] or null: pad frame | NaN ROI | NaN uv
    uint8_t* blockages;    // [nx][ny] or null
    uint8_t* blocked;      // [nx][ny] or null
    uint8_t* loop_cells;   // [nx][ny] or null
    float* gradx;          // [nx][ny] or null
    float* grady;          // [nx][ny] or null
    uint32_t* n_cells;     // 1 word or null
};

// One row of a 3-column neighbourhood: y - 1, y, y + 1.
template <typename T>
struct Row3 {
    T l, c, r;
};

template <typename T>
__device__ __forceinline__ Row3<T> spread(T c) {
    return Row3<T>{__shfl_up_sync(0xffffffffu, c, 1), c, __shfl_down_sync(0xffffffffu, c, 1)};
}

// get_flow_vector of a pixel with its neighbours (rows a, b, c = x - 1, x, x + 1):
// the lower diagonal neighbours, 0 if one of the other four is lower
template <typename T>
__device__ __forceinline__ uint32_t blockage_code(const Row3<T>& a, const Row3<T>& b, const Row3<T>& c) {
    const T h = b.c;
    uint32_t nn = 0;
    if (a.l < h) nn |= FV_SW;
    if (c.l < h) nn |= FV_SE;
    if (a.r < h) nn |= FV_NW;
    if (c.r < h) nn |= FV_NE;
    return (b.l < h || a.c < h || c.c < h || b.r < h) ? 0u : nn;
}

// The codes of a row, kept where they name one neighbour alone (what the blocked
// neighbours are found from).  Columns off the grid take the edge's code
// (the second generic_filter's 'reflect').
__device__ __forceinline__ Row3<uint32_t> single_codes(uint32_t code, int y, int ny) {
    Row3<uint32_t> e = spread((code & (code - 1u)) == 0u ? code : 0u);
    if (y == 0) e.l = e.c;
    if (y == ny - 1) e.r = e.c;
    return e;
}

// velocities of a row: unit vector and, for the slope, the raw speed
struct Vel {
    float u, v, raw;
};

// ALL: every output is wanted (the stage's call), so none is tested for.
template <typename T, bool ALL>
__global__ void __launch_bounds__(PP_WARPS * 32, 7)
k_preprocess(const T* __restrict__ roi, int nx, int ny, int rows, float pixel_size, float pixel_rcp, int pad,
             double vecsum_threshold, float vecsum2_lo, float vecsum2_hi, float divergence_threshold,
             float curl_threshold, int normalize, PreOut out) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int y0 = (blockIdx.x * PP_WARPS + (threadIdx.x >> 5)) * PP_OUT;
    if (y0 >= ny) return;  // (whole warps)
    const int y = y0 - 2 + lane;
    const bool own = lane >= 2 && lane < 2 + PP_OUT && y < ny;
    const int x0 = blockIdx.y * rows, x1 = min(nx, x0 + rows);
    const T* column = roi + clampi(y, ny);
    // a row of the ROI, clamped (scipy's 'reflect' of a 3-wide window repeats
    // the edge pixel; the gradient and the loop fixes read no halo outside the
    // grid)
    auto load = [&](int x) { return __ldg(column + (size_t)clampi(x, nx) * ny); };
    // gradient and velocity of pixel (x, y), rows a, b, c around it
    auto velocity = [&](int x, const Row3<T>& a, const Row3<T>& b, const Row3<T>& c, float& gu, float& gv) {
        const float h = (float)b.c, up = (float)c.c, down = (float)a.c, left = (float)b.l, right = (float)b.r;
        // np.gradient, edge_order 1 (shapes below 2 are refused on the host)
        float gx = (up - down) * 0.5f, gy = (right - left) * 0.5f;
        if (x == 0) gx = up - h;
        if (x == nx - 1) gx = h - down;
        if (y == 0) gy = right - h;
        if (y == ny - 1) gy = h - left;
        // pixel_rcp (NaN: the pixel size is out of the range this needs) gives
        // the IEEE quotients of what unit_of_fast accepts; one that fell to 0 is
        // out of range
        gu = quotient_from(gx, pixel_size, pixel_rcp);
        gv = quotient_from(gy, pixel_size, pixel_rcp);
        Vel w{-gu, -gv, 1.0f};
        const bool whole = (gu != 0.0f || gx == 0.0f) && (gv != 0.0f || gy == 0.0f);
        if (!whole || !unit_of_fast(w.u, w.v, w.raw)) {
            // No gradient at all: w is what the definition gives (speed_of).
            // Level ground is common, in rounded heights above all: with its
            // double path 2000 x 2001 level pixels took 219 us, where relief
            // takes 144; they take 128 now.
            if (!whole || gu != 0.0f || gv != 0.0f) {
                gu = __fdiv_rn(gx, pixel_size);
                gv = __fdiv_rn(gy, pixel_size);
                const float3 e = unit_of_exact(-gu, -gv);
                w = Vel{e.x, e.y, e.z};
            }
        }
        return w;
    };
    // check_has_loop of the cells (x, y) .. (x + 1, y + 1) from the unit
    // velocities of rows x (p) and x + 1 (q): the lanes' answers as bits
    auto loops = [&](int x, const Vel& p, const Vel& q) -> unsigned {
        const float u01 = __shfl_down_sync(FULL, p.u, 1), v01 = __shfl_down_sync(FULL, p.v, 1);
        const float u11 = __shfl_down_sync(FULL, q.u, 1), v11 = __shfl_down_sync(FULL, q.v, 1);
        const float vx = (((p.u + q.u) + u11) + u01) * 0.25f;
        const float vy = (((p.v + q.v) + v11) + v01) * 0.25f;
        const float div = (((-p.u - p.v) + (q.u - q.v)) + (u11 + v11)) + (-u01 + v01);
        const float curl = (((p.u - p.v) + (q.u + q.v)) + (-u11 + v11)) + (-u01 - v01);
        bool hit = x >= 0 && x <= nx - 2 && y >= 0 && y <= ny - 2 && div <= divergence_threshold &&
                   fabsf(curl) >= curl_threshold;
        // the speed (numba: double dot product and sqrt, rounded to float32)
        // below its threshold, decided by its square but within 2^-18 of it
        const float s2 = vx * vx + vy * vy;
        bool slow = s2 < vecsum2_lo;
        if (hit && !slow && !(s2 > vecsum2_hi)) slow = (double)hypot_f32(vx, vy) < vecsum_threshold;
        return __ballot_sync(FULL, hit && slow);
    };

    // rows x0 - 1 and x0 of the velocities, codes and cells
    Row3<T> ha = spread(load(x0 - 2)), hb = spread(load(x0 - 1)), hc = spread(load(x0));
    float gu = 0.0f, gv = 0.0f;
    Vel vb{0.0f, 0.0f, 1.0f};
    if (x0 > 0) vb = velocity(x0 - 1, ha, hb, hc, gu, gv);
    Row3<uint32_t> ea = single_codes(blockage_code(ha, hb, hc), y, ny);
    ha = hb;
    hb = hc;
    hc = spread(load(x0 + 1));
    Vel vc = velocity(x0, ha, hb, hc, gu, gv);
    uint32_t code = blockage_code(ha, hb, hc);
    Row3<uint32_t> eb = single_codes(code, y, ny);
    if (x0 == 0) ea = eb;  // the row above the grid takes the edge's codes
    unsigned cells_above = loops(x0 - 1, vb, vc);
    vb = vc;

    const float inv_sqrt2 = __double2float_rn(__ddiv_rn(1.0, __dsqrt_rn(2.0)));
    const float diagonal = __fdiv_rn(1.0f, hypot_f32(1.0f, 1.0f));
    const int nyp = ny + 2 * pad;
    uint32_t n_cells = 0;
    // rows ha, hb, hc of the ROI, vb and eb are at x - 1, x, x + 1, x and x
    for (int x = x0; x < x1; ++x) {
        const size_t gi = (size_t)x * ny + y;
        if (own) {
            if (ALL || out.gradx) out.gradx[gi] = gu;
            if (ALL || out.grady) out.grady[gi] = gv;
        }
        const Row3<T> hd = spread(load(x + 2));
        uint32_t code_below = code;
        Row3<uint32_t> ec = eb;  // (the row below the grid takes the edge's codes)
        vc = Vel{0.0f, 0.0f, 1.0f};
        if (x + 1 < nx) {
            vc = velocity(x + 1, hb, hc, hd, gu, gv);
            code_below = blockage_code(hb, hc, hd);
            ec = single_codes(code_below, y, ny);
        }
        const unsigned cells = loops(x, vb, vc);
        const bool cell = (cells >> lane) & 1u;
        float u = vb.u, v = vb.v;
        // break_out_of_loop for a pixel marked by any of its four cells
        const unsigned near = cells | cells_above;
        const bool marked = ((near | (near << 1)) >> lane) & 1u;
        if (marked && x >= 1 && x <= nx - 2 && y >= 1 && y <= ny - 2) {
            // break_out_of_loop's vectors: W, E, S, N, SW, SE, NW, NE
            // (dx + 1 in bits 0-1, dy + 1 in bits 2-3)
            T h_min = (T)3.402823466e38f;
            uint32_t to = 0u | (1u << 2);
            auto lower = [&](T h, uint32_t dx1, uint32_t dy1) {
                if (h_min > h) { h_min = h; to = dx1 | (dy1 << 2); }
            };
            lower(ha.c, 0u, 1u);
            lower(hc.c, 2u, 1u);
            lower(hb.l, 1u, 0u);
            lower(hb.r, 1u, 2u);
            lower(ha.l, 0u, 0u);
            lower(hc.l, 2u, 0u);
            lower(ha.r, 0u, 2u);
            lower(hc.r, 2u, 2u);
            const float step = (to & 5u) ? 1.0f : diagonal;  // one of dx, dy is 0
            u = (float)((int)(to & 3u) - 1) * step;
            v = (float)((int)(to >> 2) - 1) * step;
        }
        // fix_blockages: blockages, then blocked neighbours
        uint32_t c1 = (ea.l & FV_SW) | (ec.l & FV_SE) | (ea.r & FV_NW) | (ec.r & FV_NE);
        if (eb.l & (FV_SW | FV_SE)) c1 |= FV_S;
        if (ea.c & (FV_SW | FV_NW)) c1 |= FV_W;
        if (ec.c & (FV_NE | FV_SE)) c1 |= FV_E;
        if (eb.r & (FV_NW | FV_NE)) c1 |= FV_N;
        if (code | c1) {
            int dx, dy;
            flow_vector(c1 ? c1 : code, dx, dy);
            u = dx ? (float)dx * inv_sqrt2 : 0.0f;
            v = dy ? (float)dy * inv_sqrt2 : 0.0f;
        }
        const float raw = vb.raw;  // speed of the unfixed gradient
        if (normalize) {
            float sp;
            if (!unit_of_fast(u, v, sp) && (u != 0.0f || v != 0.0f)) {
                const float3 e = unit_of_exact(u, v);
                u = e.x;
                v = e.y;
            }
        } else {
            u = u * raw;
            v = v * raw;
        }
        const bool bad = isnan(u) || isnan(v);
        if (bad) { u = 0.0f; v = 0.0f; }
        if (own) {
            const float slope = atanf(raw) * (180.0f / 3.14159265358979323846f);
            const uint8_t bad8 = bad ? 1 : 0, gone8 = (bad || isnan((float)hb.c)) ? 1 : 0;
            n_cells += cell;
            if (ALL || out.loop_cells) out.loop_cells[gi] = cell;
            if (ALL || out.blockages) out.blockages[gi] = (uint8_t)code;
            if (ALL || out.blocked) out.blocked[gi] = (uint8_t)c1;
            const size_t pi = (size_t)(x + pad) * nyp + (y + pad);
            out.uv[pi] = make_float2(u, v);
            if (ALL || out.slope) out.slope[pi] = slope;
            if (ALL || out.uv_mask) out.uv_mask[pi] = bad8;
            if (ALL || out.mask) out.mask[pi] = gone8;
            if (pad && (x == 0 || x == nx - 1 || y == 0 || y == ny - 1)) {
                // the edge-padding replicas of an edge pixel
                const int xa = (x == 0) ? 0 : x + pad, xb = (x == nx - 1) ? nx + 2 * pad - 1 : x + pad;
                const int ya = (y == 0) ? 0 : y + pad, yb = (y == ny - 1) ? nyp - 1 : y + pad;
                for (int qx = xa; qx <= xb; ++qx) {
                    for (int qy = ya; qy <= yb; ++qy) {
                        const size_t qi = (size_t)qx * nyp + qy;
                        if (qi == pi) continue;
                        out.uv[qi] = make_float2(u, v);
                        if (ALL || out.slope) out.slope[qi] = slope;
                        if (ALL || out.uv_mask) out.uv_mask[qi] = bad8;
                        if (ALL || out.mask) out.mask[qi] = 1;  // the pad frame
                    }
                }
            }
        }
        ha = hb;
        hb = hc;
        hc = hd;
        vb = vc;
        ea = eb;
        eb = ec;
        code = code_below;
        cells_above = cells;
    }
    if (ALL || out.n_cells) {
        n_cells = __reduce_add_sync(FULL, n_cells);
        if (lane == 0 && n_cells) atomicAdd(out.n_cells, n_cells);
    }
}

}  // namespace slm

using namespace slm;

// the largest float at or below v (NaN for NaN): f <= v and f <= float_at_most(v)
// are the same for every float f
static float float_at_most(double v) {
    const float f = (float)v;
    return (double)f > v ? std::nextafterf(f, -std::numeric_limits<float>::infinity()) : f;
}

extern "C" {

int slm_preprocess(const void* roi, int roi_dtype, uint32_t nx, uint32_t ny, const slm_preprocess_params* prm,
                   float* uv, float* slope, uint8_t* uv_mask, uint8_t* mask, uint8_t* blockages,
                   uint8_t* blocked_neighbors, uint8_t* loop_cells, float* gradx, float* grady,
                   uint32_t* n_loop_cells, void* stream) {
    clear_error();
    SLM_REQUIRE(roi && uv && prm, "NULL roi, uv or params");
    SLM_REQUIRE(roi_dtype == SLM_F32 || roi_dtype == SLM_F64, "roi_dtype must be SLM_F32 or SLM_F64");
    SLM_REQUIRE(nx >= 2 && ny >= 2, "the gradient needs at least 2 pixels along each axis (got %u x %u)", nx, ny);
    SLM_REQUIRE(prm->pad_width < 65536, "pad_width too large");
    const uint64_t nxp = (uint64_t)nx + 2ull * prm->pad_width, nyp = (uint64_t)ny + 2ull * prm->pad_width;
    SLM_REQUIRE(nxp < (1ull << 31) && nyp < (1ull << 31) && nxp * nyp < (1ull << 40), "grid too large");
    SLM_REQUIRE(aligned(uv, 8), "uv must be 8-byte aligned");
    SLM_REQUIRE(aligned(roi, roi_dtype == SLM_F64 ? 8 : 4), "roi misaligned");
    cudaStream_t s = (cudaStream_t)stream;
    PreOut o{(float2*)uv, slope, uv_mask, mask, blockages, blocked_neighbors, loop_cells, gradx, grady,
             n_loop_cells};
    if (n_loop_cells) SLM_CUDA(cudaMemsetAsync(n_loop_cells, 0, sizeof(uint32_t), s));
    // row ranges: 8 warps for each scheduler where the grid allows, 2 to 64
    // rows each (a range forms one row of velocities and codes twice, which
    // costs nothing where warps are missing)
    const uint32_t strips = (ny + PP_OUT - 1) / PP_OUT;
    const uint64_t want = (uint64_t)num_sms() * 4u * 8u;
    uint32_t rows = (uint32_t)std::min<uint64_t>(64u, std::max<uint64_t>(2u, (uint64_t)nx * strips / want));
    rows = std::max(rows, (nx + 65534u) / 65535u);
    const dim3 grid((strips + PP_WARPS - 1) / PP_WARPS, (nx + rows - 1) / rows);
    SLM_REQUIRE(grid.y < 65536, "nx too large for the row ranges");
    const float ps = (float)prm->pixel_size;
    // quotients by the pixel size through its reciprocal need both well inside
    // the float range; NaN otherwise, which no guard accepts
    const float rcp = (ps >= 0x1p-30f && ps <= 0x1p30f) ? 1.0f / ps : std::numeric_limits<float>::quiet_NaN();
    // the squared threshold with a margin of 2^-18 either way; one far out of
    // the range of speeds, at or below 0, or NaN, never decides by the square
    const double thr = prm->vecsum_threshold;
    const bool square = thr >= 0x1p-40 && thr <= 0x1p40;
    const float lo = square ? (float)(thr * thr * (1.0 - 0x1p-18)) : 0.0f;
    const float hi = square ? (float)(thr * thr * (1.0 + 0x1p-18)) : std::numeric_limits<float>::infinity();
    // a float32 against a double threshold: against the nearest float32 on the
    // side that keeps the answer
    const float div_thr = float_at_most(prm->divergence_threshold), curl_thr = -float_at_most(-prm->curl_threshold);
    const bool all = slope && uv_mask && mask && blockages && blocked_neighbors && loop_cells && gradx && grady &&
                     n_loop_cells;
#define SLM_PREPROCESS(T, ALL)                                                                                   \
    k_preprocess<T, ALL><<<grid, PP_WARPS * 32, 0, s>>>((const T*)roi, (int)nx, (int)ny, (int)rows, ps, rcp,          \
                                                   (int)prm->pad_width, thr, lo, hi, div_thr, curl_thr,          \
                                                   prm->do_normalize_speed ? 1 : 0, o)
    if (roi_dtype == SLM_F64) {
        if (all) SLM_PREPROCESS(double, true);
        else SLM_PREPROCESS(double, false);
    } else {
        if (all) SLM_PREPROCESS(float, true);
        else SLM_PREPROCESS(float, false);
    }
#undef SLM_PREPROCESS
    SLM_LAUNCHED("k_preprocess");
    return SLM_OK;
}

}  // extern "C"
