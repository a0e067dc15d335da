// scheduler.cu -- learned trajectory-length scheduler: a small BF16 CNN that
// reads a 16x16x2 patch of the flow field around a seed pixel and predicts
// log(1 + RK steps) of the seed's downstream and upstream trajectories, its
// training kernels, and the counting sort that turns predictions into the
// order the field tracer issues seeds in.  Ordering never changes a result:
// the tracer's per-pixel sums are integer and every trajectory's RNG stream
// follows its seed index.
//
// Network (all operands rounded to bfloat16, fp32 accumulation):
//   conv1  4x4 stride 4, 2 -> 32 channels, ReLU   (16 tiles x 32 features)
//   conv2  2x2 stride 2, 32 -> 64 channels, ReLU  (4 positions x 128 features)
//   dense  256 -> 2
// Feature orders: X1[t][f], t = 4*ti + tj, f = 2*(4*di + dj) + c, pixel
// (cx-8+4ti+di, cy-8+4tj+dj) clamped to the padded grid; X2[u][g], u = 2*ui+uj,
// g = 32*(2*ei+ej) + o reads A1[4*(2ui+ei) + (2uj+ej)][o]; X3[h] = A2[h/64][h%64].
//
// Training runs as batched GEMMs on the tensor cores (slm_gemm, gemm_tc.cu:
// tcgen05 with bf16 operands and fp32 accumulators in tensor memory, split-K
// for the weight gradients); inference is one fused kernel per warp of 16
// seeds (mma.sync m16n8k16 bf16 -> fp32).
#include <algorithm>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include "capi_util.cuh"

namespace slm {

constexpr int CNN_F1 = 32, CNN_C1 = 32, CNN_T1 = 16;
constexpr int CNN_F2 = 128, CNN_C2 = 64, CNN_U2 = 4;
constexpr int CNN_F3 = 256, CNN_OUT = 2;

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// ------------------------------------------------------------------ gather
// X1 rows for sample s: X1[(s*16 + t)*32 + f]
__global__ void k_patch_gather(const float2* __restrict__ uv, uint32_t nxp, uint32_t nyp, uint32_t pad,
                               const float2* __restrict__ seeds, const uint32_t* __restrict__ index,
                               uint32_t n, float* __restrict__ x1) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;  // one thread per (sample, tile, cell)
    if (tid >= n * 256u) return;
    const uint32_t s = tid >> 8, t = (tid >> 4) & 15u, m = tid & 15u;
    const uint32_t seed = index ? index[s] : s;
    const float2 sp = seeds[seed];
    const int cx = (int)sp.x + (int)pad, cy = (int)sp.y + (int)pad;
    const int ti = t >> 2, tj = t & 3, di = m >> 2, dj = m & 3;
    int x = cx - 8 + 4 * ti + di, y = cy - 8 + 4 * tj + dj;
    x = x < 0 ? 0 : (x >= (int)nxp ? (int)nxp - 1 : x);
    y = y < 0 ? 0 : (y >= (int)nyp ? (int)nyp - 1 : y);
    const float2 v = uv[(size_t)x * nyp + y];
    float* row = x1 + ((size_t)s * 16 + t) * 32 + 2 * m;
    row[0] = bf16r(v.x);
    row[1] = bf16r(v.y);
}

// A1 [n*16][32] -> X2 [n*4][128]
__global__ void k_a1_to_x2(const float* __restrict__ a1, uint32_t n, float* __restrict__ x2) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= n * 512u) return;
    const uint32_t s = tid >> 9, u = (tid >> 7) & 3u, g = tid & 127u;
    const uint32_t e = g >> 5, o = g & 31u;
    const uint32_t ui = u >> 1, uj = u & 1u, ei = e >> 1, ej = e & 1u;
    const uint32_t t = 4u * (2u * ui + ei) + (2u * uj + ej);
    x2[tid] = a1[((size_t)s * 16 + t) * 32 + o];
}

// dX2 [n*4][128] -> dA1 [n*16][32] (each A1 element feeds exactly one X2 element)
__global__ void k_dx2_to_da1(const float* __restrict__ dx2, uint32_t n, float* __restrict__ da1) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= n * 512u) return;
    const uint32_t s = tid >> 9, u = (tid >> 7) & 3u, g = tid & 127u;
    const uint32_t e = g >> 5, o = g & 31u;
    const uint32_t ui = u >> 1, uj = u & 1u, ei = e >> 1, ej = e & 1u;
    const uint32_t t = 4u * (2u * ui + ei) + (2u * uj + ej);
    da1[((size_t)s * 16 + t) * 32 + o] = dx2[tid];
}

// dZ = dA * (Z > 0)
__global__ void k_relu_backward(const float* __restrict__ da, const float* __restrict__ z, size_t n,
                                float* __restrict__ dz) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dz[i] = z[i] > 0.0f ? da[i] : 0.0f;
}

// Column sums of dZ [rows][cols] added into db[cols].  A block, or a cluster of
// CTAS of them, takes `width` columns, one a lane, so a warp reads 32 / width rows
// at once, each warp every (CTAS * 32)th of such groups of rows; the warps' sums
// are added in order by the first block, which reads the others' shared memory,
// so the result does not depend on the order they run in.
constexpr uint32_t BIAS_CTAS = 8, BIAS_THREADS = 1024;

template <uint32_t CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(BIAS_THREADS)
k_bias_grad(const float* __restrict__ dz, size_t rows, int cols, uint32_t width, float* __restrict__ db) {
    __shared__ float part[BIAS_THREADS / 32][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t rank = blockIdx.x % CTAS;
    const int c = (int)((blockIdx.x / CTAS) * width + lane % width);
    const uint32_t per_warp = 32u / width;  // rows a warp reads at once
    const size_t step = (size_t)CTAS * (BIAS_THREADS / 32) * per_warp;
    float s = 0.0f;
    if (c < cols) {
        size_t r = ((size_t)rank * (BIAS_THREADS / 32) + warp) * per_warp + lane / width;
        float v[16];  // sixteen loads in flight
        for (; r + 15 * step < rows; r += 16 * step) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __ldg(dz + (r + j * step) * cols + c);
#pragma unroll
            for (int j = 0; j < 16; ++j) s += v[j];
        }
        if (r < rows) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = r + j * step < rows ? __ldg(dz + (r + j * step) * cols + c) : 0.0f;
#pragma unroll
            for (int j = 0; j < 16; ++j) s += v[j];
        }
    }
    for (uint32_t o = width; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    part[warp][lane] = s;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    if (CTAS > 1) cluster.sync();
    else __syncthreads();
    if (rank == 0 && warp == 0 && lane < width && c < cols) {
        float t = 0.0f;
        for (uint32_t b = 0; b < CTAS; ++b) {
            const float* p = CTAS > 1 ? cluster.map_shared_rank(&part[0][0], b) : &part[0][0];
            for (uint32_t w = 0; w < BIAS_THREADS / 32; ++w) t += p[w * 32 + lane];
        }
        atomicAdd(db + c, t);  // (gradients of several streams may add into one db)
    }
    if (CTAS > 1) cluster.sync();  // the other blocks' shared memory stays until it is read
}

// dY = 2 W (Y - T) inv_n, loss += sum W (Y - T)^2 inv_n (W = 1 without weights)
__global__ void k_mse(const float* __restrict__ y, const float* __restrict__ t, const float* __restrict__ w,
                      size_t n_el, float inv_n, float* __restrict__ dy, float* __restrict__ loss) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.0f;
    if (i < n_el) {
        const float d = y[i] - t[i];
        const float wi = (w ? w[i] : 1.0f) * inv_n;
        dy[i] = 2.0f * d * wi;
        l = d * d * wi;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, l);
}

// Adam on fp32 master weights; also writes the bf16-rounded working copy.
__global__ void k_adam(float* __restrict__ w, float* __restrict__ wq, const float* __restrict__ g,
                       float* __restrict__ m, float* __restrict__ v, size_t n, float lr, float b1,
                       float b2, float eps, float c1, float c2, int round_w) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    wq[i] = round_w ? bf16r(wi) : wi;
}

// ------------------------------------------------------------------ inference
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
                 "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// a seed whose pixel is not in the padded grid
__device__ __forceinline__ bool off_grid(float2 sp, uint32_t nxp, uint32_t nyp, uint32_t pad) {
    const int cx = (int)sp.x + (int)pad, cy = (int)sp.y + (int)pad;
    return cx < 0 || cx >= (int)nxp || cy < 0 || cy >= (int)nyp;
}

// Shared-memory layout of the inference kernel (bf16 pairs as uint32):
//   W1t [32 n][16 kpairs], W2t [64 n][64 kpairs], W3t [8 n][128 kpairs] (n-major,
//   so a B fragment (k pair, n) is one 32-bit word); biases fp32; per warp an
//   A1 stage [4 seeds][16 t][16 pairs] and an A2/X3 stage [16 seeds][128 pairs].
constexpr int INF_WARPS = 4;
struct InferSmem {
    uint32_t w1[32][16 + 1];
    uint32_t w2[64][64 + 1];
    uint32_t w3[8][128 + 1];
    float b1[32], b2[64], b3[8];
    uint32_t a1[INF_WARPS][4][16][16 + 1];
    uint32_t x3[INF_WARPS][16][128 + 1];
};

__global__ void __launch_bounds__(INF_WARPS * 32)
k_cnn_infer(const float2* __restrict__ uv, uint32_t nxp, uint32_t nyp, uint32_t pad,
            const float2* __restrict__ seeds, const uint32_t* __restrict__ index, uint32_t n,
            const float* __restrict__ w1,
            const float* __restrict__ b1, const float* __restrict__ w2, const float* __restrict__ b2,
            const float* __restrict__ w3, const float* __restrict__ b3, float* __restrict__ out,
            const uint32_t* __restrict__ outside) {
    // outside (NULL: every seed): only the seeds off the grid, if it counted any
    if (outside && *outside == 0u) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    InferSmem& S = *reinterpret_cast<InferSmem*>(smem_raw);
    for (int i = threadIdx.x; i < 32 * 16; i += blockDim.x) {
        const int nn = i / 16, kp = i % 16;
        S.w1[nn][kp] = pack_bf16(w1[(2 * kp) * CNN_C1 + nn], w1[(2 * kp + 1) * CNN_C1 + nn]);
    }
    for (int i = threadIdx.x; i < 64 * 64; i += blockDim.x) {
        const int nn = i / 64, kp = i % 64;
        S.w2[nn][kp] = pack_bf16(w2[(2 * kp) * CNN_C2 + nn], w2[(2 * kp + 1) * CNN_C2 + nn]);
    }
    for (int i = threadIdx.x; i < 8 * 128; i += blockDim.x) {
        const int nn = i / 128, kp = i % 128;
        S.w3[nn][kp] = nn < CNN_OUT ? pack_bf16(w3[(2 * kp) * CNN_OUT + nn], w3[(2 * kp + 1) * CNN_OUT + nn]) : 0u;
    }
    for (int i = threadIdx.x; i < 32; i += blockDim.x) S.b1[i] = b1[i];
    for (int i = threadIdx.x; i < 64; i += blockDim.x) S.b2[i] = b2[i];
    for (int i = threadIdx.x; i < 8; i += blockDim.x) S.b3[i] = i < CNN_OUT ? b3[i] : 0.0f;
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tig = lane & 3;
    const uint32_t groups = (n + 15) / 16;
    for (uint32_t grp = blockIdx.x * INF_WARPS + warp; grp < groups; grp += gridDim.x * INF_WARPS) {
        if (outside) {
            const uint32_t s = grp * 16 + (lane & 15);
            const float2 sp = seeds[index ? __ldg(index + min(s, n - 1)) : min(s, n - 1)];
            if (!__any_sync(0xffffffffu, off_grid(sp, nxp, nyp, pad))) continue;
        }
        // 16 seeds per warp pass; conv1 + conv2 in 4 quarters of 4 seeds
        for (int q = 0; q < 4; ++q) {
            for (int sl = 0; sl < 4; ++sl) {
                const uint32_t s = grp * 16 + q * 4 + sl;
                const uint32_t sc = s < n ? s : n - 1;
                const float2 sp = seeds[index ? __ldg(index + sc) : sc];
                const int cx = (int)sp.x + (int)pad, cy = (int)sp.y + (int)pad;
                // conv1: M = 16 tiles, K = 32, N = 32
                float c[4][4] = {};
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    uint32_t a[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int t = gid + ((r & 1) ? 8 : 0);
                        const int m = ks * 8 + tig + ((r & 2) ? 4 : 0);
                        const int ti = t >> 2, tj = t & 3, di = m >> 2, dj = m & 3;
                        int x = cx - 8 + 4 * ti + di, y = cy - 8 + 4 * tj + dj;
                        x = x < 0 ? 0 : (x >= (int)nxp ? (int)nxp - 1 : x);
                        y = y < 0 ? 0 : (y >= (int)nyp ? (int)nyp - 1 : y);
                        const float2 v = uv[(size_t)x * nyp + y];
                        a[r] = pack_bf16(v.x, v.y);
                    }
#pragma unroll
                    for (int nt = 0; nt < 4; ++nt) {
                        const int nn = nt * 8 + gid;
                        mma_bf16(c[nt], a, S.w1[nn][ks * 8 + tig], S.w1[nn][ks * 8 + tig + 4]);
                    }
                }
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) {
                    const int o = nt * 8 + tig * 2;
                    const float v0 = fmaxf(c[nt][0] + S.b1[o], 0.0f), v1 = fmaxf(c[nt][1] + S.b1[o + 1], 0.0f);
                    const float v2 = fmaxf(c[nt][2] + S.b1[o], 0.0f), v3 = fmaxf(c[nt][3] + S.b1[o + 1], 0.0f);
                    S.a1[warp][sl][gid][o / 2] = pack_bf16(v0, v1);
                    S.a1[warp][sl][gid + 8][o / 2] = pack_bf16(v2, v3);
                }
            }
            __syncwarp();
            // conv2: M = 16 rows (4 seeds x 4 positions), K = 128, N = 64
            float c2[8][4] = {};
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                uint32_t a[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int row = gid + ((r & 1) ? 8 : 0);
                    const int sl = row >> 2, u = row & 3;
                    const int kp = ks * 8 + tig + ((r & 2) ? 4 : 0);   // k pair index (0..63)
                    const int g = 2 * kp, e = g >> 5, o = g & 31;
                    const int ui = u >> 1, uj = u & 1, ei = e >> 1, ej = e & 1;
                    const int t = 4 * (2 * ui + ei) + (2 * uj + ej);
                    a[r] = S.a1[warp][sl][t][o / 2];
                }
#pragma unroll
                for (int nt = 0; nt < 8; ++nt) {
                    const int nn = nt * 8 + gid;
                    mma_bf16(c2[nt], a, S.w2[nn][ks * 8 + tig], S.w2[nn][ks * 8 + tig + 4]);
                }
            }
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const int o2 = nt * 8 + tig * 2;
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int row = gid + hh * 8;
                    const int sl = row >> 2, u = row & 3;
                    const float v0 = fmaxf(c2[nt][2 * hh] + S.b2[o2], 0.0f);
                    const float v1 = fmaxf(c2[nt][2 * hh + 1] + S.b2[o2 + 1], 0.0f);
                    S.x3[warp][q * 4 + sl][(u * 64 + o2) / 2] = pack_bf16(v0, v1);
                }
            }
            __syncwarp();
        }
        // dense: M = 16 seeds, K = 256, N = 8 (2 used); the four positions' 64
        // products are summed apart and then added, as k_cnn_grid has them, so
        // a seed's prediction does not depend on which of the two forms it
        float c3[4][4] = {};
#pragma unroll
        for (int ks = 0; ks < 16; ++ks) {
            uint32_t a[4];
            a[0] = S.x3[warp][gid][ks * 8 + tig];
            a[1] = S.x3[warp][gid + 8][ks * 8 + tig];
            a[2] = S.x3[warp][gid][ks * 8 + tig + 4];
            a[3] = S.x3[warp][gid + 8][ks * 8 + tig + 4];
            mma_bf16(c3[ks >> 2], a, S.w3[gid][ks * 8 + tig], S.w3[gid][ks * 8 + tig + 4]);
        }
        float y[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) y[r] = (((c3[0][r] + c3[1][r]) + c3[2][r]) + c3[3][r]) + S.b3[r & 1];
        if (tig == 0) {
            const uint32_t s0 = grp * 16 + gid, s1 = s0 + 8;
            if (s0 < n) {
                const size_t o = index ? __ldg(index + s0) : s0;
                if (!outside || off_grid(seeds[o], nxp, nyp, pad)) {
                    out[2 * o] = y[0];
                    out[2 * o + 1] = y[1];
                }
            }
            if (s1 < n) {
                const size_t o = index ? __ldg(index + s1) : s1;
                if (!outside || off_grid(seeds[o], nxp, nyp, pad)) {
                    out[2 * o] = y[2];
                    out[2 * o + 1] = y[3];
                }
            }
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ dense inference
// Predictions for every pixel of a grid.  The patches of neighbouring seeds
// overlap: conv1's output at a tile depends only on where the tile lies, and
// conv2's on its position too, so over a grid each is formed once per pixel
// position instead of 16 and 4 times per seed,
//
//   A1(Q) = bf16(relu(W1 uv[Q .. Q+3] + b1))         (pixels clamped to the grid)
//   A2(Q) = bf16(relu(W2 A1(Q + 4(ei, ej)) + b2))
//   out(P) = b3 + sum over u of W3_u A2(P - 8 + 8(ui, uj))
//
// 9.8 k products per pixel against 50 k per seed, and no patch gathers (2 KB
// per seed).  The products, their order and the roundings are k_cnn_infer's,
// whose dense layer sums the four positions apart as well: same bits.
//
// A block walks down a strip of GRID_OUT columns, GRID_ROWS rows at a time.
// A1 and the dense layer's partial sums D stay in rings of rows in shared
// memory, so nothing is formed twice along x and 64 / 56 times along y.
// conv2 is 95 % of the work: a warp owns two 16-position tiles, so each weight
// fragment read from shared memory serves two products; A2 never leaves the
// registers (an accumulator's layout is the next product's operand layout).
// Row strides of 20 and 68 words keep the fragment loads free of bank
// conflicts.
//
// Measured (B200, 3.07 M seeds, one per pixel of 1500 x 2048, spatial order
// included): 3.54 -> 0.375 ms; the grid kernel itself 0.27 ms (350 TFLOP/s of
// mma.sync work, its fragment loads about as busy as the tensor pipe).
constexpr int GRID_OUT = 56;              // output columns of a strip
constexpr int GRID_Q = GRID_OUT + 8;      // A2 columns
constexpr int GRID_A = 80;                // A1 columns: GRID_Q + 4, in tiles of 16
constexpr int GRID_UV = GRID_A + 4;       // flow columns (GRID_A + 3 are read)
constexpr int GRID_ROWS = 4;
constexpr int GRID_THREADS = 256;

struct GridSmem {
    uint32_t uv[8][GRID_UV];              // rows of bf16 (u, v) pairs
    uint32_t a1[8][GRID_A][16 + 4];
    uint32_t w1[32][16 + 4], w2[64][64 + 4], w3[8][32 + 4];
    float b1[32], b2[64];
    float2 d[12][GRID_Q][4];              // [row][column][u]
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const uint32_t* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// flow rows k0 .. k0 + n - 1 (row k is pixel row x0 - 8 + k) into their slots
__device__ __forceinline__ void grid_load_uv(GridSmem& S, const float2* __restrict__ uv, int nxp, int nyp, int x0,
                                             int y0, int k0, int n) {
    for (int i = threadIdx.x; i < n * GRID_UV; i += GRID_THREADS) {
        const int k = k0 + i / GRID_UV, c = i % GRID_UV;
        const int x = min(max(x0 - 8 + k, 0), nxp - 1), y = min(max(y0 - 8 + c, 0), nyp - 1);
        const float2 v = __ldg(uv + (size_t)x * nyp + y);
        S.uv[k & 7][c] = pack_bf16(v.x, v.y);
    }
}

// A1 rows k0 .. k0 + GRID_ROWS - 1
__device__ __forceinline__ void grid_conv1(GridSmem& S, int k0, int warp, int lane) {
    const int gid = lane >> 2, tig = lane & 3;
    for (int tile = warp; tile < GRID_ROWS * (GRID_A / 16); tile += GRID_THREADS / 32) {
        const int k = k0 + tile / (GRID_A / 16), c0 = (tile % (GRID_A / 16)) * 16;
        float c[4][4] = {};
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint32_t a[4];
#pragma unroll
            for (int r = 0; r < 4; ++r)
                a[r] = S.uv[(k + 2 * ks + (r >> 1)) & 7][c0 + gid + ((r & 1) ? 8 : 0) + tig];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
                mma_bf16(c[nt], a, S.w1[nt * 8 + gid][ks * 8 + tig], S.w1[nt * 8 + gid][ks * 8 + tig + 4]);
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const int o = nt * 8 + tig * 2;
            S.a1[k & 7][c0 + gid][o / 2] = pack_bf16(fmaxf(c[nt][0] + S.b1[o], 0.0f), fmaxf(c[nt][1] + S.b1[o + 1], 0.0f));
            S.a1[k & 7][c0 + gid + 8][o / 2] =
                pack_bf16(fmaxf(c[nt][2] + S.b1[o], 0.0f), fmaxf(c[nt][3] + S.b1[o + 1], 0.0f));
        }
    }
}

// conv2 and the dense layer's products of rows k0 .. k0 + GRID_ROWS - 1: warp
// w owns columns 32 (w & 1) .. + 31 of row k0 + w / 2
__device__ __forceinline__ void grid_conv2(GridSmem& S, int k0, int warp, int lane) {
    const int gid = lane >> 2, tig = lane & 3;
    const int k = k0 + (warp >> 1), c0 = (warp & 1) * 32;
    const int arow = (lane & 7) + ((lane >> 3) & 1) * 8, aword = (lane >> 4) * 4;
    const int brow = (lane & 7) + (lane >> 4) * 8, bword = ((lane >> 3) & 1) * 4;
    float c[2][8][4] = {};
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
        const int e = ks >> 1, slot = (k + 4 * (e >> 1)) & 7, at = c0 + 4 * (e & 1) + arow;
        uint32_t a[2][4];
        ldmatrix_x4(a[0], &S.a1[slot][at][(ks & 1) * 8 + aword]);
        ldmatrix_x4(a[1], &S.a1[slot][at + 16][(ks & 1) * 8 + aword]);
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            uint32_t b[4];
            ldmatrix_x4(b, &S.w2[np * 16 + brow][ks * 8 + bword]);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                mma_bf16(c[t][2 * np], a[t], b[0], b[1]);
                mma_bf16(c[t][2 * np + 1], a[t], b[2], b[3]);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        float d[4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            uint32_t a[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float(&v)[4] = c[t][2 * ks + h];
                const int o = (2 * ks + h) * 8 + tig * 2;
                a[2 * h] = pack_bf16(fmaxf(v[0] + S.b2[o], 0.0f), fmaxf(v[1] + S.b2[o + 1], 0.0f));
                a[2 * h + 1] = pack_bf16(fmaxf(v[2] + S.b2[o], 0.0f), fmaxf(v[3] + S.b2[o + 1], 0.0f));
            }
            mma_bf16(d, a, S.w3[gid][ks * 8 + tig], S.w3[gid][ks * 8 + tig + 4]);
        }
        // column 2u + o of the product is output o of position u
        S.d[k % 12][c0 + 16 * t + gid][tig] = make_float2(d[0], d[1]);
        S.d[k % 12][c0 + 16 * t + gid + 8][tig] = make_float2(d[2], d[3]);
    }
}

// map [nxp][nyp] float2: the predictions of a seed at each pixel of the
// padded grid.  Blocks: strips of GRID_OUT columns (x), row ranges (y) of
// rows_per_block (a multiple of GRID_ROWS).
__global__ void __launch_bounds__(GRID_THREADS, 2)
k_cnn_grid(const float2* __restrict__ uv, int nxp, int nyp, int rows_per_block, const float* __restrict__ w1,
           const float* __restrict__ b1, const float* __restrict__ w2, const float* __restrict__ b2,
           const float* __restrict__ w3, const float* __restrict__ b3, float2* __restrict__ map) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GridSmem& S = *reinterpret_cast<GridSmem*>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int y0 = blockIdx.x * GRID_OUT, x0 = blockIdx.y * rows_per_block;
    const int rows = min(rows_per_block, nxp - x0);
    for (int i = threadIdx.x; i < 32 * 16; i += GRID_THREADS) {
        const int n = i % 32, kp = i / 32;
        S.w1[n][kp] = pack_bf16(w1[2 * kp * CNN_C1 + n], w1[(2 * kp + 1) * CNN_C1 + n]);
    }
    for (int i = threadIdx.x; i < 64 * 64; i += GRID_THREADS) {
        const int n = i % 64, kp = i / 64;
        S.w2[n][kp] = pack_bf16(w2[2 * kp * CNN_C2 + n], w2[(2 * kp + 1) * CNN_C2 + n]);
    }
    // dense weights as [2u + o][k pairs of position u]
    for (int i = threadIdx.x; i < 8 * 32; i += GRID_THREADS) {
        const int n = i / 32, kp = i % 32, h = 64 * (n >> 1) + 2 * kp;
        S.w3[n][kp] = pack_bf16(w3[h * CNN_OUT + (n & 1)], w3[(h + 1) * CNN_OUT + (n & 1)]);
    }
    if (threadIdx.x < 32) S.b1[threadIdx.x] = b1[threadIdx.x];
    if (threadIdx.x < 64) S.b2[threadIdx.x] = b2[threadIdx.x];
    const float o0 = __ldg(b3), o1 = __ldg(b3 + 1);
    grid_load_uv(S, uv, nxp, nyp, x0, y0, 0, 7);
    __syncthreads();
    grid_conv1(S, 0, warp, lane);
    // rows k of A2 and D: pixel row x0 - 8 + k; outputs start at k = 8
    for (int k0 = 0; k0 < rows + 8; k0 += GRID_ROWS) {
        __syncthreads();  // the last pass's readers of the slots written next
        grid_load_uv(S, uv, nxp, nyp, x0, y0, k0 + 7, 4);
        __syncthreads();
        grid_conv1(S, k0 + 4, warp, lane);
        __syncthreads();
        grid_conv2(S, k0, warp, lane);
        __syncthreads();
        if (k0 >= 8) {
            for (int i = threadIdx.x; i < GRID_ROWS * GRID_OUT; i += GRID_THREADS) {
                const int k = k0 + i / GRID_OUT, c = i % GRID_OUT;
                const int x = x0 - 8 + k, y = y0 + c;
                if (k - 8 >= rows || y >= nyp) continue;
                const float2 d0 = S.d[(k - 8) % 12][c][0], d1 = S.d[(k - 8) % 12][c + 8][1];
                const float2 d2 = S.d[k % 12][c][2], d3 = S.d[k % 12][c + 8][3];
                map[(size_t)x * nyp + y] =
                    make_float2((((d0.x + d1.x) + d2.x) + d3.x) + o0, (((d0.y + d1.y) + d2.y) + d3.y) + o1);
            }
        }
    }
}

// out [n][2] from the map of predictions; *outside counts the seeds whose
// pixel is not in the grid (k_cnn_infer takes those)
__global__ void k_cnn_pick(const float2* __restrict__ map, uint32_t nxp, uint32_t nyp, uint32_t pad,
                           const float2* __restrict__ seeds, const uint32_t* __restrict__ index, uint32_t n,
                           float* __restrict__ out, uint32_t* __restrict__ outside) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const size_t i = index ? __ldg(index + j) : j;
    const float2 sp = __ldg(seeds + i);
    if (off_grid(sp, nxp, nyp, pad)) {
        atomicAdd(outside, 1u);
        return;
    }
    const float2 v = __ldg(map + (size_t)((int)sp.x + (int)pad) * nyp + ((int)sp.y + (int)pad));
    out[2 * i] = v.x;
    out[2 * i + 1] = v.y;
}

// ------------------------------------------------------------------ ordering
// Seed orders are counting sorts of the seed indices by a small integer key
// (a bin); seeds within one bin keep no particular order, which is harmless:
// the traced fields do not depend on the order.

// bin of a predicted log length: higher prediction -> lower bin (issued first)
__device__ __forceinline__ uint32_t pred_bin(float v, float lo, float hi, uint32_t nb) {
    const float t = fminf(fmaxf((v - lo) / (hi - lo), 0.0f), 1.0f);  // NaN -> 0
    const uint32_t b = (uint32_t)(t * (float)(nb - 1) + 0.5f);
    return nb - 1u - b;
}

struct PredKey {
    const float* __restrict__ pred;
    uint32_t stride, col;
    float lo, hi;
    uint32_t nb;
    __device__ __forceinline__ uint32_t operator()(uint32_t i) const {
        return pred_bin(pred[(size_t)i * stride + col], lo, hi, nb);
    }
};

// Spatial key: the block_px x block_px block of the seed's pixel, blocks in
// x-major order (the grids' own layout), so seeds traced together lie close
// together and their uv / mask / slc / slt lines stay in L2.  With a
// prediction, seeds predicted at or above `thr` come first (class 0).
struct SpatialKey {
    const float2* __restrict__ seeds;
    uint32_t nx, ny, bs, nby, nblocks;
    const float* __restrict__ pred;
    uint32_t stride, col;
    float thr;
    __device__ __forceinline__ void pixel(uint32_t i, uint32_t& xi, uint32_t& yi) const {
        const float2 c = seeds[i];
        xi = (uint32_t)fminf(fmaxf(c.x + 0.5f, 0.0f), (float)(nx - 1u));  // NaN -> 0
        yi = (uint32_t)fminf(fmaxf(c.y + 0.5f, 0.0f), (float)(ny - 1u));
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t i) const {
        uint32_t xi, yi;
        pixel(i, xi, yi);
        const uint32_t cls = (pred && !(pred[(size_t)i * stride + col] >= thr)) ? 1u : 0u;
        return cls * nblocks + (xi / bs) * nby + yi / bs;
    }
};

constexpr uint32_t SMEM_BINS = 4096;  // bins counted in shared memory per block

template <class K>
__global__ void k_key_hist(K key, uint32_t n, uint32_t nb, uint32_t* __restrict__ hist) {
    extern __shared__ uint32_t sh[];
    const bool local = nb <= SMEM_BINS;
    if (local) {
        for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) sh[b] = 0;
        __syncthreads();
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t b = key(i);
        if (local) atomicAdd(sh + b, 1u);
        else atomicAdd(hist + b, 1u);
    }
    if (local) {
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x)
            if (sh[b]) atomicAdd(hist + b, sh[b]);
    }
}

// Exclusive prefix sum of a[0..n) in place, one block of 1024 threads.
__global__ void __launch_bounds__(1024) k_scan_u32(uint32_t* __restrict__ a, uint32_t n) {
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t carry;
    const unsigned FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < n; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t v = i < n ? a[i] : 0u;
        uint32_t x = v;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = lane < nw ? wsum[lane] : 0u;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, w, o);
                if (lane >= o) w += y;
            }
            wsum[lane] = w;
        }
        __syncthreads();
        const uint32_t excl = carry + (warp ? wsum[warp - 1] : 0u) + x - v;
        if (i < n) a[i] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + v;
        __syncthreads();
    }
}

// Each block places a contiguous range of seeds: per-bin counts in shared
// memory, one global reservation per (block, bin), then local slots.
template <class K>
__global__ void k_key_scatter(K key, uint32_t n, uint32_t nb, uint32_t* __restrict__ cursor,
                              uint32_t* __restrict__ order) {
    extern __shared__ uint32_t sh[];
    const uint32_t chunk = (n + gridDim.x - 1) / gridDim.x;
    const uint32_t b0 = blockIdx.x * chunk;
    const uint32_t b1 = min(n, b0 + chunk);
    if (nb > SMEM_BINS) {
        for (uint32_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) order[atomicAdd(cursor + key(i), 1u)] = i;
        return;
    }
    for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) sh[b] = 0;
    __syncthreads();
    for (uint32_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) atomicAdd(sh + key(i), 1u);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) {
        const uint32_t c = sh[b];
        sh[b] = c ? atomicAdd(cursor + b, c) : 0u;
    }
    __syncthreads();
    for (uint32_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) order[atomicAdd(sh + key(i), 1u)] = i;
}

// The seeds of a block (bin b: order[ends[b - 1] .. ends[b])) by its 8 x 8 pixel
// parts.  The counting sort leaves them in the seed list's shuffled order, so the
// lanes of a warp start all over the block and share no cache line: with one
// trajectory a seed the tracer then waits for L1, not for issue (a warp's gather
// of one tap is up to 32 lines).  Measured, both directions, order included: 4096^2
// fan terrain, d = 1, RK4 140.7 -> 82 ms; odd incised relief, d = 1, RK4 25.8 ->
// 17.8 ms; d = 2 and 3, where the trajectories of a seed are neighbours anyway, 0
// to 3 %.  16 pixel parts gain two thirds of that, 4 pixel parts the same; the
// parts as bins of the counting sort itself leave its shared counts (3.1e6 seeds:
// 49, here 37 us more).
//
// Seeds sparser than one in PART_SPARSE pixels share no lines whatever their
// order.  4096^2 fan, RK4, order and trace in ms without / with parts: one seed
// in 64 pixels 0.027 + 8.84 / 0.044 + 8.00, in 256 0.018 + 4.70 / 0.035 + 4.65,
// in 1024 0.016 + 4.15 / 0.032 + 4.13; incised relief, RK2: in 64 0.015 + 3.76 /
// 0.020 + 3.64, in 256 0.013 + 3.52 / 0.019 + 3.56.
constexpr uint32_t PART_PX = 8, PART_MAX_BLOCK = 64, PART_SPARSE = 256;
constexpr uint32_t PART_PER = 16, PART_SEEDS = 256 * PART_PER;  // seeds a block of threads holds
__global__ void __launch_bounds__(256) k_part_order(SpatialKey key, const uint32_t* __restrict__ ends,
                                                    uint32_t* __restrict__ order) {
    constexpr uint32_t PARTS = (PART_MAX_BLOCK / PART_PX) * (PART_MAX_BLOCK / PART_PX);
    __shared__ uint32_t counts[PARTS];
    const uint32_t lo = blockIdx.x ? ends[blockIdx.x - 1u] : 0u, n = ends[blockIdx.x] - lo;
    if (n > PART_SEEDS || n < 2u) return;  // (several seeds a pixel: left as they are)
    const uint32_t t = threadIdx.x, bs = key.bs;
    if (t < PARTS) counts[t] = 0;
    __syncthreads();
    uint32_t seed[PART_PER], at[PART_PER];
#pragma unroll
    for (uint32_t k = 0; k < PART_PER; ++k) seed[k] = t + 256u * k < n ? order[lo + t + 256u * k] : 0u;
#pragma unroll
    for (uint32_t k = 0; k < PART_PER; ++k) {
        if (t + 256u * k >= n) continue;
        uint32_t xi, yi;
        key.pixel(seed[k], xi, yi);
        const uint32_t part = (xi % bs) / PART_PX * (PART_MAX_BLOCK / PART_PX) + (yi % bs) / PART_PX;
        at[k] = part | atomicAdd(counts + part, 1u) << 8;
    }
    __syncthreads();
    if (t < 32u) {
        const uint32_t a = counts[2u * t], b = counts[2u * t + 1u];
        uint32_t x = a + b;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (t >= o) x += y;
        }
        counts[2u * t] = x - a - b;
        counts[2u * t + 1u] = x - b;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < PART_PER; ++k)
        if (t + 256u * k < n) order[lo + counts[at[k] & 0xffu] + (at[k] >> 8)] = seed[k];
}

template <class K>
static int counting_order(const K& key, uint32_t n, uint32_t nb, uint32_t* bins, uint32_t* order,
                          cudaStream_t s) {
    SLM_CUDA(cudaMemsetAsync(bins, 0, (size_t)nb * sizeof(uint32_t), s));
    const size_t smem = nb <= SMEM_BINS ? (size_t)nb * sizeof(uint32_t) : 0;
    unsigned grid = (n + 255) / 256;
    const unsigned cap = (unsigned)num_sms() * 4u;
    if (grid > cap) grid = cap;
    k_key_hist<K><<<grid, 256, smem, s>>>(key, n, nb, bins);
    SLM_LAUNCHED("k_key_hist");
    k_scan_u32<<<1, 1024, 0, s>>>(bins, nb);
    SLM_LAUNCHED("k_scan_u32");
    k_key_scatter<K><<<grid, 256, smem, s>>>(key, n, nb, bins, order);
    SLM_LAUNCHED("k_key_scatter");
    return SLM_OK;
}

}  // namespace slm

using namespace slm;

extern "C" {

int slm_cnn_gather(const float* uv, uint32_t nx_padded, uint32_t ny_padded, uint32_t pad,
                   const float* seed_point, const uint32_t* index, uint32_t n, float* x1, void* stream) {
    clear_error();
    if (n == 0) return SLM_OK;
    SLM_REQUIRE(uv && seed_point && x1, "NULL buffer");
    const uint64_t threads = (uint64_t)n * 256u;
    SLM_REQUIRE(threads < (1ull << 32), "too many samples");
    k_patch_gather<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const float2*>(uv), nx_padded, ny_padded, pad,
        reinterpret_cast<const float2*>(seed_point), index, n, x1);
    SLM_LAUNCHED("k_patch_gather");
    return SLM_OK;
}

int slm_cnn_rearrange(const float* src, uint32_t n, float* dst, int backward, void* stream) {
    clear_error();
    if (n == 0) return SLM_OK;
    const uint64_t threads = (uint64_t)n * 512u;
    SLM_REQUIRE(threads < (1ull << 32), "too many samples");
    const unsigned grid = (unsigned)((threads + 255) / 256);
    if (backward) k_dx2_to_da1<<<grid, 256, 0, (cudaStream_t)stream>>>(src, n, dst);
    else k_a1_to_x2<<<grid, 256, 0, (cudaStream_t)stream>>>(src, n, dst);
    SLM_LAUNCHED("k_a1_to_x2/k_dx2_to_da1");
    return SLM_OK;
}

int slm_relu_backward(const float* da, const float* z, uint64_t n, float* dz, void* stream) {
    clear_error();
    if (n == 0) return SLM_OK;
    k_relu_backward<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(da, z, n, dz);
    SLM_LAUNCHED("k_relu_backward");
    return SLM_OK;
}

int slm_bias_grad(const float* dz, uint64_t rows, int cols, float* db, void* stream) {
    clear_error();
    SLM_REQUIRE(cols > 0, "cols must be > 0");
    cudaStream_t s = (cudaStream_t)stream;
    uint32_t width = 1;  // lanes side by side on a row
    while (width < 32u && width < (uint32_t)cols) width <<= 1;
    // One block a group of columns while a lane has at most 64 rows with groups
    // of 8 columns (a memory sector); the widest groups that leave a lane 16.
    // Above that a cluster of blocks.  Measured, us (a block of 256 threads a column /
    // a cluster for all sizes / this): 100 x 32 1.6 / 4.8 / 2.6; 1000 x 64 2.6 / 5.5 /
    // 3.0; 100 x 4096 5.4 / 20.3 / 3.2; 4096 x 64 5.4 / 6.1 / 4.5; 4096 x 2 4.3 / 4.9 /
    // 3.0; 8192 x 32 8.7 / 7.2 / 7.2; 65536 x 32 56.6 / 21.8 / 21.7.
    const auto lane_rows = [&](uint32_t w) { return rows / ((BIAS_THREADS / 32u) * (32u / w)); };
    const uint32_t least = width < 8u ? width : 8u;
    if (lane_rows(least) < 64u) {
        while (width > least && lane_rows(width) >= 16u) width >>= 1;
        k_bias_grad<1><<<((uint32_t)cols + width - 1u) / width, BIAS_THREADS, 0, s>>>(dz, rows, cols, width, db);
    } else {
        const uint32_t groups = ((uint32_t)cols + width - 1u) / width;
        k_bias_grad<BIAS_CTAS><<<groups * BIAS_CTAS, BIAS_THREADS, 0, s>>>(dz, rows, cols, width, db);
    }
    SLM_LAUNCHED("k_bias_grad");
    return SLM_OK;
}

int slm_mse(const float* y, const float* t, const float* w, uint64_t n_el, float inv_n, float* dy, float* loss,
            void* stream) {
    clear_error();
    if (n_el == 0) return SLM_OK;
    k_mse<<<(unsigned)((n_el + 255) / 256), 256, 0, (cudaStream_t)stream>>>(y, t, w, n_el, inv_n, dy, loss);
    SLM_LAUNCHED("k_mse");
    return SLM_OK;
}

int slm_adam(float* w, float* wq, const float* g, float* m, float* v, uint64_t n, float lr, float b1,
             float b2, float eps, int step, int round_w, void* stream) {
    clear_error();
    if (n == 0) return SLM_OK;
    const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    k_adam<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(w, wq, g, m, v, n, lr, b1, b2, eps,
                                                                         c1, c2, round_w);
    SLM_LAUNCHED("k_adam");
    return SLM_OK;
}

static int launch_infer(const float* uv, uint32_t nx_padded, uint32_t ny_padded, uint32_t pad,
                        const float* seed_point, const uint32_t* index, uint32_t n, const float* w1, const float* b1,
                        const float* w2, const float* b2, const float* w3, const float* b3, float* out,
                        const uint32_t* outside, cudaStream_t s) {
    const size_t smem = sizeof(InferSmem);
    SLM_CUDA(cudaFuncSetAttribute(k_cnn_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint32_t groups = (n + 15) / 16;
    unsigned grid = (groups + INF_WARPS - 1) / INF_WARPS;
    const unsigned cap = (unsigned)num_sms() * 8u;
    if (grid > cap) grid = cap;
    k_cnn_infer<<<grid, INF_WARPS * 32, smem, s>>>(
        reinterpret_cast<const float2*>(uv), nx_padded, ny_padded, pad,
        reinterpret_cast<const float2*>(seed_point), index, n, w1, b1, w2, b2, w3, b3, out, outside);
    SLM_LAUNCHED("k_cnn_infer");
    return SLM_OK;
}

int slm_cnn_infer(const float* uv, uint32_t nx_padded, uint32_t ny_padded, uint32_t pad,
                  const float* seed_point, const uint32_t* index, uint32_t n, const float* w1,
                  const float* b1,
                  const float* w2, const float* b2, const float* w3, const float* b3, float* out,
                  void* stream) {
    clear_error();
    if (n == 0) return SLM_OK;
    SLM_REQUIRE(uv && seed_point && w1 && b1 && w2 && b2 && w3 && b3 && out, "NULL buffer");
    return launch_infer(uv, nx_padded, ny_padded, pad, seed_point, index, n, w1, b1, w2, b2, w3, b3, out, nullptr,
                        (cudaStream_t)stream);
}

size_t slm_cnn_infer_grid_workspace(uint32_t nx_padded, uint32_t ny_padded) {
    return (size_t)nx_padded * ny_padded * sizeof(float2) + 256;
}

int slm_cnn_infer_grid(const float* uv, uint32_t nx_padded, uint32_t ny_padded, uint32_t pad,
                       const float* seed_point, const uint32_t* index, uint32_t n, const float* w1,
                       const float* b1, const float* w2, const float* b2, const float* w3, const float* b3,
                       float* out, void* workspace, size_t workspace_bytes, void* stream) {
    clear_error();
    if (n == 0) return SLM_OK;
    SLM_REQUIRE(uv && seed_point && w1 && b1 && w2 && b2 && w3 && b3 && out && workspace, "NULL buffer");
    SLM_REQUIRE(nx_padded > 0 && ny_padded > 0 && nx_padded < (1u << 24) && ny_padded < (1u << 24) &&
                    (uint64_t)nx_padded * ny_padded < (1ull << 32),
                "grid size");
    const size_t need = slm_cnn_infer_grid_workspace(nx_padded, ny_padded);
    SLM_REQUIRE(workspace_bytes >= need, "workspace holds %zu bytes, needs %zu", workspace_bytes, need);
    SLM_REQUIRE(aligned(workspace, 8) && aligned(uv, 8) && aligned(seed_point, 8), "misaligned buffer");
    cudaStream_t s = (cudaStream_t)stream;
    float2* map = static_cast<float2*>(workspace);
    uint32_t* outside = reinterpret_cast<uint32_t*>(map + (size_t)nx_padded * ny_padded);
    SLM_CUDA(cudaMemsetAsync(outside, 0, sizeof(uint32_t), s));
    // Row ranges: a block of `rows` rows forms rows + 8 of them (and stages the
    // weights, about 8 rows' worth of time), and two blocks run on an SM at a
    // time, so take the range count with the least waves x (rows + 16).
    const uint32_t strips = (ny_padded + GRID_OUT - 1) / GRID_OUT, resident = 2u * (uint32_t)num_sms();
    uint32_t rows = 0;
    uint64_t best = ~0ull;
    for (uint32_t r = 8; r <= 512; r += GRID_ROWS) {
        const uint64_t blocks = (uint64_t)strips * ((nx_padded + r - 1) / r);
        const uint64_t cost = (blocks + resident - 1) / resident * (r + 16);
        if (cost < best) best = cost, rows = r;
    }
    const dim3 grid(strips, (nx_padded + rows - 1) / rows);
    SLM_REQUIRE(grid.y < 65536, "nx_padded too large");
    const size_t smem = sizeof(GridSmem);
    SLM_CUDA(cudaFuncSetAttribute(k_cnn_grid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_cnn_grid<<<grid, GRID_THREADS, smem, s>>>(reinterpret_cast<const float2*>(uv), (int)nx_padded, (int)ny_padded,
                                                (int)rows, w1, b1, w2, b2, w3, b3, map);
    SLM_LAUNCHED("k_cnn_grid");
    k_cnn_pick<<<(n + 255) / 256, 256, 0, s>>>(map, nx_padded, ny_padded, pad,
                                               reinterpret_cast<const float2*>(seed_point), index, n, out, outside);
    SLM_LAUNCHED("k_cnn_pick");
    return launch_infer(uv, nx_padded, ny_padded, pad, seed_point, index, n, w1, b1, w2, b2, w3, b3, out, outside, s);
}

int slm_order_by_prediction(const float* pred, uint32_t stride, uint32_t col, uint32_t n, float lo,
                            float hi, uint32_t n_bins, uint32_t* bins, uint32_t* order, void* stream) {
    clear_error();
    if (n == 0) return SLM_OK;
    SLM_REQUIRE(pred && bins && order && n_bins >= 2 && hi > lo, "bad ordering arguments");
    return counting_order(PredKey{pred, stride, col, lo, hi, n_bins}, n, n_bins, bins, order,
                          (cudaStream_t)stream);
}

uint32_t slm_order_spatial_bins(uint32_t nx, uint32_t ny, uint32_t block_px, int with_prediction) {
    if (nx == 0 || ny == 0 || block_px == 0) return 0;
    const uint64_t nbl = (uint64_t)((nx + block_px - 1) / block_px) * ((ny + block_px - 1) / block_px);
    const uint64_t nb = nbl * (with_prediction ? 2u : 1u);
    return nb < (1ull << 32) ? (uint32_t)nb : 0u;
}

int slm_order_spatial(const float* seed_point, uint32_t n, uint32_t nx, uint32_t ny, uint32_t block_px,
                      const float* pred, uint32_t stride, uint32_t col, float threshold, uint32_t* bins,
                      uint32_t n_bins_capacity, uint32_t* order, void* stream) {
    clear_error();
    if (n == 0) return SLM_OK;
    SLM_REQUIRE(seed_point && bins && order, "NULL buffer");
    SLM_REQUIRE(nx > 0 && ny > 0 && block_px > 0, "bad grid or block size");
    const uint32_t nb = slm_order_spatial_bins(nx, ny, block_px, pred != nullptr);
    SLM_REQUIRE(nb > 0 && nb <= n_bins_capacity, "bins holds %u entries, needs %u", n_bins_capacity, nb);
    const uint32_t nby = (ny + block_px - 1) / block_px;
    const uint32_t nblocks = pred ? nb / 2u : nb;
    SpatialKey key{reinterpret_cast<const float2*>(seed_point), nx, ny, block_px, nby, nblocks, pred,
                   stride, col, threshold};
    const int rc = counting_order(key, n, nb, bins, order, (cudaStream_t)stream);
    if (rc || block_px <= PART_PX || block_px > PART_MAX_BLOCK || nb > 0x7fffffffu) return rc;
    if ((uint64_t)n * PART_SPARSE < (uint64_t)nx * ny) return rc;
    k_part_order<<<nb, 256, 0, (cudaStream_t)stream>>>(key, bins, order);  // (the scatter left the bins' ends)
    SLM_LAUNCHED("k_part_order");
    return SLM_OK;
}

}  // extern "C"
