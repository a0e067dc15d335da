// kde.cu -- kernel-density estimation of log-distributions (histogram + fp64
// half-kernel smoothing), uni- and bivariate.
//
// Same arithmetic as the reference's opencl/kde.cl (k_sample :20-92,
// histogram_bivariate :109-123, pdf_bivariate_rows :144-228,
// pdf_bivariate_cols :249-361, histogram_univariate :383-394, pdf_univariate
// :426-526), including its mix of signed/unsigned 32-bit index arithmetic and
// the binary32 macros widened to double.  Histogram counts are exact (integer
// atomics).  The smoothing sums are fp64 in the reference's order; exp() and
// cos() are CUDA's, so smoothed values can differ from a host libm in the last
// bits of the double before the final rounding to float.
//
// Layout: histograms uint32 [n_hist_bins] or [n_hist_bins^2] (row = x bin),
// partial pdf float [n_hist_bins^2], pdf float [n_pdf_points] or
// [n_pdf_points^2].  The rows and cols passes take the kernel weights they
// reuse from a per-block shared-memory table.
#include <algorithm>
#include <cmath>
#include "capi_util.cuh"

namespace slm {

__device__ __forceinline__ double k_sample(uint32_t kind, double x, double w) {
    switch (kind) {
    case 0: return fabs(x) < w ? 1.0 : 0.0;
    case 1: return fmax((double)1.0f - fabs(x / w), 0.0);
    case 2: return fmax((double)1.0f - (x / w) * (x / w), 0.0);
    case 3: return fmax(cos(1.57079632679489661923 * x), 0.0);
    default: {
        const double s = w * (double)0.4f;
        return exp((double)-0.5f * (x / s) * (x / s));
    }
    }
}

constexpr uint32_t HIST_BLOCK = 512;

// float -> uint as C's truncation through a 64-bit integer
__device__ __forceinline__ uint32_t f2u(float v) { return (uint32_t)__float2ll_rz(v); }

__device__ __forceinline__ uint32_t bin_univariate(float v, const slm_params& p) {
    const float bin_x = __fdiv_rn(v - p.logx_min, p.logx_range);
    const uint32_t idx = f2u(bin_x * (float)p.n_hist_bins);
    return idx < p.n_hist_bins - 1u ? idx : p.n_hist_bins - 1u;
}

// A univariate histogram has few bins for its data (2048 for a grid's pixels),
// so counting in memory is a queue of atomics at each popular bin.  With
// LOCAL a block counts in shared memory and adds its bins at the end: 2 M
// values in 2048 bins take 232 us without, 11 us with (B200).
template <bool LOCAL>
__global__ void __launch_bounds__(HIST_BLOCK)
k_histogram_univariate(const slm_params p, const float* __restrict__ data, uint32_t n,
                       uint32_t* __restrict__ hist) {
    extern __shared__ uint32_t bins[];
    if (LOCAL) {
        for (uint32_t b = threadIdx.x; b < p.n_hist_bins; b += HIST_BLOCK) bins[b] = 0u;
        __syncthreads();
    }
    uint32_t* count = LOCAL ? bins : hist;
    const uint32_t stride = gridDim.x * HIST_BLOCK;
    for (uint64_t g = (uint64_t)blockIdx.x * HIST_BLOCK + threadIdx.x; g < n; g += stride)
        atomicAdd(count + bin_univariate(__ldg(data + g), p), 1u);
    if (LOCAL) {
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < p.n_hist_bins; b += HIST_BLOCK)
            if (bins[b]) atomicAdd(hist + b, bins[b]);
    }
}

__global__ void k_histogram_bivariate(const slm_params p, const float2* __restrict__ data,
                                      uint32_t n, uint32_t* __restrict__ hist) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    const uint32_t nb = p.n_hist_bins;
    const float2 v = data[g];
    const float bx = __fdiv_rn(v.x - p.logx_min, p.logx_range);
    const float by = __fdiv_rn(v.y - p.logy_min, p.logy_range);
    uint32_t ix = f2u(bx * (float)(nb - 1u));
    uint32_t iy = f2u(by * (float)(nb - 1u));
    ix = ix < nb - 1u ? ix : nb - 1u;
    iy = iy < nb - 1u ? iy : nb - 1u;
    atomicAdd(hist + (iy + nb * ix), 1u);
}

// one thread per pdf point (kde.cl:426-526).  The weight of (k, h) is every
// point's: the block forms PDF_TABLE of them at a time in shared memory (an
// exponential and divisions each), in the order the points use them.
constexpr uint32_t PDF_BLOCK = 32, PDF_TABLE = 1024;

__global__ void __launch_bounds__(PDF_BLOCK)
k_pdf_univariate(const slm_params p, const uint32_t* __restrict__ hist, float* __restrict__ pdf) {
    __shared__ double table[PDF_TABLE];
    const uint32_t pdf_idx = blockIdx.x * PDF_BLOCK + threadIdx.x;
    const uint32_t nbpp = p.n_hist_bins / p.n_pdf_points;
    const double half_dx = (double)__fdiv_rn(p.pdf_dx, 2.0f);
    const uint64_t total = ((uint64_t)p.n_kdf_part_points_x + 1u) * nbpp;
    double acc = 0.0, kw = 0.0;
    uint32_t k = 0, h = 0;  // of the weight at hand
    for (uint64_t t0 = 0; t0 < total; t0 += PDF_TABLE) {
        const uint32_t m = (uint32_t)(total - t0 < PDF_TABLE ? total - t0 : PDF_TABLE);
        __syncthreads();
        for (uint32_t t = threadIdx.x; t < m; t += PDF_BLOCK) {
            const uint32_t tk = (uint32_t)((t0 + t) / nbpp), th = (uint32_t)((t0 + t) % nbpp);
            const double edge = (double)tk * (double)p.pdf_dx - half_dx;
            table[t] = k_sample(p.kdf_kind, edge + (double)p.bin_dx * ((double)th + 0.5), (double)p.kdf_width_x);
        }
        __syncthreads();
        if (pdf_idx >= p.n_pdf_points) continue;
        for (uint32_t t = 0; t < m; ++t) {
            const double kv = table[t];
            const int32_t col_r = (int32_t)(pdf_idx + k);
            const int32_t col_l = (int32_t)(pdf_idx - k + 1u);
            if (col_r < (int32_t)p.n_pdf_points) {
                acc += (double)__ldg(hist + ((uint32_t)col_r * nbpp + h)) * kv;
            }
            if (k != 0u && col_l > 0) acc += (double)__ldg(hist + ((uint32_t)col_l * nbpp - h - 1u)) * kv;
            if (col_r < (int32_t)p.n_pdf_points) kw += kv;
            if (k != 0u && col_l > 0) kw += kv;
            if (++h == nbpp) {
                h = 0;
                ++k;
            }
        }
    }
    if (pdf_idx < p.n_pdf_points) pdf[pdf_idx] = (float)((double)(float)acc / kw);
}

// one thread per histogram bin; weights k_sample(k, n_y + 0.5), k = 0..n_y,
// shared per block (kde.cl:144-228)
__global__ void k_pdf_bivariate_rows(const slm_params p, const uint32_t* __restrict__ hist,
                                     float* __restrict__ partial) {
    extern __shared__ double wtab[];
    const uint32_t nk = p.n_kdf_part_points_y + 1u;
    const double k_width = (double)p.n_kdf_part_points_y + 0.5;
    for (uint32_t k = threadIdx.x; k < nk; k += blockDim.x)
        wtab[k] = k_sample(p.kdf_kind, (double)k, k_width);
    __syncthreads();
    const uint32_t nb = p.n_hist_bins;
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= nb * nb) return;
    const int32_t col = (int32_t)(gid % nb);
    const int32_t row = (int32_t)(gid / nb);
    double acc = 0.0, kw = 1.0;
    for (uint32_t k = 0; k < nk; ++k) {
        const int32_t col_r = col + (int32_t)k;
        const int32_t col_l = col - (int32_t)k + 1;
        const double kv = wtab[k];
        const bool ok_r = col_r < (int32_t)nb;
        const bool ok_l = (k != 0u) && (col_l >= 0);
        const uint32_t hr = (uint32_t)row * nb + (uint32_t)col_r;
        const uint32_t hl = (uint32_t)row * nb + (uint32_t)col_l;
        if (ok_r) acc += kv * (double)hist[hr];
        if (ok_l) acc += kv * (double)hist[hl];
        if (ok_r) kw += kv;
        if (ok_l) kw += kv;
    }
    partial[gid] = (float)(acc / kw);
}

// one thread per pdf point; weights k_sample(hrow + k*nbpp, n_x + 0.5) shared
// per block (kde.cl:249-361)
__global__ void k_pdf_bivariate_cols(const slm_params p, const float* __restrict__ partial,
                                     float* __restrict__ pdf) {
    extern __shared__ double wtab[];
    const uint32_t nb = p.n_hist_bins, np = p.n_pdf_points;
    const uint32_t nbpp = nb / np;
    const uint32_t nk = p.n_kdf_part_points_x + 1u;
    const double k_width = (double)p.n_kdf_part_points_x + 0.5;
    for (uint32_t t = threadIdx.x; t < nk * nbpp; t += blockDim.x) {
        const uint32_t k = t / nbpp, hrow = t % nbpp;
        wtab[t] = k_sample(p.kdf_kind, (double)(int32_t)hrow + ((double)k) * (double)nbpp, k_width);
    }
    __syncthreads();
    const uint32_t pdf_idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (pdf_idx >= np * np) return;
    const int32_t pcol = (int32_t)(pdf_idx % np);
    const int32_t prow = (int32_t)(pdf_idx / np);
    double acc = 0.0, kw = 1.0;
    for (uint32_t k = 0; k < nk; ++k) {
        const int32_t row_dn = prow + (int32_t)k;
        const int32_t row_up = prow - (int32_t)k;
        const int32_t off_dn = (int32_t)(((uint32_t)pcol + (uint32_t)row_dn * nb) * nbpp);
        const int32_t off_up = (int32_t)(((uint32_t)pcol + (uint32_t)row_up * nb) * nbpp);
        for (int32_t hrow = 0; hrow < (int32_t)nbpp; ++hrow) {
            const double kv = wtab[k * nbpp + (uint32_t)hrow];
            for (int32_t hcol = 0; hcol < (int32_t)nbpp; ++hcol) {
                const int32_t i_dn = (int32_t)((uint32_t)off_dn + (uint32_t)hrow * nb + (uint32_t)hcol);
                const int32_t i_up = (int32_t)((uint32_t)off_up + (nbpp - 1u - (uint32_t)hrow) * nb
                                               + (uint32_t)hcol);
                const bool ok_dn = i_dn < (int32_t)(nb * nb);
                const bool ok_up = (k != 0u) && (i_up >= 0);
                if (ok_dn) acc += kv * (double)partial[(uint32_t)i_dn];
                if (ok_up) acc += kv * (double)partial[(uint32_t)i_up];
                if (ok_dn) kw += kv;
                if (ok_up) kw += kv;
            }
        }
    }
    pdf[pdf_idx] = (float)(acc / kw);
}

// ------------------------------------------------------------------ spread of the data
// Sums of d and d^2, d = value - the column's first value, per column of rows
// of COLS floats, in double.  Each block sums a fixed range of rows, and one
// block then adds the blocks' sums in order, so the result does not depend on
// the order blocks run in.
constexpr uint32_t MOMENT_BLOCK = 256;

template <int COLS>
__device__ __forceinline__ void block_sum(double (&v)[2 * COLS], double* out) {
    __shared__ double part[MOMENT_BLOCK / 32][2 * COLS];
#pragma unroll
    for (int c = 0; c < 2 * COLS; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
    if ((threadIdx.x & 31u) == 0)
        for (int c = 0; c < 2 * COLS; ++c) part[threadIdx.x >> 5][c] = v[c];
    __syncthreads();
    if (threadIdx.x < 2 * COLS) {
        double s = 0.0;
        for (uint32_t w = 0; w < MOMENT_BLOCK / 32; ++w) s += part[w][threadIdx.x];
        out[threadIdx.x] = s;
    }
}

template <int COLS>
__global__ void __launch_bounds__(MOMENT_BLOCK)
k_moments(const float* __restrict__ data, uint64_t n, uint64_t rows_per_block, double* __restrict__ partial) {
    const uint64_t lo = (uint64_t)blockIdx.x * rows_per_block;
    const uint64_t hi = lo + rows_per_block < n ? lo + rows_per_block : n;
    double v[2 * COLS] = {}, first[COLS];
    for (int c = 0; c < COLS; ++c) first[c] = (double)__ldg(data + c);
    for (uint64_t i = lo + threadIdx.x; i < hi; i += MOMENT_BLOCK)
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            const double d = (double)__ldg(data + COLS * i + c) - first[c];
            v[2 * c] += d;
            v[2 * c + 1] += d * d;
        }
    block_sum<COLS>(v, partial + (uint64_t)blockIdx.x * 2 * COLS);
}

template <int COLS>
__global__ void __launch_bounds__(MOMENT_BLOCK)
k_moments_sum(const double* __restrict__ partial, uint32_t blocks, double* __restrict__ out) {
    double v[2 * COLS] = {};
    for (uint32_t b = threadIdx.x; b < blocks; b += MOMENT_BLOCK)
#pragma unroll
        for (int c = 0; c < 2 * COLS; ++c) v[c] += partial[(uint64_t)b * 2 * COLS + c];
    block_sum<COLS>(v, out);
}

// out[i] = hist[i] / scale
__global__ void k_scale_counts(const uint32_t* __restrict__ hist, uint64_t n, double scale, double* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = __ddiv_rn((double)hist[i], scale);
}

}  // namespace slm

using namespace slm;

static int check_kde(const slm_params* p, bool bivariate) {
    SLM_REQUIRE(p != nullptr, "params is NULL");
    SLM_REQUIRE(p->n_hist_bins > 0 && p->n_pdf_points > 0, "n_hist_bins and n_pdf_points must be > 0");
    SLM_REQUIRE(p->n_hist_bins % p->n_pdf_points == 0,
                "n_hist_bins (%u) must be a multiple of n_pdf_points (%u)", p->n_hist_bins,
                p->n_pdf_points);
    SLM_REQUIRE(p->kdf_kind <= 4, "kdf_kind %u unknown", p->kdf_kind);
    if (bivariate)
        SLM_REQUIRE((uint64_t)p->n_hist_bins * p->n_hist_bins < (1ull << 31),
                    "n_hist_bins^2 must fit a signed 32-bit index");
    return SLM_OK;
}

extern "C" {

int slm_histogram_univariate(const slm_params* p, const float* sl, uint32_t n_data, uint32_t* hist,
                             void* stream) {
    clear_error();
    int rc = check_kde(p, false);
    if (rc) return rc;
    if (n_data == 0) return SLM_OK;
    SLM_REQUIRE(sl && hist, "NULL buffer");
    // Counting in memory takes n / bins (the queue of atomics at a popular bin),
    // counting in shared memory a block's values, four a bin, and its bins at the
    // end: bins.  The lines cross at n ~ bins^2 / 180, and not below 16384 values,
    // where both are a few us.  Measured, us (memory / shared): 64 bins, 9000
    // values 2.9 / 3.7, 20000 5.1 / 3.9; 2048 bins, 40000 5.3 / 6.1, 60000 7.9 /
    // 5.6; 4096 bins, 100000 7.7 / 8.7, 200000 14.5 / 8.6; 8192 bins, 200000 7.9 /
    // 15.5, 400000 15.6 / 15.5; 12288 bins, 60000 2.8 / 25.7, 1 M 27.2 / 22.0.
    // As many blocks as four values a bin leave, two an SM at most.
    const uint64_t bins = p->n_hist_bins;
    const uint32_t wide = (uint32_t)num_sms() * 2u;
    if (bins <= 12288u && n_data >= 16384u + bins * bins / 180u) {
        const unsigned grid = std::min(n_data / std::max(4u * p->n_hist_bins, 4096u), wide);
        k_histogram_univariate<true><<<grid, HIST_BLOCK, p->n_hist_bins * sizeof(uint32_t), (cudaStream_t)stream>>>(
            *p, sl, n_data, hist);
    } else {
        const unsigned grid = std::min((n_data - 1u) / HIST_BLOCK + 1u, wide * 8u);
        k_histogram_univariate<false><<<grid, HIST_BLOCK, 0, (cudaStream_t)stream>>>(*p, sl, n_data, hist);
    }
    SLM_LAUNCHED("k_histogram_univariate");
    return SLM_OK;
}

int slm_histogram_bivariate(const slm_params* p, const float* sl, uint32_t n_data, uint32_t* hist,
                            void* stream) {
    clear_error();
    int rc = check_kde(p, true);
    if (rc) return rc;
    if (n_data == 0) return SLM_OK;
    SLM_REQUIRE(sl && hist && aligned(sl, 8), "NULL or misaligned buffer");
    const unsigned block = 256, grid = (n_data + block - 1) / block;
    k_histogram_bivariate<<<grid, block, 0, (cudaStream_t)stream>>>(
        *p, reinterpret_cast<const float2*>(sl), n_data, hist);
    SLM_LAUNCHED("k_histogram_bivariate");
    return SLM_OK;
}

int slm_pdf_univariate(const slm_params* p, const uint32_t* hist, float* pdf, void* stream) {
    clear_error();
    int rc = check_kde(p, false);
    if (rc) return rc;
    SLM_REQUIRE(hist && pdf, "NULL buffer");
    const unsigned grid = (p->n_pdf_points + PDF_BLOCK - 1) / PDF_BLOCK;
    k_pdf_univariate<<<grid, PDF_BLOCK, 0, (cudaStream_t)stream>>>(*p, hist, pdf);
    SLM_LAUNCHED("k_pdf_univariate");
    return SLM_OK;
}

int slm_pdf_bivariate_rows(const slm_params* p, const uint32_t* hist, float* partial, void* stream) {
    clear_error();
    int rc = check_kde(p, true);
    if (rc) return rc;
    SLM_REQUIRE(hist && partial, "NULL buffer");
    const size_t smem = (size_t)(p->n_kdf_part_points_y + 1u) * sizeof(double);
    SLM_REQUIRE(smem <= 160 * 1024, "n_kdf_part_points_y %u too large", p->n_kdf_part_points_y);
    if (smem > 48 * 1024)
        SLM_CUDA(cudaFuncSetAttribute(k_pdf_bivariate_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint64_t n = (uint64_t)p->n_hist_bins * p->n_hist_bins;
    const unsigned block = 256, grid = (unsigned)((n + block - 1) / block);
    k_pdf_bivariate_rows<<<grid, block, smem, (cudaStream_t)stream>>>(*p, hist, partial);
    SLM_LAUNCHED("k_pdf_bivariate_rows");
    return SLM_OK;
}

int slm_pdf_bivariate_cols(const slm_params* p, const float* partial, float* pdf, void* stream) {
    clear_error();
    int rc = check_kde(p, true);
    if (rc) return rc;
    SLM_REQUIRE(partial && pdf, "NULL buffer");
    const uint32_t nbpp = p->n_hist_bins / p->n_pdf_points;
    const size_t smem = (size_t)(p->n_kdf_part_points_x + 1u) * nbpp * sizeof(double);
    SLM_REQUIRE(smem <= 160 * 1024, "n_kdf_part_points_x %u too large", p->n_kdf_part_points_x);
    if (smem > 48 * 1024)
        SLM_CUDA(cudaFuncSetAttribute(k_pdf_bivariate_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint64_t n = (uint64_t)p->n_pdf_points * p->n_pdf_points;
    const unsigned block = 128, grid = (unsigned)((n + block - 1) / block);
    k_pdf_bivariate_cols<<<grid, block, smem, (cudaStream_t)stream>>>(*p, partial, pdf);
    SLM_LAUNCHED("k_pdf_bivariate_cols");
    return SLM_OK;
}

// the block count is fixed, so the sums' order is
static constexpr uint32_t MOMENT_BLOCKS = 512;

size_t slm_column_moments_workspace(uint32_t cols) { return (size_t)MOMENT_BLOCKS * 2 * cols * sizeof(double); }

int slm_column_moments(const float* data, uint64_t n_rows, uint32_t cols, double* out, void* workspace,
                       size_t workspace_bytes, void* stream) {
    clear_error();
    SLM_REQUIRE(data && out && workspace && n_rows > 0, "NULL buffer or no rows");
    SLM_REQUIRE(cols == 1 || cols == 2, "cols must be 1 or 2");
    SLM_REQUIRE(workspace_bytes >= slm_column_moments_workspace(cols), "workspace holds %zu bytes, needs %zu",
                workspace_bytes, slm_column_moments_workspace(cols));
    SLM_REQUIRE(aligned(out, 8) && aligned(workspace, 8) && aligned(data, 4), "misaligned buffer");
    cudaStream_t s = (cudaStream_t)stream;
    double* partial = static_cast<double*>(workspace);
    const uint64_t rows = (n_rows + MOMENT_BLOCKS - 1) / MOMENT_BLOCKS;
    const uint32_t blocks = (uint32_t)((n_rows + rows - 1) / rows);
    if (cols == 1) {
        k_moments<1><<<blocks, MOMENT_BLOCK, 0, s>>>(data, n_rows, rows, partial);
        k_moments_sum<1><<<1, MOMENT_BLOCK, 0, s>>>(partial, blocks, out);
    } else {
        k_moments<2><<<blocks, MOMENT_BLOCK, 0, s>>>(data, n_rows, rows, partial);
        k_moments_sum<2><<<1, MOMENT_BLOCK, 0, s>>>(partial, blocks, out);
    }
    SLM_LAUNCHED("k_moments");
    return SLM_OK;
}

int slm_scale_counts(const uint32_t* hist, uint64_t n, double scale, double* out, void* stream) {
    clear_error();
    if (n == 0) return SLM_OK;
    SLM_REQUIRE(hist && out && aligned(out, 8), "NULL or misaligned buffer");
    SLM_REQUIRE(n < (1ull << 39), "too many counts");
    k_scale_counts<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(hist, n, scale, out);
    SLM_LAUNCHED("k_scale_counts");
    return SLM_OK;
}

}  // extern "C"
