// seeds_device.cu -- create_seeds' seed list built in device memory.
//
// The same rows in the same order as slm_create_seeds (argwhere(~mask) - pad,
// then NumPy's legacy np.random.shuffle after np.random.seed(rng_seed);
// useful.py:470-517), without the host's random-access pass over the rows:
//
//   1. argwhere: slm_pick_seeds' order-preserving compaction of the mask;
//   2. the swap partners j(i), i = n-1 .. 1: drawn on the host with the
//      generator of slm_create_seeds (mt19937.hpp) by a drawing thread, and
//      copied to the device in chunks as they become final;
//   3. the permutation the swaps (i, j(i)), i = n-1 .. 1, compose to, each row
//      on its own.  Followed backwards in time (i = 1, 2, ..), what ends in
//      row r is untouched by the swaps below r; swap r brings it from row
//      j(r); and from then on, lying in row p, it is moved only by a swap
//      i > p with j(i) = p, which brings it from row i.  So with
//        next(r)  = the least i > r with j(i) = j(r),
//        first(p) = the least i > p with j(i) = p,
//      row r ends with the initial row q, q = j(r) if there is no next(r),
//      else next(r) followed through first() to its end.  About ln(n / r)
//      links on average.  The partners are chained by their target as they
//      arrive (chains of ln(n / target) on average), first() by an atomic
//      minimum; the rows are then gathered in one pass.
//
// Measured (B200), the whole seed list against the earlier rounds of reserving
// and committing swaps (two launches and a synchronisation each, 49 rounds for
// 1 M rows): 64^2 rows 1.0 -> 0.27 ms, 1024^2 3.8 -> 1.9 ms, 3000^2 27.4 -> 24.7
// ms, 8192^2 197 -> 184 ms.  What is left is the drawing thread, 1.7 to 2.7 ns a
// row.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <memory>
#include <new>
#include <thread>

#include "capi_util.cuh"
#include "mt19937.hpp"

namespace slm {

typedef unsigned long long u64;

constexpr uint32_t NO_SWAP = 0xffffffffu;

// partners per chunk copied while the next ones are drawn
static uint32_t swap_chunk(uint32_t n) { return std::min(1u << 22, std::max(1u << 16, n / 8u)); }

// swaps i = lo .. hi chained by target, and first() of the targets
__global__ void k_fy_chain(const uint32_t* __restrict__ js, uint32_t lo, uint32_t hi, uint32_t* __restrict__ head,
                           uint32_t* __restrict__ link, uint32_t* __restrict__ first) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k <= hi - lo; k += gridDim.x * blockDim.x) {
        const uint32_t i = lo + k, j = js[i];
        link[i] = atomicExch(head + j, i);
        if (j != i) atomicMin(first + j, i);
    }
}

// out[r] = the initial row that ends in row r
__global__ void k_fy_gather(const uint32_t* __restrict__ js, uint32_t n, const uint32_t* __restrict__ head,
                            const uint32_t* __restrict__ link, const uint32_t* __restrict__ first,
                            const float2* __restrict__ rows, float2* __restrict__ out) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const uint32_t j = r ? js[r] : 0u;
    uint32_t next = NO_SWAP;  // (the chain holds each swap once: at most n links)
    for (uint32_t i = head[j]; i != NO_SWAP; i = link[i])
        if (i > r && i < next) next = i;
    uint32_t q = j;
    // first(q) > q, so this ends
    for (uint32_t i = next; i != NO_SWAP; i = first[q]) q = i;
    out[r] = rows[q];
}

static size_t up256(size_t b) { return (b + 255) & ~(size_t)255; }

// Joins the drawing thread on every way out of slm_create_seeds_device.
struct Joiner {
    std::thread t;
    ~Joiner() {
        if (t.joinable()) t.join();
    }
};

}  // namespace slm

using namespace slm;

extern "C" {

size_t slm_create_seeds_device_workspace(uint64_t n_pixels) {
    if (n_pixels == 0 || n_pixels >= (1ull << 32)) return 0;
    const size_t n = (size_t)n_pixels;
    return up256(slm_pick_seeds_workspace((uint32_t)n_pixels)) + 4 * up256(4 * n) + up256(8 * n);
}

int slm_create_seeds_device(const uint8_t* mask, uint32_t nx_padded, uint32_t ny_padded, uint32_t pad,
                            int do_shuffle, uint32_t rng_seed, float* seed_point, uint64_t capacity,
                            uint64_t* n_seeds, uint32_t* generator_state, void* workspace, size_t workspace_bytes,
                            void* stream) {
    clear_error();
    SLM_REQUIRE(mask && seed_point && n_seeds && workspace, "NULL buffer");
    const uint64_t n_px = (uint64_t)nx_padded * ny_padded;
    SLM_REQUIRE(n_px > 0 && n_px < (1ull << 32), "grid size");
    const size_t need = slm_create_seeds_device_workspace(n_px);
    SLM_REQUIRE(workspace_bytes >= need, "workspace holds %zu bytes, needs %zu", workspace_bytes, need);
    SLM_REQUIRE(aligned(seed_point, 8) && aligned(workspace, 256), "seed_point must be 8-byte and workspace "
                "256-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    const size_t n_all = (size_t)n_px;
    char* w = static_cast<char*>(workspace);
    const size_t pick_bytes = up256(slm_pick_seeds_workspace((uint32_t)n_px));
    void* pick_ws = w;
    const size_t words = up256(4 * n_all);
    uint32_t* js_d = reinterpret_cast<uint32_t*>(w + pick_bytes);
    uint32_t* head = reinterpret_cast<uint32_t*>(w + pick_bytes + words);
    uint32_t* first = reinterpret_cast<uint32_t*>(w + pick_bytes + 2 * words);
    uint32_t* link = reinterpret_cast<uint32_t*>(w + pick_bytes + 3 * words);
    float2* rows = reinterpret_cast<float2*>(w + pick_bytes + 4 * words);

    // 1. argwhere(~mask) - pad, row-major, as float32 rows
    uint32_t n = 0;
    const uint32_t cap32 = capacity < 0xffffffffull ? (uint32_t)capacity : 0xffffffffu;
    const int rc = slm_pick_seeds(mask, nullptr, 0u, 0, nx_padded, ny_padded, pad,
                                  do_shuffle ? reinterpret_cast<float*>(rows) : seed_point, cap32, &n, pick_ws,
                                  pick_bytes, stream);
    *n_seeds = n;
    if (rc != SLM_OK) return rc;

    slm_mt::Mt19937 mt;
    mt.seed(rng_seed);
    if (do_shuffle && n <= 1) {
        if (n) SLM_CUDA(cudaMemcpyAsync(seed_point, rows, sizeof(float2), cudaMemcpyDeviceToDevice, s));
    } else if (do_shuffle) {
        // 2. the swap partners, drawn as slm_create_seeds draws them, by a
        // drawing thread (inline if no thread can be started) ...
        std::unique_ptr<uint32_t[]> js(new (std::nothrow) uint32_t[n]);
        if (!js) {  // no exception crosses the C ABI
            set_error("no host memory for %u swap partners", n);
            return SLM_ERR_CAPACITY;
        }
        std::atomic<uint64_t> final_above{n};  // js[i] is final for every i >= final_above
        SLM_CUDA(cudaMemsetAsync(head, 0xff, words, s));
        SLM_CUDA(cudaMemsetAsync(first, 0xff, words, s));
        Joiner drawer;
        try {
            drawer.t = std::thread([&] { mt.intervals_down(n - 1u, js.get(), &final_above); });
        } catch (...) {
            mt.intervals_down(n - 1u, js.get(), &final_above);
        }
        // 3. ... while this thread copies each chunk of final partners to the
        // device and chains it
        const uint32_t chunk = swap_chunk(n), max_grid = (uint32_t)num_sms() * 8u;
        uint32_t todo = n - 1u;  // swaps todo .. 1 remain
        while (todo >= 1u) {
            const uint64_t ready = final_above.load(std::memory_order_acquire);
            const uint32_t lo = ready > 1u ? (uint32_t)ready : 1u;
            if (lo > todo || (lo > 1u && todo - lo + 1u < chunk)) {
                std::this_thread::sleep_for(std::chrono::microseconds(20));
                continue;
            }
            const uint32_t count = todo - lo + 1u;
            SLM_CUDA(cudaMemcpyAsync(js_d + lo, js.get() + lo, (size_t)count * 4u, cudaMemcpyHostToDevice, s));
            k_fy_chain<<<std::min((count + 255u) / 256u, max_grid), 256, 0, s>>>(js_d, lo, todo, head, link, first);
            SLM_LAUNCHED("k_fy_chain");
            todo = lo - 1u;
        }
        k_fy_gather<<<(n + 255u) / 256u, 256, 0, s>>>(js_d, n, head, link, first, rows,
                                                      reinterpret_cast<float2*>(seed_point));
        SLM_LAUNCHED("k_fy_gather");
        SLM_CUDA(cudaStreamSynchronize(s));  // the partners' copies have left js
        if (drawer.t.joinable()) drawer.t.join();
    }
    if (generator_state) {
        for (int k = 0; k < 624; ++k) generator_state[k] = mt.key[k];
        generator_state[624] = (uint32_t)mt.pos;
    }
    return SLM_OK;
}

}  // extern "C"
