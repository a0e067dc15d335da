// trace.cu -- streamline tracing kernels and their C ABI.
//
//   k_fields_plain       one thread per (seed, sub-pixel) trajectory
//   k_fields_persistent  persistent warps; a lane whose trajectory ends takes
//                        the next one from a global work queue, so warps stay
//                        full however uneven the trajectory lengths are
//   k_trajectory         one thread per seed, records char2 steps
//
// Both field kernels produce identical slc/slt: every trajectory is computed
// bit-exactly as the reference's jittered_trajectory
// (opencl/jittertrajectory.cl:42-88) and the per-pixel sums are integer sums,
// independent of order.  Each lane merges consecutive visits to the same pixel
// (a step is at most integrator_step_factor px, so a trajectory usually visits
// a pixel several times in a row) and adds the merged count and length sum
// with one 64-bit atomic each when it moves to another pixel.
#include "capi_util.cuh"
#include "trace_fast.cuh"


static_assert(sizeof(slm_tile) == 40, "slm_tile layout is part of the ABI");

// Resident blocks of 256 threads per SM the field kernels are compiled for
// (64 registers a thread; 48, five blocks, spill the RK4 step).
constexpr int FIELD_BLOCKS = 4;

namespace slm {

// Run-length merge of pixel visits for one lane.
struct Acc {
    uint32_t idx, cnt;
    u64 sum;
};

__device__ __forceinline__ void acc_flush(Acc& a, u64* __restrict__ slc, u64* __restrict__ slt) {
    if (a.cnt) {
        atomicAdd(slt + a.idx, a.sum);
        atomicAdd(slc + a.idx, (u64)a.cnt);
        a.cnt = 0;
    }
}

// *p += v if `on` (predicated: no branch around it)
__device__ __forceinline__ void add_if(bool on, u64* p, u64 v) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q red.global.add.u64 [%1], %2;\n\t}"
                 :
                 : "r"((uint32_t)on), "l"(p), "l"(v));  // nothing here reads the sums
}

// *p if `on`, else 1 (predicated: no branch around it)
__device__ __forceinline__ uint32_t load_if(bool on, const uint8_t* p) {
    uint32_t v;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\tmov.u32 %0, 1;\n\t@q ld.global.nc.u8 %0, [%2];\n\t}"
        : "=r"(v)
        : "r"((uint32_t)on), "l"(p));
    return v;
}

// writearray.cl:31-40: slt += (uint)(l+0.5), slc += 1, if `visits`.  A lane on
// a trajectory has a run open (its start opened or continued one), so the
// visits of its steps need not ask.
template <bool OPEN>
__device__ __forceinline__ void acc_visit(Acc& a, uint32_t idx, float l, bool visits, u64* __restrict__ slc,
                                          u64* __restrict__ slt) {
    const uint32_t v = __float2uint_rz(l + 0.5f);
    // selects and predicated atomics, no branch: some lane of a warp changes
    // pixel in nearly every step
    const bool open = OPEN || a.cnt != 0u;
    const bool same = (idx == a.idx) & open;
    const bool flush = visits & !same & open;
    add_if(flush, slt + a.idx, a.sum);
    add_if(flush, slc + a.idx, (u64)a.cnt);
    const uint32_t cnt = (same ? a.cnt : 0u) + 1u;
    const u64 sum = (same ? a.sum : 0ull) + v;
    a.cnt = visits ? cnt : a.cnt;
    a.sum = visits ? sum : a.sum;
    a.idx = visits ? idx : a.idx;
}

// State of one jittered field trajectory between steps.
struct FieldLane {
    Vec2 a;
    float l, dt;
    uint32_t n, rng;   // RK steps so far (the one that ends on a masked pixel included)
    uint32_t item;     // queue position
    bool alive;
    F2 t;              // 2^23 + pixel of a, and the byte offset of that
    uint32_t off;      // pixel's vector in uv (kept for the fast step)
};

// A grid as a lane sees it: its geometry, the fast step's form of it, its
// first pixel in the uv / mask arrays and the offset from a pixel's index
// there to its accumulators.
struct FieldGrid {
    Geo g;
    FastGeo f;
    uint32_t base, acc_offset;
};

// A trajectory ready to start: its first point, generator state and pixel (in
// the uv / mask arrays), its queue position, and what its kernel adds.
struct FieldStart {
    Vec2 a;
    uint32_t rng, idx, item, tag;
};

// The start of sub-pixel `sub` (= j*d + i) of the seed at `c`, whose RNG
// stream is that of seed index `rng_idx` (integratefields.cl:83-113;
// jittertrajectory.cl:56-62), on the grid of geometry g and first pixel
// `base`; false if it lies on a masked pixel (a trajectory without visits or
// steps).
template <int FORM>
__device__ __forceinline__ bool start_at(FieldStart& st, float2 c, uint32_t rng_idx, uint32_t sub,
                                         const uint8_t* __restrict__ mask, const slm_params& p, const Geo& g,
                                         uint32_t base) {
    const uint32_t d = p.subpixel_seed_point_density;
    const uint32_t j = sub / d, i = sub % d;
    st.a.x = c.x + ((float)i * p.subpixel_seed_step - p.subpixel_seed_halfspan);
    st.a.y = c.y + ((float)j * p.subpixel_seed_step - p.subpixel_seed_halfspan);
    st.rng = seed_rng(rng_idx);
    // the fast draws form (state + 1) * A without wrapping the sum: the state
    // whose successor wraps to 0 has the same successor as the modulus - 1
    if (FORM && st.rng == 0xffffffffu) st.rng = LEHMER_M - 1u;
    st.idx = base + pixel_of(st.a, p, g);
    return __ldg(mask + st.idx) == 0;
}

// Put the lane on the trajectory `st` of the grid G: its first visit.
template <int FORM>
__device__ __forceinline__ void field_begin(FieldLane& s, const FieldStart& st, const slm_params& p,
                                            const FieldGrid& G, Acc& acc, u64* __restrict__ slc,
                                            u64* __restrict__ slt) {
    s.a = st.a;
    s.rng = st.rng;
    s.l = 0.0f;
    s.dt = G.g.dt_max;
    s.n = 0;
    s.item = st.item;
    if (FORM) {
        s.t = pixel_magic_clamped(s.a, p.pad_width_pp5, G.g.nxp, G.g.nyp);
        s.off = 8u * st.idx;
    }
    acc_visit<false>(acc, G.acc_offset + st.idx, 0.0f, true, slc, slt);
    s.alive = (0.0f < p.max_length) && (0u < p.max_n_steps);
}

// queue item -> (queue position, sub-pixel index)
__device__ __forceinline__ void split_item(u64 item, uint32_t dd, uint32_t& pos, uint32_t& sub) {
    if (item < 0x100000000ull) {  // 32-bit division unless the queue is huge
        const uint32_t it = (uint32_t)item;
        pos = it / dd;
        sub = it - pos * dd;
    } else {
        pos = (uint32_t)(item / dd);
        sub = (uint32_t)(item - (u64)pos * dd);
    }
}

// The start of trajectory `item` = (seed - seed_begin) * d*d + j*d + i of one
// grid.
//
// `order` (optional) maps queue positions to seed indices, so trajectories can
// be traced in any order; the RNG stream still follows the seed index, so no
// trajectory changes.
template <int FORM>
__device__ __forceinline__ bool start_of(FieldStart& st, u64 item, uint32_t seed_begin,
                                         const float2* __restrict__ seeds, const uint32_t* __restrict__ order,
                                         const uint8_t* __restrict__ mask, const slm_params& p, const Geo& g) {
    const uint32_t d = p.subpixel_seed_point_density;
    uint32_t pos, sub;
    split_item(item, d * d, pos, sub);
    const uint32_t seed_idx = order ? __ldg(order + seed_begin + pos) : seed_begin + pos;
    st.item = (uint32_t)item;
    return start_at<FORM>(st, __ldg(seeds + seed_idx), seed_idx, sub, mask, p, g, 0u);
}

// One pass of the while loop of jittered_trajectory with
// runge_kutta_step_write_sl_data (rungekutta.cl:163-186).  The Euler branch
// of that loop is unreachable (get_array_idx clamps into the grid).  FORM, but
// for STEP_GENERAL: the launch meets fast_params, and the grid fast_grid
// (GATED: or it has no interior, so that every step is rk_step's).
//
// All lanes of a warp run it together (WARP): those without a live trajectory
// compute along on whatever point they have, reading within the grid, and
// leave no visit and no count.
template <int ORDER, int FORM, bool GATED, bool WARP>
__device__ __forceinline__ void field_step(FieldLane& s, const uint8_t* __restrict__ mask,
                                           const float2* __restrict__ uv, const slm_params& p,
                                           const FastConst& k, const FieldGrid& G, Acc& acc,
                                           u64* __restrict__ slc, u64* __restrict__ slt) {
    float dl, dt;
    uint32_t idx;
    const bool on = !WARP || s.alive;
    if (FORM) {
        FastStep st;
        const bool ok = step_fast<ORDER, FORM, GATED>(s.a, s.t, s.off, s.dt, G.g.cf, s.rng, uv, G.f, k, st);
        float ex = st.d2.x - st.d1.x, ey = st.d2.y - st.d1.y;
        dt = G.g.dt_max;
        // rare: a guard failed, or the next dt is not DT_MAX by the cheap test
        const bool rare = on & !(ok & (s.dt * s.dt * G.f.kerr >= __fmaf_rn(ey, ey, ex * ex)));
        if (WARP ? __any_sync(0xffffffffu, rare) : rare) {
            if (rare) {
                if (!ok) {
                    st = step_exact<ORDER, true>(s.a, s.dt, s.rng, G.g.cf, uv, G.base, p, G.g.nxp, G.g.nyp);
                    ex = st.d2.x - st.d1.x;
                    ey = st.d2.y - st.d1.y;
                }
                dt = next_dt_fast(ex, ey, s.dt, G.g.dt_max, G.g.gs, G.f.gs_rcp, p.adjusted_max_error);
            }
        }
        s.rng = st.rng;
        s.off = st.off;
        s.a = st.next;
        s.t = st.t;
        dl = quantised_length(__fmaf_rn(st.d2.y, st.d2.y, st.d2.x * st.d2.x));
        // a batch's tiles may lie beyond the byte offsets' range (their steps are
        // then step_exact's); a single grid that is traced fast does not
        idx = GATED ? st.idx : st.off >> 3;
        s.alive = load_if(on, mask + idx) == 0u;
    } else {
        const Step st = rk_step<ORDER, true>(s.a, s.dt, s.rng, uv + G.base, p, G.g);
        idx = G.base + st.idx;
        const float err = vlen(div_gs(st.d2.x - st.d1.x, G.g), div_gs(st.d2.y - st.d1.y, G.g));
        dl = vlen(st.d2.x, st.d2.y);
        dt = next_dt(s.dt, err, p, G.g);
        s.a = st.next;
        s.alive = __ldg(mask + idx) == 0;
    }
    // a masked pixel ends the trajectory without a visit
    s.l = s.l + dl;
    s.n += (uint32_t)on;
    s.dt = dt;  // (a halted trajectory has no next step)
    acc_visit<true>(acc, G.acc_offset + idx, s.l, s.alive, slc, slt);
    s.alive = s.alive & !(dl < p.integration_halt_threshold) & (s.l < p.max_length) & (s.n < p.max_n_steps);
}

// The grid of a launch's parameter block.
__device__ __forceinline__ FieldGrid grid_of(const slm_params& p, const FastGeo& f) {
    return FieldGrid{geo_of(p), f, 0u, 0u};
}

// per-trajectory RK step count, saturated to 16 bits, indexed by queue position
template <bool RECORD>
__device__ __forceinline__ void record_end(const FieldLane& s, uint16_t* __restrict__ item_steps) {
    if (RECORD) item_steps[s.item] = (uint16_t)(s.n < 65535u ? s.n : 65535u);
}

__device__ __forceinline__ void warp_add_counters(u64 steps, u64 ntraj, u64* work) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        steps += __shfl_xor_sync(0xffffffffu, steps, o);
        ntraj += __shfl_xor_sync(0xffffffffu, ntraj, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(work + 1, steps);
        atomicAdd(work + 2, ntraj);
    }
}

// Steps of a lane's finished trajectories, gathered when the lane takes its
// next one (a trajectory's own count is 32 bits wide, a launch's is not).
struct LaneCount {
    u64 steps, ntraj;
};

__device__ __forceinline__ void count_trajectory(LaneCount& c, FieldLane& s) {
    c.steps += s.n;
    s.n = 0;
}

template <int ORDER, bool RECORD, int FORM>
__global__ void __launch_bounds__(256, FIELD_BLOCKS)
k_fields_plain(const __grid_constant__ slm_params p, const __grid_constant__ FastGeo f,
               const __grid_constant__ FastConst k, const float2* __restrict__ seeds, uint32_t seed_begin,
               u64 n_items, const uint8_t* __restrict__ mask, const float2* __restrict__ uv,
               u64* __restrict__ slc, u64* __restrict__ slt, u64* __restrict__ work,
               const uint32_t* __restrict__ order, uint16_t* __restrict__ item_steps) {
    const u64 item = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    LaneCount c{0ull, 0ull};
    Acc acc{0u, 0u, 0ull};
    const FieldGrid G = grid_of(p, f);
    if (item < n_items) {
        FieldLane s;
        FieldStart st;
        s.alive = false;
        s.n = 0;
        s.item = (uint32_t)item;
        if (start_of<FORM>(st, item, seed_begin, seeds, order, mask, p, G.g))
            field_begin<FORM>(s, st, p, G, acc, slc, slt);
        c.ntraj = 1;
        while (s.alive) {
            field_step<ORDER, FORM, false, false>(s, mask, uv, p, k, G, acc, slc, slt);
        }
        record_end<RECORD>(s, item_steps);
        count_trajectory(c, s);
        acc_flush(acc, slc, slt);
    }
    warp_add_counters(c.steps, c.ntraj, work);
}

// The loop of a persistent warp: take trajectories from the queue (its head,
// work[0], must be 0 at launch), start them on idle lanes, advance every live
// one step by step until refill_min lanes (all, once nothing is left to start)
// are idle.  Each trajectory ends within max_n_steps steps, so the loops end;
// their tests are warp-uniform.
//   prepare(item, st)  form the start of queue item `item`, false if it has none
//   place(st)          make the lane's grid that of st
//
// Starts are formed 32 at a time, by all lanes, into a stash in shared memory
// that idle lanes draw on: a start costs half a step's instructions and four
// dependent loads, and formed by the two to four idle lanes it cost the warp as
// much as by 32 (2.8 steps' time, every 15 steps, where a trajectory is 122
// steps long).  Near the end of the queue (four trajectories a lane left, more
// than all the stashes hold) a warp takes only as many as it has idle lanes, so
// that none waits in one warp's stash while another's lanes idle: with one or
// two a lane 256^2 hills take 6.8 ms, not 6.2.
//
// The stepping is a loop of its own, closed by one vote, and its lanes step
// together (field_step), so that it has no branch that could diverge but for
// the rare one.  Measured, with the stash 2 lanes idle at a refill, without 4:
// 4096^2 fan terrain, RK4 (122 steps a trajectory): 289 -> 274 ms; odd incised
// relief, RK4 (92): 43.7 -> 41.3 ms; 256^2 hills, RK2 (880): 6.5 -> 6.2 ms; 24
// tiles, RK2 (740): 104 -> 94.5 ms (make_fast_geo's wider interior included).
template <int ORDER, bool RECORD, int FORM, bool GATED, class Prepare, class Place>
__device__ __forceinline__ void field_loop(FieldLane& s, LaneCount& c, Acc& acc, FieldGrid& G, u64 n_items,
                                           uint32_t refill_min, const slm_params& p, const FastConst& k,
                                           const uint8_t* __restrict__ mask, const float2* __restrict__ uv,
                                           u64* __restrict__ slc, u64* __restrict__ slt, u64* __restrict__ work,
                                           uint16_t* __restrict__ item_steps, Prepare prepare, Place place) {
    __shared__ FieldStart stashes[256 / 32][32];
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    FieldStart* stash = stashes[threadIdx.x >> 5];
    const u64 plenty = 4ull * gridDim.x * blockDim.x;
    unsigned live = 0, held = 0;  // lanes on a trajectory; starts in the stash
    bool drained = false, bulk = n_items > plenty;
    while (true) {
        // here at least refill_min lanes are idle
        if (held != 0u || !drained) {
            const unsigned idle = ~live;
            if (held == 0u) {
                const unsigned want = bulk ? 32u : (unsigned)__popc(idle);
                u64 head = 0;
                if (lane == 0u) head = atomicAdd(work, (u64)want);
                head = __shfl_sync(FULL, head, 0);
                drained = head + want >= n_items;
                bulk = head + want + plenty < n_items;
                const u64 item = head + lane;
                FieldStart st;
                bool ok = false;
                if (lane < want && item < n_items) {
                    c.ntraj++;
                    ok = prepare(item, st);
                    if (RECORD && !ok) item_steps[item] = 0;
                }
                const unsigned ready = __ballot_sync(FULL, ok);
                if (ok) stash[__popc(ready & below)] = st;
                held = __popc(ready);
                __syncwarp();
            }
            const unsigned rank = __popc(idle & below);
            if (!s.alive && rank < held) {
                const FieldStart st = stash[held - 1u - rank];
                place(st);
                count_trajectory(c, s);
                field_begin<FORM>(s, st, p, G, acc, slc, slt);
                if (RECORD && !s.alive) record_end<RECORD>(s, item_steps);
            }
            __syncwarp();  // the stash is read before it is written again
            held -= min(held, (unsigned)__popc(idle));
            live = __ballot_sync(FULL, s.alive);
            if ((held != 0u || !drained) && (uint32_t)__popc(~live) >= refill_min) continue;
        }
        if (live == 0u) break;
        const int keep = held == 0u && drained ? 0 : 32 - (int)refill_min;
        do {
            if (FORM) {
                const bool on = s.alive;
                field_step<ORDER, FORM, GATED, true>(s, mask, uv, p, k, G, acc, slc, slt);
                if (RECORD && on && !s.alive) record_end<RECORD>(s, item_steps);
            } else if (s.alive) {
                field_step<ORDER, FORM, GATED, false>(s, mask, uv, p, k, G, acc, slc, slt);
                if (RECORD && !s.alive) record_end<RECORD>(s, item_steps);
            }
            live = __ballot_sync(FULL, s.alive);
        } while (__popc(live) > keep);
    }
}

// After the loop: the lanes' last runs and counts.
__device__ __forceinline__ void field_end(FieldLane& s, LaneCount& c, Acc& acc, u64* slc, u64* slt, u64* work) {
    count_trajectory(c, s);
    acc_flush(acc, slc, slt);
    warp_add_counters(c.steps, c.ntraj, work);
}

template <int ORDER, bool RECORD, int FORM>
__global__ void __launch_bounds__(256, FIELD_BLOCKS)
k_fields_persistent(const __grid_constant__ slm_params p, const __grid_constant__ FastGeo f,
                    const __grid_constant__ FastConst k, const float2* __restrict__ seeds, uint32_t seed_begin,
                    u64 n_items, const uint8_t* __restrict__ mask, const float2* __restrict__ uv,
                    u64* __restrict__ slc, u64* __restrict__ slt, u64* __restrict__ work,
                    const uint32_t* __restrict__ order, uint16_t* __restrict__ item_steps,
                    uint32_t refill_min) {
    FieldGrid G = grid_of(p, f);
    FieldLane s{};
    Acc acc{0u, 0u, 0ull};
    LaneCount c{0ull, 0ull};
    field_loop<ORDER, RECORD, FORM, false>(
        s, c, acc, G, n_items, refill_min, p, k, mask, uv, slc, slt, work, item_steps,
        [&](u64 item, FieldStart& st) { return start_of<FORM>(st, item, seed_begin, seeds, order, mask, p, G.g); },
        [](const FieldStart&) {});
    field_end(s, c, acc, slc, slt, work);
}

// ------------------------------------------------------------------ both directions
// Both directions of one grid in one persistent launch: queue items
// [0, n) trace downstream, [n, 2n) upstream, so the long trajectories that end
// one direction run alongside the other direction's bulk instead of as its
// own tail.  A lane keeps its trajectory's COMBO_FACTOR (the only per-
// direction value of the step) and its accumulator offset (0, or up_stride
// for the upstream slc/slt); every trajectory is the single-direction
// kernels'.
template <int ORDER, int FORM>
__global__ void __launch_bounds__(256, FIELD_BLOCKS)
k_fields_pair(const __grid_constant__ slm_params p, const __grid_constant__ FastGeo f,
              const __grid_constant__ FastConst k, float cf_up, const float2* __restrict__ seeds,
              uint32_t seed_begin, u64 n_items, const uint8_t* __restrict__ mask, const float2* __restrict__ uv,
              u64* __restrict__ slc, u64* __restrict__ slt, uint32_t up_stride, u64* __restrict__ work,
              const uint32_t* __restrict__ order, const uint32_t* __restrict__ order_up,
              uint32_t refill_min) {
    FieldGrid G = grid_of(p, f);
    const float cf_down = G.g.cf;
    FieldLane s{};
    Acc acc{0u, 0u, 0ull};
    LaneCount c{0ull, 0ull};
    u64 steps_up = 0;
    field_loop<ORDER, false, FORM, false>(
        s, c, acc, G, 2 * n_items, refill_min, p, k, mask, uv, slc, slt, work, nullptr,
        [&](u64 item, FieldStart& st) {
            const bool up = item >= n_items;
            st.tag = up;
            return start_of<FORM>(st, up ? item - n_items : item, seed_begin, seeds, up ? order_up : order, mask, p,
                                  G.g);
        },
        [&](const FieldStart& st) {
            if (G.acc_offset) steps_up += s.n;
            G.acc_offset = st.tag ? up_stride : 0u;
            G.g.cf = st.tag ? cf_up : cf_down;
        });
    if (G.acc_offset) steps_up += s.n;
    field_end(s, c, acc, slc, slt, work);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) steps_up += __shfl_xor_sync(0xffffffffu, steps_up, o);
    if ((threadIdx.x & 31u) == 0u) atomicAdd(work + 3, steps_up);
}

// ------------------------------------------------------------------ batched tiles
// Last tile whose first seed is <= x (tiles sorted by seed_begin; the host
// checks the table), found by binary search over the L1-cached table.
__device__ __forceinline__ uint32_t find_tile(const slm_tile* __restrict__ tiles, uint32_t n_tiles,
                                              uint32_t x) {
    uint32_t lo = 0, hi = n_tiles;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&tiles[mid].seed_begin) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Many grids (DTM tiles of any sizes) in one persistent launch.  The queue
// runs over every trajectory of every tile; a lane that takes an item looks up
// its tile and keeps the tile's geometry (Geo) and pixel base with its
// trajectory, so lanes of one warp may trace different tiles.  Each
// trajectory is computed exactly as a single-grid launch on its tile computes
// it (RNG stream of the tile-local seed index).  work[3] receives 1 if a seed
// falls outside its tile's range (an inconsistent table).
template <int ORDER, bool RECORD, int FORM>
__global__ void __launch_bounds__(256, FIELD_BLOCKS)
k_fields_batched(const __grid_constant__ slm_params p, const __grid_constant__ FastConst k, const slm_tile* __restrict__ tiles, uint32_t n_tiles,
                 const float2* __restrict__ seeds, u64 n_items, const uint8_t* __restrict__ mask,
                 const float2* __restrict__ uv, u64* __restrict__ slc, u64* __restrict__ slt,
                 u64* __restrict__ work, const uint32_t* __restrict__ order,
                 uint16_t* __restrict__ item_steps, uint32_t refill_min) {
    const uint32_t dd = p.subpixel_seed_point_density * p.subpixel_seed_point_density;
    FieldLane s{};
    FieldGrid G{make_geo(2u, 2u, 0.0f, 0.0f, 1.0f), make_fast_geo(2u, 2u, 1.0f, 1.0f, 0.0f, 0u), 0u, 0u};
    Acc acc{0u, 0u, 0ull};
    LaneCount c{0ull, 0ull};
    const auto tile_geo = [&](const slm_tile& T) {
        return make_geo(__ldg(&T.nx_padded), __ldg(&T.ny_padded), __ldg(&T.combo_factor), __ldg(&T.dt_max),
                        __ldg(&T.grid_scale));
    };
    field_loop<ORDER, RECORD, FORM, true>(
        s, c, acc, G, n_items, refill_min, p, k, mask, uv, slc, slt, work, item_steps,
        [&](u64 item, FieldStart& st) {
            uint32_t pos, sub;
            split_item(item, dd, pos, sub);
            const uint32_t seed = order ? __ldg(order + pos) : pos;
            st.item = (uint32_t)item;
            st.tag = find_tile(tiles, n_tiles, seed);
            const slm_tile& T = tiles[st.tag];
            const uint32_t local = seed - __ldg(&T.seed_begin);
            if (local >= __ldg(&T.n_seeds)) {
                atomicOr(reinterpret_cast<unsigned long long*>(work + 3), 1ull);
                return false;
            }
            return start_at<FORM>(st, __ldg(seeds + seed), local, sub, mask, p, tile_geo(T),
                                  (uint32_t)__ldg(&T.grid_offset));
        },
        [&](const FieldStart& st) {
            const slm_tile& T = tiles[st.tag];
            G.g = tile_geo(T);
            G.base = (uint32_t)__ldg(&T.grid_offset);
            if (FORM) {
                G.f = make_fast_geo(G.g.nxp, G.g.nyp, G.g.gs, G.g.dt_max, p.adjusted_max_error, G.base);
                // a tile the fast step cannot take has no interior pixel
                if (!fast_grid(G.g.nxp, G.g.nyp, G.base, G.g.cf, G.g.dt_max, p.trajectory_resolution))
                    G.f.rx = -1.0f;
            }
        });
    field_end(s, c, acc, slc, slt, work);
}

// ------------------------------------------------------------------ trajectories
__device__ __forceinline__ float edge_dt(float x, float u) {
    float dt = 0.0f;
    const float right = __fdiv_rn((float)__float2int_rz(x + 1.5f) - (x + 0.5f), u);
    const float left = __fdiv_rn(-((x + 0.5f) - (float)__float2int_rz(x + 0.5f)), u);
    if (u > 0.0f) dt = right;
    if (u < 0.0f) dt = left;
    return dt;
}

__device__ __forceinline__ float min_mag(float x, float y) {
    if (fabsf(x) < fabsf(y)) return x;
    if (fabsf(y) < fabsf(x)) return y;
    return fminf(x, y);
}

__device__ __forceinline__ void put_step(int8_t* rec, uint32_t n, float dx, float dy, float res) {
    const uint32_t lo = (uint8_t)cvt_i8(dx * res), hi = (uint8_t)cvt_i8(dy * res);
    reinterpret_cast<uint16_t*>(rec)[n] = (uint16_t)(lo | (hi << 8));
}

// One warp a block, with a walk_share of the trajectories: the launch is bound by
// the latency of its longest walk's steps, one after another.  1000 trajectories
// of 2000 RK2 steps at most, each way: 32 to a warp 2.29 ms, one 1.86 ms.
constexpr unsigned TRAJ_BLOCK = 32;

// trajectory_record (trajectory.cl:41-80) with runge_kutta_step_record and
// euler_step_record (rungekutta.cl:49-120)
template <int ORDER>
__global__ void __launch_bounds__(TRAJ_BLOCK)
k_trajectory(const __grid_constant__ slm_params p, const __grid_constant__ WalkGrid wg, uint32_t n_chunk,
             uint32_t per_warp, const float2* __restrict__ seeds,
             const uint8_t* __restrict__ mask, const float2* __restrict__ uv,
             int8_t* __restrict__ traj, uint16_t* __restrict__ nsteps_out,
             float* __restrict__ length_out) {
    const uint64_t item = (uint64_t)blockIdx.x * per_warp + threadIdx.x;
    if (threadIdx.x >= per_warp || item >= n_chunk) return;
    const uint32_t g = (uint32_t)item;
    const uint32_t seed_idx = p.seeds_chunk_offset + g;
    if (seed_idx >= p.n_seed_points) return;
    int8_t* rec = traj + 2ull * g * p.max_n_steps;
    const float res = (float)p.trajectory_resolution;
    const float2 c = __ldg(seeds + seed_idx);
    Vec2 a{c.x, c.y}, prev = a;
    uint32_t n = 0;
    float l = 0.0f, dt = p.dt_max;
    uint32_t idx = pixel_of(a, p);
    while (!__ldg(mask + idx) && (l < p.max_length && n < p.max_n_steps)) {
        const Step st = plain_step<ORDER>(a, dt, uv, p, wg);
        idx = st.idx;
        if (!__ldg(mask + idx)) {
            float dl = step_length(st.d2, wg);
            if (dl < p.integration_halt_threshold) {
                a.x = a.x + st.d1.x;
                a.y = a.y + st.d1.y;
                dl = step_length(st.d1, wg);
                idx = pixel_of(a, p);
            } else {
                a = st.next;
            }
            const bool stuck = dl < p.integration_halt_threshold;
            if (!stuck) dt = walk_dt(st.d2.x - st.d1.x, st.d2.y - st.d1.y, dt, p, wg);
            l = l + dl;
            put_step(rec, n, a.x - prev.x, a.y - prev.y, res);
            n++;
            if (stuck) break;
            prev = a;
        } else {
            // DOWNUP_SIGN is an unsigned literal: upstream it widens to 4294967296.0f
            const float sg = __uint2float_rn(p.downup_sign);
            const float sx = st.u1.x * sg, sy = st.u1.y * sg;
            const float dtx = edge_dt(a.x, sx), dty = edge_dt(a.y, sy);
            dt = min_mag(dtx, dty);
            a.x = a.x + sx * dt;
            a.y = a.y + sy * dt;
            a.x = quant(a.x, res);
            a.y = quant(a.y, res);
            a.x = fminf(fmaxf(a.x, -0.5f), p.nxf_mp5);
            a.y = fminf(fmaxf(a.y, -0.5f), p.nyf_mp5);
            const float dl = vlen(a.x - prev.x, a.y - prev.y);
            l = l + dl;
            put_step(rec, n, a.x - prev.x, a.y - prev.y, res);
            n++;
            break;
        }
    }
    nsteps_out[g] = (uint16_t)n;
    length_out[g] = l;
}

// ------------------------------------------------------------------ finish
// Fields.integrate's host arithmetic on the raw sums (fields.py:146-167 and
// :293-310), in NumPy's promotion order: per pixel and direction
//   slc  (uint32 wrap of the sum, or float64 of it when exact)
//   slt  float32(slt)                    (exact: float32(float64(sum)))
//   sla  float32(float64(sqrt 2) * slt / slc)       where slc > 0, else 0
//   slt  float32(float64(slt) / d^2)                where slc > 0
//   slt  float32(slt * ds_scale[dir]),  slt = sqrt(slt)
//   slc  sqrt 2 * pow(slc / d^2, 2/3)   (float64; table[slc] when given)
// Outputs are [nxy][2] (direction innermost), as the (nxp, nyp, 2) arrays.
__global__ void k_fields_finish(const u64* __restrict__ acc, uint32_t nxy, uint32_t dd, double ds0,
                                double ds1, int exact, const double* __restrict__ table,
                                uint32_t table_len, double* __restrict__ slc_out,
                                float* __restrict__ slt_out, float* __restrict__ sla_out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nxy) return;
    const double sqrt2 = 1.4142135623730951;  // np.sqrt(2.0), correctly rounded
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const u64 c64 = acc[(size_t)(2 * d) * nxy + i];
        const u64 t64 = acc[(size_t)(2 * d + 1) * nxy + i];
        double c;
        float t;
        if (exact) {
            c = (double)c64;
            t = (float)(double)t64;
        } else {
            c = (double)(uint32_t)c64;
            t = (float)(uint32_t)t64;
        }
        float a = 0.0f;
        if (c > 0.0) {
            a = (float)((sqrt2 * (double)t) / c);
            t = (float)((double)t / (double)dd);  // d^2 is a uint32 scalar: float64 division
        }
        t = (float)((double)t * (d == 0 ? ds0 : ds1));
        t = sqrtf(t);
        double f;
        if (table && c < (double)table_len) f = table[(uint32_t)c];
        else f = sqrt2 * pow(c / (double)dd, 2.0 / 3.0);
        slc_out[2 * (size_t)i + d] = f;
        slt_out[2 * (size_t)i + d] = t;
        sla_out[2 * (size_t)i + d] = a;
    }
}

}  // namespace slm

using namespace slm;

// The form of a single-grid launch's steps: STEP_GENERAL where the grid is not
// one for step_fast.
static StepForm form_of(const slm_params& p) {
    return fast_grid(p.nx_padded, p.ny_padded, 0u, p.combo_factor, p.dt_max, p.trajectory_resolution)
               ? jittered_form(p)
               : STEP_GENERAL;
}

static FastGeo fast_geo_of(const slm_params& p) {
    return make_fast_geo(p.nx_padded, p.ny_padded, p.grid_scale, p.dt_max, p.adjusted_max_error, 0u);
}

// Resident blocks per SM of a persistent launch: the caller's, else as many as fit.
static int blocks_per_sm(const slm_launch& L, const void* kernel, int block, int* out) {
    *out = L.blocks_per_sm;
    if (*out <= 0) {
        int occ = 0;
        SLM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, block, 0));
        *out = occ > 0 ? occ : 1;
    }
    return SLM_OK;
}

static int check_grid(const slm_params* p) {
    SLM_REQUIRE(p != nullptr, "params is NULL");
    SLM_REQUIRE(p->nx_padded >= 2 && p->ny_padded >= 2, "grid too small: %u x %u",
                p->nx_padded, p->ny_padded);
    SLM_REQUIRE((u64)p->nx_padded * p->ny_padded == p->nxy_padded,
                "nxy_padded %u != nx_padded*ny_padded", p->nxy_padded);
    SLM_REQUIRE(p->trajectory_resolution > 0, "trajectory_resolution is 0");
    return SLM_OK;
}

// slm_launch.chunk: a warp starts trajectories once at least this many of its
// lanes are idle (or all are); 0 selects 2.  Measured with 1, 2, 3, 4: 274.9,
// 273.5, 276.2, 278 ms for 4096^2 fan terrain, RK4, where a trajectory ends every
// fourth step of a warp; within 1 % of one another where they are longer.
static uint32_t refill_min(const slm_launch& L) {
    if (L.chunk == 0) return 2u;
    return L.chunk <= 1 ? 1u : (L.chunk >= 32 ? 32u : (uint32_t)L.chunk);
}

template <int ORDER, bool RECORD, int FORM>
static int launch_fields(const slm_params* p, const slm_launch& L, int block, const float2* sp,
                         uint32_t begin, u64 n_items, const uint8_t* mask, const float2* u2, u64* slc,
                         u64* slt, u64* work, const uint32_t* order, uint16_t* rec, cudaStream_t s) {
    if (L.schedule == SLM_SCHED_PLAIN) {
        const u64 grid = (n_items + block - 1) / block;
        SLM_REQUIRE(grid < (1ull << 31), "too many trajectories for one launch");
        k_fields_plain<ORDER, RECORD, FORM><<<(unsigned)grid, block, 0, s>>>(*p, fast_geo_of(*p), make_fast_const(*p), sp, begin, n_items, mask, u2,
                                                                            slc, slt, work, order, rec);
        SLM_LAUNCHED("k_fields_plain");
    } else if (L.schedule == SLM_SCHED_PERSISTENT) {
        int per_sm = 0;
        const int rc = blocks_per_sm(L, (const void*)k_fields_persistent<ORDER, RECORD, FORM>, block, &per_sm);
        if (rc) return rc;
        const unsigned grid = (unsigned)(num_sms() * per_sm);
        k_fields_persistent<ORDER, RECORD, FORM><<<grid, block, 0, s>>>(*p, fast_geo_of(*p), make_fast_const(*p), sp, begin, n_items, mask, u2, slc, slt,
                                                                        work, order, rec, refill_min(L));
        SLM_LAUNCHED("k_fields_persistent");
    } else {
        set_error("unknown schedule %d", L.schedule);
        return SLM_ERR_ARGS;
    }
    return SLM_OK;
}

template <int ORDER, bool RECORD, int FORM>
static int launch_batched(const slm_params* p, const slm_launch& L, int block, const slm_tile* tiles,
                          uint32_t n_tiles, const float2* sp, u64 n_items, const uint8_t* mask,
                          const float2* u2, u64* slc, u64* slt, u64* work, const uint32_t* order,
                          uint16_t* rec, cudaStream_t s) {
    int per_sm = 0;
    const int rc = blocks_per_sm(L, (const void*)k_fields_batched<ORDER, RECORD, FORM>, block, &per_sm);
    if (rc) return rc;
    const unsigned grid = (unsigned)(num_sms() * per_sm);
    k_fields_batched<ORDER, RECORD, FORM><<<grid, block, 0, s>>>(*p, make_fast_const(*p), tiles, n_tiles, sp, n_items, mask, u2, slc, slt,
                                                                work, order, rec, refill_min(L));
    SLM_LAUNCHED("k_fields_batched");
    return SLM_OK;
}

// f<ORDER, RECORD, FORM>(...) for run-time values of the three
#define SLM_FORM_DISPATCH(f, order, record, form, ...)                     \
    ((form) == STEP_JITTERED ? f<order, record, STEP_JITTERED>(__VA_ARGS__) \
     : (form) == STEP_FAINT  ? f<order, record, STEP_FAINT>(__VA_ARGS__)    \
                             : f<order, record, STEP_GENERAL>(__VA_ARGS__))
#define SLM_FIELDS_DISPATCH(f, rk4, record, form, ...)                          \
    ((rk4) ? ((record) ? SLM_FORM_DISPATCH(f, 4, true, form, __VA_ARGS__)        \
                       : SLM_FORM_DISPATCH(f, 4, false, form, __VA_ARGS__))      \
           : ((record) ? SLM_FORM_DISPATCH(f, 2, true, form, __VA_ARGS__)        \
                       : SLM_FORM_DISPATCH(f, 2, false, form, __VA_ARGS__)))

extern "C" {

size_t slm_fields_workspace_words(void) { return 4; }

int slm_integrate_fields(const slm_params* p, const slm_launch* launch, const float* seed_point,
                         const uint8_t* mask, const float* uv, uint32_t* mapping, uint64_t* slc,
                         uint64_t* slt, uint64_t* workspace, void* stream) {
    return slm_integrate_fields_scheduled(p, launch, seed_point, mask, uv, mapping, slc, slt,
                                          workspace, nullptr, nullptr, stream);
}

int slm_integrate_fields_scheduled(const slm_params* p, const slm_launch* launch,
                                   const float* seed_point, const uint8_t* mask, const float* uv,
                                   uint32_t* mapping, uint64_t* slc, uint64_t* slt,
                                   uint64_t* workspace, const uint32_t* seed_order,
                                   uint16_t* item_steps, void* stream) {
    (void)mapping;
    clear_error();
    int rc = check_grid(p);
    if (rc) return rc;
    SLM_REQUIRE(seed_point && mask && uv && slc && slt && workspace, "NULL buffer");
    SLM_REQUIRE(aligned(uv, 8) && aligned(seed_point, 8), "uv/seed_point must be 8-byte aligned");
    SLM_REQUIRE(aligned(slc, 8) && aligned(slt, 8) && aligned(workspace, 8),
                "slc/slt/workspace must be 8-byte aligned");
    SLM_REQUIRE(p->subpixel_seed_point_density >= 1, "subpixel_seed_point_density is 0");
    slm_launch def{SLM_SCHED_PERSISTENT, SLM_RK2, 256, 0, 0, {0, 0, 0}};
    const slm_launch& L = launch ? *launch : def;
    SLM_REQUIRE(L.integrator == SLM_RK2 || L.integrator == SLM_RK4, "integrator must be 2 or 4");
    const int block = L.block_threads > 0 ? L.block_threads : 256;
    SLM_REQUIRE(block % 32 == 0 && block <= 256, "block_threads must be a multiple of 32, <= 256");
    cudaStream_t s = (cudaStream_t)stream;
    SLM_CUDA(cudaMemsetAsync(workspace, 0, slm_fields_workspace_words() * sizeof(uint64_t), s));
    const uint32_t begin = p->seeds_chunk_offset;
    if (begin >= p->n_seed_points) return SLM_OK;
    const u64 dd = (u64)p->subpixel_seed_point_density * p->subpixel_seed_point_density;
    const u64 n_items = (u64)(p->n_seed_points - begin) * dd;
    SLM_REQUIRE(!item_steps || n_items < (1ull << 32), "step recording needs fewer than 2^32 trajectories");
    const float2* sp = reinterpret_cast<const float2*>(seed_point);
    const float2* u2 = reinterpret_cast<const float2*>(uv);
    u64* w = (u64*)workspace;
    return SLM_FIELDS_DISPATCH(launch_fields, L.integrator == SLM_RK4, item_steps != nullptr, form_of(*p), p, L, block,
                               sp, begin, n_items, mask, u2, (u64*)slc, (u64*)slt, w, seed_order, item_steps, s);
}

int slm_integrate_fields_pair(const slm_params* p_down, const slm_params* p_up, const slm_launch* launch,
                              const float* seed_point, const uint8_t* mask, const float* uv, uint64_t* slc,
                              uint64_t* slt, uint64_t up_stride, uint64_t* workspace, const uint32_t* seed_order,
                              const uint32_t* seed_order_up, void* stream) {
    clear_error();
    int rc = check_grid(p_down);
    if (rc) return rc;
    SLM_REQUIRE(p_up != nullptr, "params is NULL");
    // the two parameter blocks may differ only in the direction
    SLM_REQUIRE(p_up->nxy_padded == p_down->nxy_padded && p_up->nx_padded == p_down->nx_padded &&
                p_up->n_seed_points == p_down->n_seed_points &&
                p_up->seeds_chunk_offset == p_down->seeds_chunk_offset &&
                p_up->subpixel_seed_point_density == p_down->subpixel_seed_point_density &&
                p_up->max_n_steps == p_down->max_n_steps && p_up->max_length == p_down->max_length &&
                p_up->dt_max == p_down->dt_max && p_up->grid_scale == p_down->grid_scale &&
                p_up->combo_factor == -p_down->combo_factor,
                "downstream and upstream parameters differ in more than the direction");
    SLM_REQUIRE(seed_point && mask && uv && slc && slt && workspace, "NULL buffer");
    SLM_REQUIRE(aligned(uv, 8) && aligned(seed_point, 8), "uv/seed_point must be 8-byte aligned");
    SLM_REQUIRE(aligned(slc, 8) && aligned(slt, 8) && aligned(workspace, 8),
                "slc/slt/workspace must be 8-byte aligned");
    SLM_REQUIRE(up_stride >= p_down->nxy_padded && up_stride + p_down->nxy_padded < (1ull << 32),
                "up_stride must be >= nxy_padded and leave the upstream arrays below 2^32 elements");
    SLM_REQUIRE(p_down->subpixel_seed_point_density >= 1, "subpixel_seed_point_density is 0");
    slm_launch def{SLM_SCHED_PERSISTENT, SLM_RK2, 256, 0, 0, {0, 0, 0}};
    const slm_launch& L = launch ? *launch : def;
    SLM_REQUIRE(L.schedule == SLM_SCHED_PERSISTENT, "the pair form runs the persistent schedule");
    SLM_REQUIRE(L.integrator == SLM_RK2 || L.integrator == SLM_RK4, "integrator must be 2 or 4");
    const int block = L.block_threads > 0 ? L.block_threads : 256;
    SLM_REQUIRE(block % 32 == 0 && block <= 256, "block_threads must be a multiple of 32, <= 256");
    cudaStream_t s = (cudaStream_t)stream;
    SLM_CUDA(cudaMemsetAsync(workspace, 0, slm_fields_workspace_words() * sizeof(uint64_t), s));
    const uint32_t begin = p_down->seeds_chunk_offset;
    if (begin >= p_down->n_seed_points) return SLM_OK;
    const u64 dd = (u64)p_down->subpixel_seed_point_density * p_down->subpixel_seed_point_density;
    const u64 n_items = (u64)(p_down->n_seed_points - begin) * dd;
    const float2* sp = reinterpret_cast<const float2*>(seed_point);
    const float2* u2 = reinterpret_cast<const float2*>(uv);
    const bool rk4 = L.integrator == SLM_RK4;
    const StepForm form = form_of(*p_down);
    const auto kernel = form == STEP_JITTERED ? (rk4 ? k_fields_pair<4, STEP_JITTERED> : k_fields_pair<2, STEP_JITTERED>)
                        : form == STEP_FAINT  ? (rk4 ? k_fields_pair<4, STEP_FAINT> : k_fields_pair<2, STEP_FAINT>)
                                              : (rk4 ? k_fields_pair<4, STEP_GENERAL> : k_fields_pair<2, STEP_GENERAL>);
    int per_sm = 0;
    rc = blocks_per_sm(L, (const void*)kernel, block, &per_sm);
    if (rc) return rc;
    const unsigned grid = (unsigned)(num_sms() * per_sm);
    const uint32_t* o_up = seed_order_up ? seed_order_up : seed_order;
    kernel<<<grid, block, 0, s>>>(*p_down, fast_geo_of(*p_down), make_fast_const(*p_down), p_up->combo_factor, sp, begin, n_items, mask, u2, (u64*)slc, (u64*)slt,
                                  (uint32_t)up_stride, (u64*)workspace, seed_order, o_up, refill_min(L));
    SLM_LAUNCHED("k_fields_pair");
    return SLM_OK;
}

int slm_integrate_fields_batched(const slm_params* p, const slm_launch* launch, const slm_tile* tiles,
                                 uint32_t n_tiles, uint32_t n_seeds, const float* seed_point,
                                 const uint8_t* mask, const float* uv, uint64_t* slc, uint64_t* slt,
                                 uint64_t* workspace, const uint32_t* seed_order, uint16_t* item_steps,
                                 void* stream) {
    clear_error();
    SLM_REQUIRE(p != nullptr, "params is NULL");
    SLM_REQUIRE(tiles && n_tiles >= 1, "no tiles");
    SLM_REQUIRE(seed_point && mask && uv && slc && slt && workspace, "NULL buffer");
    SLM_REQUIRE(aligned(uv, 8) && aligned(seed_point, 8) && aligned(tiles, 8),
                "uv/seed_point/tiles must be 8-byte aligned");
    SLM_REQUIRE(aligned(slc, 8) && aligned(slt, 8) && aligned(workspace, 8),
                "slc/slt/workspace must be 8-byte aligned");
    SLM_REQUIRE(p->subpixel_seed_point_density >= 1, "subpixel_seed_point_density is 0");
    SLM_REQUIRE(p->trajectory_resolution > 0, "trajectory_resolution is 0");
    slm_launch def{SLM_SCHED_PERSISTENT, SLM_RK2, 256, 0, 0, {0, 0, 0}};
    const slm_launch& L = launch ? *launch : def;
    SLM_REQUIRE(L.schedule == SLM_SCHED_PERSISTENT, "batched tracing runs the persistent schedule");
    SLM_REQUIRE(L.integrator == SLM_RK2 || L.integrator == SLM_RK4, "integrator must be 2 or 4");
    const int block = L.block_threads > 0 ? L.block_threads : 256;
    SLM_REQUIRE(block % 32 == 0 && block <= 256, "block_threads must be a multiple of 32, <= 256");
    cudaStream_t s = (cudaStream_t)stream;
    SLM_CUDA(cudaMemsetAsync(workspace, 0, slm_fields_workspace_words() * sizeof(uint64_t), s));
    if (n_seeds == 0) return SLM_OK;
    const u64 dd = (u64)p->subpixel_seed_point_density * p->subpixel_seed_point_density;
    const u64 n_items = (u64)n_seeds * dd;
    SLM_REQUIRE(!item_steps || n_items < (1ull << 32), "step recording needs fewer than 2^32 trajectories");
    const float2* sp = reinterpret_cast<const float2*>(seed_point);
    const float2* u2 = reinterpret_cast<const float2*>(uv);
    u64* w = (u64*)workspace;
    return SLM_FIELDS_DISPATCH(launch_batched, L.integrator == SLM_RK4, item_steps != nullptr, jittered_form(*p), p, L, block,
                               tiles, n_tiles, sp, n_items, mask, u2, (u64*)slc, (u64*)slt, w, seed_order, item_steps, s);
}

int slm_fields_finish(const uint64_t* acc, uint32_t nxy_padded, uint32_t density, double ds_scale_down,
                      double ds_scale_up, int exact, const double* slc_table, uint32_t table_len,
                      double* slc_out, float* slt_out, float* sla_out, void* stream) {
    clear_error();
    if (nxy_padded == 0) return SLM_OK;
    SLM_REQUIRE(acc && slc_out && slt_out && sla_out, "NULL buffer");
    SLM_REQUIRE(density >= 1, "density is 0");
    SLM_REQUIRE(aligned(acc, 8) && aligned(slc_out, 8) && aligned(slt_out, 4) && aligned(sla_out, 4),
                "misaligned buffer");
    k_fields_finish<<<(nxy_padded + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        (const u64*)acc, nxy_padded, density * density, ds_scale_down, ds_scale_up, exact, slc_table,
        slc_table ? table_len : 0u, slc_out, slt_out, sla_out);
    SLM_LAUNCHED("k_fields_finish");
    return SLM_OK;
}

int slm_integrate_trajectory(const slm_params* p, int32_t integrator, uint32_t n_chunk,
                             const float* seed_point, const uint8_t* mask, const float* uv,
                             uint32_t* mapping, int8_t* trajectories, uint16_t* nsteps,
                             float* length, void* stream) {
    (void)mapping;
    clear_error();
    int rc = check_grid(p);
    if (rc) return rc;
    SLM_REQUIRE(integrator == SLM_RK2 || integrator == SLM_RK4, "integrator must be 2 or 4");
    if (n_chunk == 0) return SLM_OK;
    SLM_REQUIRE(seed_point && mask && uv && trajectories && nsteps && length, "NULL buffer");
    SLM_REQUIRE(aligned(uv, 8) && aligned(seed_point, 8), "uv/seed_point must be 8-byte aligned");
    SLM_REQUIRE(aligned(trajectories, 2) && aligned(nsteps, 2) && aligned(length, 4),
                "trajectory buffers misaligned");
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t per_warp = walk_share(n_chunk);
    const unsigned grid = (n_chunk + per_warp - 1) / per_warp;
    const WalkGrid wg = make_walk_grid(*p);
    const float2* sp = reinterpret_cast<const float2*>(seed_point);
    const float2* u2 = reinterpret_cast<const float2*>(uv);
    if (integrator == SLM_RK4)
        k_trajectory<4><<<grid, TRAJ_BLOCK, 0, s>>>(*p, wg, n_chunk, per_warp, sp, mask, u2, trajectories, nsteps, length);
    else
        k_trajectory<2><<<grid, TRAJ_BLOCK, 0, s>>>(*p, wg, n_chunk, per_warp, sp, mask, u2, trajectories, nsteps, length);
    SLM_LAUNCHED("k_trajectory");
    return SLM_OK;
}

}  // extern "C"

// ------------------------------------------------------------------ no-alloc variant
// Some callers cannot call cudaMalloc: a host application that hands a plugin
// only its own pre-allocated buffers, or a binding of the reference's
// six-buffer integrate_fields signature, which has no workspace argument.
// For them, slm_integrate_fields_noalloc keeps the field tracer's scratch (the
// work-queue head and the step/trajectory counters) in the file-scope device
// array below instead of a caller-allocated workspace.  The array is modest
// (SLM_NOALLOC_SCRATCH_WORDS 64-bit words, 512 bytes) and every GPU that loads
// this library holds it until the process exits.
namespace slm {

static __device__ __align__(256) unsigned long long g_noalloc_scratch[SLM_NOALLOC_SCRATCH_WORDS];

// Device address of g_noalloc_scratch in the current context.  In host code
// the array's name is only a host-side stand-in, so the address comes from
// cudaGetSymbolAddress.  It is looked up on every call (a cheap query) rather
// than cached: an address belongs to the context the module was loaded in, and
// a cached one would go stale after cudaDeviceReset or in a caller's own
// context.
static int noalloc_scratch(u64** out) {
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess) {
        int dev = -1;
        cudaGetDevice(&dev);
        set_error("cudaGetSymbolAddress(scratch) failed on device %d: %s", dev, cudaGetErrorString(e));
        return SLM_ERR_CUDA;
    }
    *out = static_cast<u64*>(ptr);
    return SLM_OK;
}

}  // namespace slm

extern "C" int slm_integrate_fields_noalloc(const slm_params* p, const slm_launch* launch,
                                            const float* seed_point, const uint8_t* mask,
                                            const float* uv, uint32_t* mapping, uint64_t* slc,
                                            uint64_t* slt, void* stream) {
    clear_error();
    const size_t need = slm_fields_workspace_words();
    if (need > SLM_NOALLOC_SCRATCH_WORDS) {
        set_error("field tracer needs %zu scratch words, the static array holds %d",
                  need, SLM_NOALLOC_SCRATCH_WORDS);
        return SLM_ERR_CAPACITY;
    }
    u64* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    // slm_integrate_fields clears the scratch words it uses (queue head and
    // counters) on the stream before its launch, so a previous call's contents
    // never leak into this one.
    return slm_integrate_fields(p, launch, seed_point, mask, uv, mapping, slc, slt,
                                reinterpret_cast<uint64_t*>(scratch), stream);
}

// ------------------------------------------------------------------ self-test
namespace slm {
// counts[0] += inputs whose div6 differs from the IEEE quotient (NaN equals
// NaN); counts[1] = the largest such input bit pattern + 1 (0: none)
__global__ void k_selftest_div6(u64* counts) {
    u64 bad = 0, last = 0;
    for (u64 b = (u64)blockIdx.x * blockDim.x + threadIdx.x; b < (1ull << 32); b += (u64)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((uint32_t)b);
        const float want = __fdiv_rn(x, 6.0f), got = div6(x);
        const bool same = __float_as_uint(want) == __float_as_uint(got) || (want != want && got != got);
        if (!same) {
            bad++;
            last = b + 1;
        }
    }
    if (bad) {
        atomicAdd(counts, bad);
        atomicMax(counts + 1, last);
    }
}
}  // namespace slm

// counts[0] += inputs whose cvt_i8 differs from the x86 conversion the
// reference's float -> char follows (cvttss2si: truncation in range, INT32_MIN
// for NaN and out of range; the low byte kept); counts[1] as for div6
__global__ void k_selftest_cvt_i8(u64* counts) {
    u64 bad = 0, last = 0;
    for (u64 b = (u64)blockIdx.x * blockDim.x + threadIdx.x; b < (1ull << 32); b += (u64)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((uint32_t)b);
        int32_t w = (int32_t)0x80000000;
        if (x >= -2147483648.0f && x < 2147483648.0f) w = __float2int_rz(x);
        if ((int8_t)(w & 0xff) != cvt_i8(x)) {
            bad++;
            last = b + 1;
        }
    }
    if (bad) {
        atomicAdd(counts, bad);
        atomicMax(counts + 1, last);
    }
}

// counts[0] += floats s from 2^-100 up for which unit_math.cuh could give a wrong
// root or quotient: the root is not the IEEE square root, or the reciprocal
// of the root or of a float next to it (a length whose square is s but for its
// low bits) breaks one of the two bounds there.  counts[1] as for div6
__global__ void k_selftest_unit(u64* counts) {
    u64 bad = 0, last = 0;
    for (u64 v = (u64)ROOT_MIN_BITS + (u64)blockIdx.x * blockDim.x + threadIdx.x; v <= ROOT_MAX_BITS;
         v += (u64)gridDim.x * blockDim.x) {
        const float s = __uint_as_float((uint32_t)v);
        const float y0 = rsqrt_estimate(s), root = root_from(s, y0);
        bool ok = root == __fsqrt_rn(s);
        for (int k = -1; k <= 1; ++k) {
            const float len = __uint_as_float(__float_as_uint(root) + (uint32_t)k);
            const float y = reciprocal_from(len, y0);
            const double b = (double)__uint_as_float((__float_as_uint(len) & 0x7fffffu) | 0x3f800000u);
            const double d = fabs((double)y * (double)len - 1.0);
            ok = ok && d * (b + 0x1p-23) < 0x1p-23 && d <= 0x1p-25 * b * (1.0 + 0x1p-18);
        }
        if (!ok) {
            bad++;
            last = v + 1;
        }
    }
    if (bad) {
        atomicAdd(counts, bad);
        atomicMax(counts + 1, last);
    }
}

// a float in [1/2, 8) of either sign from a hash of x
__device__ __forceinline__ float hashed_float(uint32_t x) {
    x = (x ^ (x >> 16)) * 0x7feb352du;
    x = (x ^ (x >> 15)) * 0x846ca68bu;
    x ^= x >> 16;
    return __uint_as_float((x & 0x807fffffu) | (((x >> 23 & 3u) + 126u) << 23));
}

// counts[0] += pairs of a * b + c for which the packed product and sum are not
// the scalar ones, counts[1] += pairs for which a fused operation is not
__global__ void k_selftest_packed(const __grid_constant__ FastConst k, u64* counts) {
    const uint32_t i = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    const float a = hashed_float(i), b = hashed_float(i + 1u), c = hashed_float(i + 2u), d = hashed_float(i + 3u);
    const float x = __fadd_rn(__fmul_rn(a, b), c), y = __fadd_rn(__fmul_rn(d, b), a);
    float px, py;
    unpack2(add2_product(mul2(pack2(a, d), pack2(b, b)), pack2(c, a), k), px, py);
    const unsigned bad = __ballot_sync(0xffffffffu, px != x || py != y);
    const unsigned fused = __ballot_sync(0xffffffffu, __fmaf_rn(a, b, c) != x || __fmaf_rn(d, b, a) != y);
    if ((threadIdx.x & 31u) == 0u) {
        if (bad) atomicAdd(counts, (u64)__popc(bad));
        if (fused) atomicAdd(counts + 1, (u64)__popc(fused));
    }
}

extern "C" int slm_selftest_packed(uint64_t* counts, void* stream) {
    clear_error();
    SLM_REQUIRE(counts && aligned(counts, 8), "counts must be two 8-byte aligned device words");
    cudaStream_t s = (cudaStream_t)stream;
    SLM_CUDA(cudaMemsetAsync(counts, 0, 2 * sizeof(uint64_t), s));
    slm_params p{};
    p.trajectory_resolution = 128;
    k_selftest_packed<<<1u << 16, 256, 0, s>>>(make_fast_const(p), (u64*)counts);
    SLM_LAUNCHED("k_selftest_packed");
    return SLM_OK;
}

extern "C" int slm_selftest_unit(uint64_t* counts, void* stream) {
    clear_error();
    SLM_REQUIRE(counts && aligned(counts, 8), "counts must be two 8-byte aligned device words");
    cudaStream_t s = (cudaStream_t)stream;
    SLM_CUDA(cudaMemsetAsync(counts, 0, 2 * sizeof(uint64_t), s));
    k_selftest_unit<<<(unsigned)(num_sms() * 8), 256, 0, s>>>((u64*)counts);
    SLM_LAUNCHED("k_selftest_unit");
    return SLM_OK;
}

extern "C" int slm_selftest_div6(uint64_t* counts, void* stream) {
    clear_error();
    SLM_REQUIRE(counts && aligned(counts, 8), "counts must be two 8-byte aligned device words");
    cudaStream_t s = (cudaStream_t)stream;
    SLM_CUDA(cudaMemsetAsync(counts, 0, 2 * sizeof(uint64_t), s));
    k_selftest_div6<<<(unsigned)(num_sms() * 8), 256, 0, s>>>((u64*)counts);
    SLM_LAUNCHED("k_selftest_div6");
    return SLM_OK;
}

extern "C" int slm_selftest_cvt_i8(uint64_t* counts, void* stream) {
    clear_error();
    SLM_REQUIRE(counts && aligned(counts, 8), "counts must be two 8-byte aligned device words");
    cudaStream_t s = (cudaStream_t)stream;
    SLM_CUDA(cudaMemsetAsync(counts, 0, 2 * sizeof(uint64_t), s));
    k_selftest_cvt_i8<<<(unsigned)(num_sms() * 8), 256, 0, s>>>((u64*)counts);
    SLM_LAUNCHED("k_selftest_cvt_i8");
    return SLM_OK;
}
