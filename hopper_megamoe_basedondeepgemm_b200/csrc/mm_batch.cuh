// The layer on one rank with more than a handful of routed rows, as one persistent sm_100a kernel of its own.
//
// With one rank nothing crosses NVLink, every SM can work out the whole routing by itself and rows need no flagged words:
//
//   routing  : every SM counts all routing entries per expert (one histogram per run of entries and warp), so the token
//              tiles and the task list follow without any exchange between SMs; the list of rows is made behind the first copies.
//   tiles    : an expert's rows form ceil(rows / tile limit) token tiles of at most 128 rows (96 with E4M3 tokens). The
//              block-scaled MMAs of a weight unit take 199 cycles for 16 rows and 288 for 128, so wide tiles are nearly free and an
//              expert's weights stream once per tile.
//   images   : SM (token mod G) copies its tokens' rows into the tiles' operand images in global memory (per streamed K
//              unit one record: the unit's 128 B of every row in the tensor core's swizzled order, then the unit's
//              scale planes), counted per tile; a task fetches the records with bulk copies.
//   GEMMs    : D[128 weight rows x N token rows] (N = the tile's rows, rounded up to 16), accumulators in TMEM. The epilogue
//              turns 16 tokens at a time through shared memory, so that all 128 threads of a group work whatever the row
//              count and a thread holds eight gate and eight up values of one token. Two groups take the tasks in turn.
//   order    : the L1 tasks dealt round-robin, but the last one to two rounds of them and all L2 tasks claimed one by one
//              (no tile is split along K, a slow SM takes fewer). L2 goes tile by tile, its last two or four tasks per SM
//              column block by column block. The weight ring runs ahead over the L1 -> L2 hand-over, so that the stream does not
//              stop there. (When this order came in: 59.2, 67.2 and 102 us with all L1 tasks dealt and L2 column by column, 57.2,
//              64.9 and 100 with it, for 13 and 64 tokens over 48 experts and 96 skewed ones from hidden states.)
//   combine  : per (token, 128-column block) behind a count per column block; routes added in slot order in fp32.
//
// Bound: HBM (the weights of the live experts once) up to about 40 rows per expert. 64 tokens, MXFP4, 48 experts (301 MB): 52 to 53.5 us a
// pass on different B200s, of which the stream is 42 at 7.1 TB/s; with four experts' weights in the place of all 48, which stay in the L2, 40. The
// multi-rank kernel takes 88. Beyond, no single thing: 512 tokens 76 to 79 us; 67 with weights from the L2 in the same way, 70 without the epilogue's
// arithmetic, 71 with a quarter of the MMAs, 72 with short records (76 without any of it, on the same GPU), and the power limit takes a tenth of
// the clock. With E4M3 tokens the units are widened into tensor memory (100 tokens: 67 to 70 us, 765 with the multi-rank kernel), and the clock is 5 % lower.
#pragma once
#include "mm_kernel.cuh"

namespace mm {

constexpr int kBMaxRows = 4096;                    // routed rows of one launch
constexpr uint32_t kBColumnTasks = 2;              // L2 tasks per SM that are claimed column block by column block, at least (`set_column_tiles`)
constexpr uint32_t kBAhead = 4;                    // K units that are asked into the L2 ahead, twice at the start of a launch
constexpr int kBAheadEntries = 2048;               // of at most so many routing entries (512 tokens of 8: 78.1 us without, 78.7 with; 256 57.2, 56.9)
constexpr int kBTaskRing = 64;                     // claimed tasks of one SM that some role has still to see, at most
constexpr int kBWStages = 12, kBRSlots = 12;       // at most: weight ring stages, token record slots
constexpr int kBServiceWarps = 4;                  // weight loader, MMA issuer, record loader, spare
constexpr int kBEpiWarps = 8;                      // two groups of four
constexpr int kBCombineWarps = 4;
constexpr int kBWorkWarps = kBEpiWarps + kBCombineWarps;    // warps 4..15 copy the rows into the images and list them
constexpr int kBRankWarps = kBServiceWarps + kBWorkWarps;   // warps 0..15 count the routing entries, a run of them each
constexpr int kBThreads = 32 * (kBServiceWarps + kBWorkWarps);
constexpr int kBExpWarps = 8;                      // E4M3 tokens: widening warps 12..19 (they take up the combine when their role ends)
constexpr int kBThreadsA8 = 32 * (kBServiceWarps + kBEpiWarps + kBExpWarps);
constexpr uint32_t kBVtStride = 152;               // floats between the tokens of `vt`
// tensor-memory columns with E4M3 tokens: scales of the weights and of the tokens (two areas of 8 each), widened units (two of 64)
constexpr uint32_t kTmScaleW = 256, kTmScaleX = 272, kTmWide = 384;
constexpr uint32_t kBBarEpi0 = 1, kBBarEpi1 = 2, kBBarWork = 3, kBBarTiles = 4, kBBarPlaced = 7;    // named barriers (5, 6: the decode kernel's)

struct BParams {
    int T, topk, E, H, I;
    int n1, n2, k1, k2;                            // weight tiles and K units of the two layers
    uint32_t unit_bytes, tile_limit;               // bytes of a streamed weight unit; rows of a token tile at most
    uint32_t x_row_bytes, x_sf_row_bytes, rx_row_bytes;
    int has_clamp, fast_math;
    float clamp, l1_scale, l2_scale, mid_gs, mid_gs_recip;         // (the reciprocal is 0 where `divide8` would not be exact)
    uint8_t* buf;
    const uint8_t* w1; const uint8_t* w2;
    __nv_bfloat16* y; int* stats;
    long long off_ctrl, off_x, off_x_sf, off_topk_idx, off_topk_w, off_rx, off_comb, off_token_tiles, off_mid_tiles, off_arrive;
    long long rx_region;
    uint32_t tile_capacity, cap_rows;              // token tiles the images, rows the receive pool and the images have room for
    long long off_routes, off_out;                 // [tokens][8] flagged routing records (launches from hidden states); [entries][H] bf16 expert outputs
    long long off_mid, off_mid_sf, off_parts;      // flagged words of the decode kernel: intermediate rows, their scale bytes, partial sums
    uint32_t mid_row_bytes;
    FeParams fe;
    uint32_t smem_ring;                            // bytes of dynamic shared memory for the two rings
    uint32_t column_tiles, column_tiles_long, column_long_from;    // tiles whose L2 tasks go column block by column block (batch kernel); the larger number from so many tiles on
    unsigned long long timeout_ns;
};

struct BShared {
    uint64_t wfull[kBWStages], wempty[kBWStages], rfull[kBRSlots], rempty[kBRSlots];
    uint64_t tmem_full[2], tmem_empty[2], xfull[2], xempty[2];
    uint32_t tmem_base, abort_flag, M, wissued, rissued, comb_next, comb_open, nw, nr, slot_bytes, spu, total, start_ok;
    uint32_t seg_shift;                            // routing entries of a run: 1 << seg_shift
    uint32_t cnt[kMaxLocalExperts], ebase[kMaxLocalExperts];
    uint32_t tile_e[kBMaxTiles];                   // expert
    uint32_t tile_row0[kBMaxTiles];                // first row (index into `rowf`)
    uint32_t tile_rows[kBMaxTiles];
    uint32_t tile_a16[kBMaxTiles];                 // 16-row groups of all tiles before this one
    uint32_t etile[kMaxLocalExperts];              // first tile of the expert
    uint32_t task[kBTaskRing];                     // claimed tasks: turn of the ring << 16 | L2 << 15 | tile << 8 | weight tile (0xFFFF: no more)
    alignas(16) uint16_t wcnt[kBRankWarps][kMaxLocalExperts];  // routing entries per (run, expert), then the exclusive sums over the runs
    alignas(16) uint8_t ex[kBMaxRows];             // expert of every routing entry (0xFF: masked, 0xFE: no such expert)
    union {
        uint16_t run_cnt[kBRankWarps][kMaxLocalExperts];   // running counts while the list of rows is made (until then)
        float vt[2][kTileTokens * kBVtStride];     // 16 tokens' accumulators of a task, per epilogue group (see b_role_epilogue)
    };
    uint16_t ef[2][128];                           // per epilogue group: routing entry and top-k weight of the task's rows
    float ew[2][128];
    uint16_t rowf[kBMaxRows];                      // routing entry (token * topk + slot) of every row, experts one after the other
};

__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
// one full 32 B sector per lane
__device__ __forceinline__ void st_global_v8(void* p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// The cold parts of failing and waiting are out of line and get what they need by value: were they members, the context would
// have to live in memory, and every access through it after a barrier or a volatile access would go there again.
__device__ __noinline__ void b_fail(uint8_t* ctrl, uint32_t* abort_flag, uint32_t code, uint32_t detail) {
    atomicCAS(reinterpret_cast<uint32_t*>(ctrl + kCtrlStatus), 0u, code | (blockIdx.x << 8) | (detail << 16));
    *reinterpret_cast<volatile uint32_t*>(abort_flag) = 1u;
}
__device__ __noinline__ bool b_wait_slow(uint64_t* bar, uint32_t parity, uint32_t code, uint32_t* abort_flag, uint64_t deadline, uint8_t* ctrl) {
    uint32_t it = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++it & 0xFFu) == 0u) {
            if (*reinterpret_cast<volatile uint32_t*>(abort_flag) != 0u) return false;
            if (globaltimer_ns() > deadline) { b_fail(ctrl, abort_flag, code, 0u); return false; }
        }
    }
    return true;
}

// What the one-rank kernels share: abort flag, deadline, bounded waits, time records.
struct BCore {
    const BParams& p;
    uint32_t* abort_flag;
    uint8_t* smem;
    uint64_t deadline;
    uint32_t par;
    __device__ __forceinline__ bool aborted() const { return *reinterpret_cast<volatile uint32_t*>(abort_flag) != 0u; }
    __device__ __forceinline__ void fail(uint32_t code, uint32_t detail = 0) const { b_fail(p.buf + p.off_ctrl, abort_flag, code, detail); }
    __device__ __forceinline__ bool expired() const { return globaltimer_ns() > deadline; }
    // for polling loops: give up when the launch is aborted or its time has run out (looked at every 64th time)
    __device__ __forceinline__ bool give_up(uint32_t& spins, uint32_t code, uint32_t detail) const {
        if ((++spins & 0x3Fu) != 0u) return false;
        if (aborted()) return true;
        if (expired()) { fail(code, detail); return true; }
        return false;
    }
    __device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity, uint32_t code) const {
        return mbar_try_wait(bar, parity) ? true : b_wait_slow(bar, parity, code, abort_flag, deadline, p.buf + p.off_ctrl);
    }
    __device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, uint32_t code) const {
        return __all_sync(0xffffffffu, wait(bar, parity, code));
    }
    // a count in global memory reaches `need` (one lane polls for its warp)
    __device__ __forceinline__ bool wait_count(const uint32_t* cnt, uint32_t need, uint32_t code, uint32_t detail) const {
        uint32_t it = 0;
        for (uint32_t v; (v = ld_acquire_gpu(cnt)) < need;) {
            if (need - v > 2u) __nanosleep(min(8u * (need - v), 300u));      // (a poll takes from what the others' counts and weights can get)
            if ((++it & 0x1Fu) == 0u) {
                if (aborted()) return false;
                if (expired()) { fail(code, detail); return false; }
            }
        }
        return true;
    }
    __device__ __forceinline__ void sm_phase(int slot, unsigned long long t = globaltimer_ns()) const {
        reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlSmPhase)[blockIdx.x * kSmPhaseSlots + slot] = t;
    }
    __device__ __forceinline__ void stamp(int slot, unsigned long long t = globaltimer_ns()) const {
        reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlStamps)[slot] = t;
    }
    __device__ __forceinline__ void stamp_max(int slot, unsigned long long t = globaltimer_ns()) const {
        atomicMax(reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlStamps) + slot, t);
    }
    // counters, `kBCountStride` words apart: `i` is a column block, kBCountClaims, or kBCountTiles + layer * kBMaxTiles + tile (layer 0:
    // rows in the token image, layer 1: L1 tasks done)
    __device__ __forceinline__ uint32_t* counter(uint32_t parity, uint32_t i) const {
        return reinterpret_cast<uint32_t*>(p.buf + p.off_token_tiles - kBCountBytes) + parity * kBCounts + i * kBCountStride;
    }
    // clears the sets of the other parity, the multi-rank kernel's arrival counts among them (one warp of every SM)
    __device__ __forceinline__ void clear_other(uint32_t lane) const {
        uint32_t* other = reinterpret_cast<uint32_t*>(p.buf + p.off_arrive) + (par ^ 1u) * 2u * p.tile_capacity;
        #pragma unroll 1
        for (uint32_t i = blockIdx.x * 32u + lane; i < 2u * p.tile_capacity; i += gridDim.x * 32u) other[i] = 0u;
        #pragma unroll 1
        for (uint32_t i = blockIdx.x * 32u + lane; i < static_cast<uint32_t>(kBCounters); i += gridDim.x * 32u) *counter(par ^ 1u, i) = 0u;
    }
};
struct BCtx : BCore {
    BShared& c;
    __device__ __forceinline__ BCtx(const BParams& p_, BShared& c_, uint8_t* smem_, uint64_t deadline_, uint32_t par_)
        : BCore{p_, &c_.abort_flag, smem_, deadline_, par_}, c(c_) {}
};

template <int kFmt> struct BFmt {
    static constexpr bool kA8 = kFmt == 2;
    static constexpr int kVec = kFmt == 1 ? 16 : 32;
    static constexpr uint32_t kPlanes = kUnitK / (4 * kVec);
    static constexpr uint32_t kAtoms = kA8 ? 2u : 1u;               // 128 B swizzle atoms of a token row per K unit
    static constexpr int kThreadsAll = kA8 ? kBThreadsA8 : kBThreads;
    // bytes of one K unit's record of a tile with `a16` groups of 16 rows
    static __device__ __forceinline__ uint32_t rec(uint32_t a16) { return a16 * 2048u * kAtoms + kPlanes * 512u; }
    // offset of a tile's image: `ku` K units, `before` 16-row groups and `m` tiles in front of it
    static __device__ __forceinline__ size_t image(uint32_t ku, uint32_t before, uint32_t m) {
        return static_cast<size_t>(ku) * (static_cast<size_t>(before) * 2048u * kAtoms + static_cast<size_t>(m) * (kPlanes * 512u));
    }
};
// a row's scale word inside a plane: the 32-lane x 4-column order of the tensor-memory scale copy
__device__ __forceinline__ uint32_t plane_off(uint32_t n) { return (n & 31u) * 16u + (n >> 5) * 4u; }
// lane 0's value, for the compiler a warp-uniform one
__device__ __forceinline__ uint32_t b_uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
// 1 / 2^(e - 127) for an exponent byte e in [1, 254], exact
__device__ __forceinline__ float pow2_recip(uint32_t e) { return __uint_as_float(e == 254u ? 0x00400000u : (254u - e) << 23); }

// Task `ti` of this SM: layer << 28 | tile << 8 | weight tile, ~0 past the last one (kBNoTask: the launch is being aborted).
// The L1 tasks are dealt round-robin up to the last full round but one; the others and the L2 tasks are claimed one by one
// by the weight loader (a slow SM takes fewer), which leaves them in a ring for the other roles.
constexpr uint32_t kBEnd = 0xFFFFFFFFu, kBNoTask = 0xFFFFFFFEu;
struct BTasks {
    const BCtx& cx;
    uint32_t my1, dealt;                             // dealt tasks of this SM, and of all SMs
    __device__ __forceinline__ explicit BTasks(const BCtx& c_) : cx(c_) {
        const uint32_t G = gridDim.x, nt1 = c_.c.M * c_.p.n1, full = udiv_small(nt1, G);
        my1 = full > 2u ? full - 1u : (blockIdx.x < nt1 ? 1u : 0u);
        dealt = full > 2u ? (full - 1u) * G : (nt1 < G ? nt1 : G);
    }
    __device__ __forceinline__ uint32_t l1(uint32_t t) const {
        const uint32_t m = udiv_small(t, cx.p.n1);
        return (m << 8) | (t - m * cx.p.n1);
    }
    __device__ __forceinline__ uint32_t get(uint32_t ti) const {
        if (ti < my1) return l1(blockIdx.x + ti * gridDim.x);
        const uint32_t k = ti - my1, tag = (k / kBTaskRing + 1u) << 16;
        volatile uint32_t* slot = &cx.c.task[k % kBTaskRing];
        uint32_t v = *slot, it = 0;
        while ((v & 0xFFFF0000u) != tag) {
            __nanosleep(20);
            if ((++it & 0xFFu) == 0u && (cx.aborted() || cx.expired())) { if (!cx.aborted()) cx.fail(kErrTaskCapacity); return kBNoTask; }
            v = *slot;
        }
        __syncwarp();
        return (v & 0xFFFFu) == 0xFFFFu ? kBEnd : ((v & 0x8000u) << 13) | (v & 0x7FFFu);
    }
};

// ============================================================================================= loaders
template <bool kA8, bool kAsk>
__device__ void b_role_weights(const BCtx& cx, uint32_t lane) {
    const BParams& p = cx.p; BShared& c = cx.c;
    const uint32_t nw = b_uniform(c.nw), step = kA8 ? 1u : b_uniform(c.spu), stage_bytes = step * p.unit_bytes, G = gridDim.x, n1 = p.n1, n2 = p.n2, M = b_uniform(c.M);
    uint8_t* ring = cx.smem + b_uniform(c.nr * c.slot_bytes);
    const uint64_t policy = l2_evict_first_policy();
    uint32_t it = 0, s = 0, ph = 0;
    BTasks tasks(cx);
    // Order of the L2 tasks: tile by tile (the first tiles' L1 outputs are complete long before the last ones'), but the last
    // tiles column block by column block: the combine starts on a column block when all tiles have it, beside the remaining ones. How many: `set_column_tiles`.
    const uint32_t NT1 = M * n1, NT2 = M * n2, tail = M >= p.column_long_from ? p.column_tiles_long : p.column_tiles, mA = tail < M ? M - tail : 0u, NA = mA * n2;
    // The stream starts when this SM's rows are in the images. What an SM has asked for comes back in order: behind 100 KB and more of weights
    // the acknowledgement of the rows' release took 2 to 3 us, and every task that wants one of them waited
    // for it (13 tokens: 51.3 -> 50.0 us a pass, 64: 60.3 -> 58.6, 512: 80.3 -> 79.8, 6 of the small layer: 15.4 -> 15.0).
    bar_sync(kBBarPlaced, 32u * (kBWorkWarps + 1));
    uint32_t* claims = cx.counter(cx.par, kBCountClaims);
    uint32_t next = 0u;
    if (tasks.my1 == 0u && lane == 0) next = atomicAdd(claims, 1u);
    #pragma unroll 1
    for (uint32_t ti = 0;; ++ti) {
        uint32_t t;
        if (ti < tasks.my1) t = tasks.l1(blockIdx.x + ti * G);
        else {
            const uint32_t k = ti - tasks.my1;
            uint32_t q = __shfl_sync(0xffffffffu, next, 0) + tasks.dealt;
            if (q < NT1) t = tasks.l1(q);
            else {
                q -= NT1;
                t = 0xFFFFu;
                if (q < NA) { const uint32_t m = udiv_small(q, n2); t = 0x8000u | (m << 8) | (q - m * n2); }
                else if (q < NT2) { const uint32_t j = udiv_small(q - NA, M - mA); *reinterpret_cast<volatile uint32_t*>(&c.comb_open) = 1u; t = 0x8000u | ((mA + q - NA - j * (M - mA)) << 8) | j; }
            }
            if (lane == 0) *reinterpret_cast<volatile uint32_t*>(&c.task[k % kBTaskRing]) = ((k / kBTaskRing + 1u) << 16) | t;
            if (t == 0xFFFFu) {                              // (the epilogue groups look at every second task: both of the next two end there)
                if (lane == 0) *reinterpret_cast<volatile uint32_t*>(&c.task[(k + 1u) % kBTaskRing]) = (((k + 1u) / kBTaskRing + 1u) << 16) | t;
                *reinterpret_cast<volatile uint32_t*>(&c.comb_open) = 1u;
                break;
            }
            t = ((t & 0x8000u) << 13) | (t & 0x7FFFu);
        }
        if (ti + 1u >= tasks.my1 && lane == 0) next = atomicAdd(claims, 1u);     // (needed after this task: its latency is hidden)
        const uint32_t layer = t >> 28, e = c.tile_e[(t >> 8) & 0xFFFFu], j = t & 0xFFu;
        const uint32_t units = layer ? p.k2 : p.k1;
        const uint8_t* src = (layer ? p.w2 : p.w1) + (static_cast<size_t>(e) * (layer ? n2 : n1) + j) * units * p.unit_bytes;
        #pragma unroll 1
        for (uint32_t u = 0; u < units; u += step, ++it, src += stage_bytes) {
            uint64_t* full = kA8 ? &c.wfull[s] : &c.rfull[s];
            if (kAsk && it == nw) {
                // the ring is full for the first time: the units behind it into the L2, while the MMAs wait for the first records
                if (lane == 0) {
                    const uint32_t here = kBAhead < units - u ? kBAhead : units - u, there = kBAhead - here;
                    bulk_prefetch_l2(src, here * p.unit_bytes);
                    if (there != 0u && ti + 1u < tasks.my1) {
                        const uint32_t next_t = tasks.l1(blockIdx.x + (ti + 1u) * G);
                        bulk_prefetch_l2(p.w1 + (static_cast<size_t>(c.tile_e[next_t >> 8]) * n1 + (next_t & 0xFFu)) * p.k1 * p.unit_bytes,
                                         (there < static_cast<uint32_t>(p.k1) ? there : p.k1) * p.unit_bytes);
                    }
                }
                __syncwarp();
            }
            if (!cx.warp_wait(kA8 ? &c.wempty[s] : &c.rempty[s], ph ^ 1u, kErrWaitEmpty)) return;
            if (elect_one()) {
                const uint32_t bytes = (units - u < step ? units - u : step) * p.unit_bytes;
                mbar_arrive_expect_tx(full, bytes);
                bulk_g2s_hint(ring + static_cast<size_t>(s) * stage_bytes, src, bytes, full, policy);
                c.wissued = it + 1u;
                if (it == 0u) {
                    reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlSmWFirst)[blockIdx.x] = globaltimer_ns();
                    cx.sm_phase(kSmFirstIssue);
                }
            }
            __syncwarp();
            if (++s == nw) { s = 0; ph ^= 1u; }
        }
    }
}

template <int kFmt>
__device__ void b_role_records(const BCtx& cx) {
    using F = BFmt<kFmt>;
    const BParams& p = cx.p; BShared& c = cx.c;
    const uint32_t lane = threadIdx.x & 31u, nr = b_uniform(c.nr), slot_bytes = b_uniform(c.slot_bytes), step = b_uniform(c.spu);
    uint32_t it = 0, s = 0, ph = 0;
    uint32_t ready = 0u, seen = ~0u;
    bool seen_l2 = false;
    BTasks tasks(cx);
    #pragma unroll 1
    for (uint32_t ti = 0;; ++ti) {
        const uint32_t t = tasks.get(ti);
        if (t >= kBNoTask) break;
        const uint32_t layer = t >> 28, m = (t >> 8) & 0xFFFFu;
        // The tile is complete: L1 its rows, L2 the outputs of all L1 weight tiles. Looked up 32 tiles at a time, one lane per
        // tile; the latest answer is kept, so that following tasks of the same tiles ask only while theirs is incomplete.
        const uint32_t window = (m >> 5) | (layer << 8);
        if (window != seen || ((ready >> (m & 31u)) & 1u) == 0u) {
            uint32_t spins = 0;
            const uint32_t mm_ = (m & ~31u) + lane;
            const uint32_t* count = cx.counter(cx.par, kBCountTiles + layer * kBMaxTiles + mm_);
            bool r = false;
            for (;;) {
                if (mm_ < c.M && (spins == 0u || mm_ == m)) r = ld_acquire_gpu(count) >= (layer ? static_cast<uint32_t>(p.n1) : c.tile_rows[mm_]);
                ready = __ballot_sync(0xffffffffu, r);
                if ((ready >> (m & 31u)) & 1u) break;
                if ((++spins & 0xFu) == 0u) {                 // (the others' answers are asked for once, this tile's until it is complete)
                    if (cx.aborted()) return;
                    if (cx.expired()) { cx.fail(layer ? kErrWaitL1Done : kErrWaitDispatchFlag, c.tile_e[m]); return; }
                }
            }
            seen = window;
            fence_proxy_async_all();                         // rows written through the generic proxy, read by bulk copies
        }
        const uint32_t a16 = (c.tile_rows[m] + 15u) >> 4, rec = F::rec(a16), units = layer ? p.k2 : p.k1;
        const uint8_t* src = p.buf + (layer ? p.off_mid_tiles : p.off_token_tiles) + F::image(units, c.tile_a16[m], m);
        if (lane == 0u && layer != 0u && !seen_l2) { seen_l2 = true; cx.sm_phase(kSmFirstL2Staged); }
        #pragma unroll 1
        for (uint32_t u = 0; u < units; u += step, ++it, src += step * rec) {
            if (!cx.warp_wait(&c.rempty[s], ph ^ 1u, kErrWaitActsEmpty)) return;
            if (elect_one()) {
                const uint32_t bytes = (units - u < step ? units - u : step) * rec;
                mbar_arrive_expect_tx(&c.rfull[s], bytes);
                bulk_g2s(cx.smem + static_cast<size_t>(s) * slot_bytes, src, bytes, &c.rfull[s]);
                c.rissued = it + 1u;
                if (it == 0u) cx.sm_phase(kSmFirstStaged);
            }
            __syncwarp();
            if (++s == nr) { s = 0; ph ^= 1u; }
        }
    }
}

// ============================================================================================= MMA issuer
template <int kFmt>
__device__ void b_role_mma(const BCtx& cx, uint32_t lane) {
    using F = BFmt<kFmt>;
    constexpr bool kA8 = F::kA8;
    constexpr uint32_t kPlanes = F::kPlanes, kStepK = kA8 ? 32u : 64u;
    constexpr uint32_t kIdesc = kA8 ? idesc_block_scaled(kFmtF8E2M1, kFmtF8E4M3, 128u, 0u, 1u)
                                    : idesc_block_scaled(kFmtMxf4E2M1, kFmtMxf4E2M1, 128u, 0u, kFmt == 1 ? 0u : 1u);
    const BParams& p = cx.p; BShared& c = cx.c;
    // Everything the instructions below take as operands is broadcast from lane 0, which tells the compiler that it is the
    // same in all lanes: the operands then stay in uniform registers. (A unit of 4 MMAs, 4 scale copies and a commit goes out in
    // 210 cycles with 16 rows and 257 with 96: the tensor pipe itself needs 199 and 256. E4M3 tokens: 206 for 16 rows, 480 for 96.)
    const uint32_t nr = b_uniform(c.nr), slot_bytes = b_uniform(c.slot_bytes), step = b_uniform(c.spu), tm = b_uniform(c.tmem_base);
    const uint32_t rec0 = b_uniform(smem_u32(cx.smem)), ring0 = rec0 + nr * slot_bytes;
    uint32_t it = 0, rs = 0, rph = 0;                                   // units consumed; record slot (without widening also weight stage), its phase bit
    BTasks tasks(cx);
    #pragma unroll 1
    for (uint32_t ti = 0;; ++ti) {
        const uint32_t t = b_uniform(tasks.get(ti));
        if (t >= kBNoTask) break;
        const uint32_t m = (t >> 8) & 0xFFFFu, units = (t >> 28) ? p.k2 : p.k1;
        const uint32_t atom = b_uniform(((c.tile_rows[m] + 15u) >> 4) * 2048u);       // bytes of one 128 B atom of the tile's rows
        const uint32_t idesc_n = kIdesc | ((atom >> 10) << 17);                       // N = rows, in units of 8
        const uint32_t rec = atom * F::kAtoms + kPlanes * 512u, acc = ti & 1u, use = (ti >> 1) & 1u, d = tm + acc * 128u;
        if (!cx.warp_wait(&c.tmem_empty[acc], use ^ 1u, kErrWaitTmemEmpty)) return;
        #pragma unroll 1
        for (uint32_t u = 0; u < units;) {
            // A turn of this loop is a barrier wait, a fence, an election and a reconvergence beside the issue itself: a stage that is
            // there already when the first is goes with it (300 tokens 72.9 us with one stage a turn, 71.4 this way; 512: 79.7, 77.0).
            if (!cx.warp_wait(&c.rfull[rs], rph, kErrWaitActsFull)) return;
            if constexpr (kA8) { if (!cx.warp_wait(&c.xfull[it & 1u], (it >> 1) & 1u, kErrWaitFull)) return; }
            const uint32_t rs1 = rs + 1u == nr ? 0u : rs + 1u, rph1 = rs1 == 0u ? rph ^ 1u : rph;
            bool more = u + step < units && mbar_test(&c.rfull[rs1], rph1);
            if constexpr (kA8) more = more && mbar_test(&c.xfull[(it + 1u) & 1u], ((it + 1u) >> 1) & 1u);
            const uint32_t n = __all_sync(0xffffffffu, more) ? 2u : 1u;
            tc_fence_after();
            if (lane == 0 && it == 0u) cx.sm_phase(kSmFirstLanded);
            if (elect_one()) {
                #pragma unroll 1
                for (uint32_t b = 0; b < n; ++b) {
                    const uint32_t slot = b ? rs1 : rs, tok0 = rec0 + slot * slot_bytes, wsm0 = ring0 + slot * (step * p.unit_bytes), u0 = u + b * step;
                    #pragma unroll
                    for (uint32_t uu = 0; uu < (kA8 ? 1u : 2u); ++uu) {
                        if (uu < step && u0 + uu < units) {
                            const uint32_t i = it + b * step + uu;
                            const uint32_t wsm = wsm0 + uu * p.unit_bytes, tok = tok0 + uu * rec;      // (E4M3 tokens: weights and their scales are in tensor memory)
                            const uint64_t adesc = smem_desc(wsm, 1024u, kLayoutSw128), bdesc = smem_desc(tok, 1024u, kLayoutSw128);
                            const uint64_t asf = smem_desc(wsm + kUnitWBytes, 128u, kLayoutNone);
                            const uint64_t bsf = smem_desc(tok + atom * F::kAtoms, 128u, kLayoutNone);
                            const uint32_t sfa = kA8 ? tm + kTmScaleW + (i & 1u) * 8u : tm + 256u + (i & 1u) * 32u, sfb = kA8 ? tm + kTmScaleX + (i & 1u) * 8u : sfa + 16u;
                            const uint32_t wide = tm + kTmWide + (i & 1u) * 64u;
                            #pragma unroll
                            for (uint32_t pl = 0; pl < kPlanes; ++pl) {
                                if constexpr (!kA8) utccp_32x128b_warpx4(sfa + pl * 4u, asf + pl * 32u);
                                utccp_32x128b_warpx4(sfb + pl * 4u, bsf + pl * 32u);
                            }
                            #pragma unroll
                            for (uint32_t ks = 0; ks < kUnitK / kStepK; ++ks) {
                                const uint32_t pl = (ks * kStepK) / (4u * F::kVec), sf_id = ((ks * kStepK) % (4u * F::kVec)) / F::kVec;
                                const uint64_t ad = adesc + (ks & 3u) * 2u;
                                const uint64_t bd = bdesc + (ks & 3u) * 2u + (kA8 ? (ks >> 2) * (atom >> 4) : 0u);
                                const uint32_t idesc = idesc_with_sf(idesc_n, sf_id, sf_id), accum = (u0 | uu | ks) != 0u ? 1u : 0u;
                                if constexpr (kA8) umma_mxf8f6f4_ta(d, wide + ks * 8u, bd, idesc, sfa + pl * 4u, sfb + pl * 4u, accum);
                                else if constexpr (kFmt == 0) umma_mxf4_block32(d, ad, bd, idesc, sfa + pl * 4u, sfb + pl * 4u, accum);
                                else umma_nvf4_block16(d, ad, bd, idesc, sfa + pl * 4u, sfb + pl * 4u, accum);
                            }
                            if constexpr (kA8) tc_commit(&c.xempty[i & 1u]);
                        }
                    }
                    tc_commit(&c.rempty[slot]);
                }
            }
            __syncwarp();
            const uint32_t done = n * step < units - u ? n * step : units - u;
            u += n * step; it += done;
            if (n == 2u) { rs = rs1; rph = rph1; }
            if (++rs == nr) { rs = 0; rph ^= 1u; }
        }
        if (elect_one()) tc_commit(&c.tmem_full[acc]);
        __syncwarp();
    }
    if (lane == 0 && it != 0u) cx.stamp_max(kStampLastWeight);
}

// ============================================================================================= weight widener (E4M3 tokens)
// kind::mxf8f6f4 wants a byte per weight. Two groups of four warps take the units in turn and write them into tensor memory,
// where the MMAs read their A operand: a thread reads the 128 packed bytes of its weight row and stores 64 columns of E2M1
// codes in bytes, the form in which tcgen05.cp would decompress them (code in bits 2 to 5). The unit's scale planes go the same way, in
// the layout that the scale copy would give them. Measured for one SM, cycles a unit: 313 with both groups (one group 508; codes turned into E4M3 bytes
// by byte permutes, in order, 669; by shifts and masks 435), beside MMAs of 206 (16 rows) to 480 (96), which take 431 to 731 with A in shared
// memory. HBM brings a unit in 790. Widened in shared memory (16 KB read, 32 KB written, those read again by
// the tensor core, and a proxy fence) a unit took 1200: 2 tokens 37.7 -> 31.9 us a pass, 100 tokens 91.4 -> 67.7.
// Shifts and masks alone leave the codes of the even elements in one word and those of the odd ones in the next: the token
// images have every eight elements of a row in the same order (`even_odd`).
constexpr uint32_t kXGroupThreads = 128;
// eight E2M1 codes -> eight bytes with the code in bits 2..5, those of the even elements first: two shifts and two masks
__device__ __forceinline__ void widen8(uint32_t w, uint32_t& even, uint32_t& odd) {
    even = (w << 2) & 0x3C3C3C3Cu;
    odd = (w >> 2) & 0x3C3C3C3Cu;
}
// the same order of eight consecutive E4M3 bytes
__device__ __forceinline__ uint2 even_odd(uint32_t a, uint32_t b) { return make_uint2(__byte_perm(a, b, 0x6420u), __byte_perm(a, b, 0x7531u)); }
__device__ __forceinline__ uint4 even_odd(const uint4& v) {
    const uint2 a = even_odd(v.x, v.y), b = even_odd(v.z, v.w);
    return make_uint4(a.x, a.y, b.x, b.y);
}
struct BWiden {
    uint4 v[8], sf[2];
    __device__ __forceinline__ void load(const uint8_t* wsm, uint32_t row) {
        #pragma unroll
        for (uint32_t c = 0; c < 8; ++c) v[c] = *reinterpret_cast<const uint4*>(wsm + row * 128u + ((c ^ (row & 7u)) << 4));
        #pragma unroll
        for (uint32_t pl = 0; pl < 2; ++pl) sf[pl] = *reinterpret_cast<const uint4*>(wsm + kUnitWBytes + pl * 512u + (row & 31u) * 16u);
    }
    // (`ta`, `tsf`: columns, with the first of the warp's lanes)
    __device__ __forceinline__ void store(uint32_t ta, uint32_t tsf) const {
        #pragma unroll
        for (uint32_t c = 0; c < 8; c += 2) {
            uint32_t r[16];
            #pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint4 q = v[c + h];
                widen8(q.x, r[8 * h], r[8 * h + 1]); widen8(q.y, r[8 * h + 2], r[8 * h + 3]);
                widen8(q.z, r[8 * h + 4], r[8 * h + 5]); widen8(q.w, r[8 * h + 6], r[8 * h + 7]);
            }
            tmem_st_32x32b_x16(ta + c * 8u, r);
        }
        tmem_st_32x32b_x8(tsf, sf[0], sf[1]);
        tmem_st_wait();
        tc_fence_before();
    }
};

// The ring has an even number of stages, so that a stage always belongs to the same group: a group that skipped a stage's
// previous use could take the older phase of its barrier for the one it wants. The decode kernel's ring too: `fit` stages have room.
__device__ __forceinline__ uint32_t even_stages(uint32_t fit, uint32_t most) { return (fit < most ? fit : most) & ~1u; }
__device__ void b_role_widen(const BCtx& cx, uint32_t grp, uint32_t xtid) {
    const BParams& p = cx.p; BShared& c = cx.c;
    const uint32_t lane = xtid & 31u, nw = c.nw;
    const uint8_t* ring = cx.smem + c.nr * c.slot_bytes;
    const uint32_t tm = c.tmem_base + ((xtid & 96u) << 16), ta = tm + kTmWide + grp * 64u, tsf = tm + kTmScaleW + grp * 8u;
    uint32_t it = 0, s = 0, ph = 0;
    BTasks tasks(cx);
    #pragma unroll 1
    for (uint32_t ti = 0;; ++ti) {
        const uint32_t t = tasks.get(ti);
        if (t >= kBNoTask) break;
        const uint32_t units = (t >> 28) ? p.k2 : p.k1;
        #pragma unroll 1
        for (uint32_t u = 0; u < units; ++u, ++it) {
            if ((it & 1u) == grp) {
                if (!cx.warp_wait(&c.wfull[s], ph, kErrWaitFull)) return;
                BWiden w;
                w.load(ring + static_cast<size_t>(s) * p.unit_bytes, xtid);
                __syncwarp();
                if (lane == 0) mbar_arrive(&c.wempty[s]);        // (the unit is in registers: its stage can be refilled)
                if (!cx.warp_wait(&c.xempty[grp], ((it >> 1) & 1u) ^ 1u, kErrWaitEmpty)) return;
                tc_fence_after();
                w.store(ta, tsf);
                __syncwarp();
                if (lane == 0) mbar_arrive(&c.xfull[grp]);
            }
            if (++s == nw) { s = 0; ph ^= 1u; }
        }
    }
}

// ============================================================================================= epilogue
// SwiGLU of 8 outputs of one token from its 8 gate and 8 up accumulators. With `fast_math` the reciprocal of 1 + exp(-gate)
// is the hardware approximation refined by one Newton-Raphson step: straight-line code, several times faster than the
// exact reciprocal with its range checks. (Compared with the correctly rounded reciprocal for every mantissa and the
// exponents 0 to 125: no difference. Beyond, from a gate of -87.3 on, the approximation is zero: those take the other way.)
__device__ __forceinline__ void b_swiglu(const BParams& p, const float (&a)[16], float wgt, bool live, float (&o)[8]) {
    float g[8], u[8];
    const bool cl = p.has_clamp != 0;
    #pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const __nv_bfloat162 gu = __floats2bfloat162_rn(a[i] * p.l1_scale, a[i + 8] * p.l1_scale);
        const float gate = __low2float(gu), up = __high2float(gu);
        const float gc = fminf(gate, p.clamp), uc = fminf(fmaxf(up, -p.clamp), p.clamp);
        g[i] = cl ? gc : gate;
        u[i] = cl ? uc : up;
    }
    float least = 0.f;
    #pragma unroll
    for (uint32_t i = 0; i < 8; ++i) least = fminf(least, g[i]);
    if (p.fast_math && (least >= -87.0f || !live)) {              // (the columns beyond the tile's rows hold anything)
        #pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            const float d = 1.0f + __expf(-g[i]);
            float r = __fdividef(1.0f, d);
            r = fmaf(r, fmaf(-d, r, 1.0f), r);
            o[i] = g[i] * r * u[i] * wgt;
        }
    } else {
        #pragma unroll
        for (uint32_t i = 0; i < 8; ++i) o[i] = g[i] * (1.0f / (1.0f + expf(-g[i]))) * u[i] * wgt;
    }
}
// x / b from y = RN(1 / b): one residual correction of the product x * y gives the correctly rounded quotient (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990), without a division's range checks.
// Its condition is that the residual is exact: with 2^-40 <= b <= 2^40 for quotients from 2^-40 up to the largest finite one.
// Where one of the eight is something else - a zero, whose sign the residual loses, or an infinity - `divide8` divides them all.
__device__ __forceinline__ void divide8(float (&o)[8], float b, float y) {
    float lo = INFINITY, hi = 0.f, d[8];
    #pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const float q = o[i] * y;
        d[i] = fmaf(fmaf(-q, b, o[i]), y, q);
        lo = fminf(lo, fabsf(q));
        hi = fmaxf(hi, fabsf(q));
    }
    if (__builtin_expect(!(lo >= 0x1p-40f && hi < INFINITY), 0)) {
        #pragma unroll
        for (uint32_t i = 0; i < 8; ++i) d[i] = __fdiv_rn(o[i], b);
    }
    #pragma unroll
    for (uint32_t i = 0; i < 8; ++i) o[i] = d[i];
}

// Requantises the 8 outputs of thread (n, q): o becomes the scaled values, the thread q = 0 gets the scale bytes of the
// token's 64 columns in sfw (two bytes, one per 32 columns, or four). All lanes of the warp call it; `live`: the token is one.
template <int kFmt>
__device__ __forceinline__ void b_requantise(const BParams& p, float (&o)[8], bool live, uint32_t& sfw) {
    constexpr bool kA8 = BFmt<kFmt>::kA8;
    constexpr int kVec = BFmt<kFmt>::kVec;
    float amax = 0.f;
    if constexpr (kVec == 16) { if (live) divide8(o, p.mid_gs, p.mid_gs_recip); }
    #pragma unroll
    for (uint32_t i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(o[i]));
    // a scale block is the 8 columns of two (16 per block) or four threads
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    if constexpr (kVec == 32) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, 1e-30f);
    uint32_t sf_byte;
    if constexpr (kVec == 32) {
        sf_byte = ceil_pow2_exp(__fdiv_rn(amax, kA8 ? 448.0f : 6.0f));
        const float inv = pow2_recip(sf_byte);                    // a power of two: the product equals the quotient
        #pragma unroll
        for (uint32_t i = 0; i < 8; ++i) o[i] *= inv;
    } else {
        sf_byte = cvt_e4m3x2(__fdiv_rn(amax, 6.0f), 0.f) & 0xFFu;
        if (sf_byte != 0u) {
            if (live) { const float sf = e4m3_to_float(sf_byte); divide8(o, sf, __frcp_rn(sf)); }
        } else {                                                  // a scale that rounds to zero: every non-zero value saturates
            #pragma unroll
            for (uint32_t i = 0; i < 8; ++i) o[i] = o[i] == 0.f ? 0.f : copysignf(6.0f, o[i]);
        }
    }
    // the token's scale bytes of this tile, gathered in the thread q = 0
    sfw = sf_byte;
    if constexpr (kVec == 32) sfw |= __shfl_down_sync(0xffffffffu, sf_byte, 4) << 8;
    else {
        sfw |= __shfl_down_sync(0xffffffffu, sf_byte, 2) << 8;
        sfw |= __shfl_down_sync(0xffffffffu, sfw, 4) << 16;
    }
}
// A task's accumulators lie with weight row l in lane l and token n in column n. 16 tokens at a time go through shared
// memory: weight row 16 q + 4 i + k of token n to vt[n * 152 + i * 40 + q * 4 + k], which neither the writes (a warp: 32
// rows of one token) nor the 16-byte reads (thread (n, q): its i = 0..3) find bank conflicts in. Thread (n = t / 8, q = t % 8)
// then owns the 16 weight rows of group q of token n: L1 8 gate rows and the 8 matching up rows, L2 16 output columns.
template <int kFmt, bool kFe>
__device__ void b_role_epilogue(const BCtx& cx, uint32_t grp, uint32_t etid) {
    using F = BFmt<kFmt>;
    constexpr bool kA8 = F::kA8;
    constexpr int kVec = F::kVec;
    const BParams& p = cx.p; BShared& c = cx.c;
    const uint32_t ew = etid >> 5, q = etid & 7u, n16 = etid >> 3;
    // the rows' top-k weights: the caller's view, or the routing records this launch's own frontend wrote
    const uint8_t* tw = kFe ? p.buf + p.off_routes + 8 : p.buf + p.off_topk_w;
    constexpr uint32_t kTwStride = kFe ? 16u : 4u;
    const uint32_t bar = grp ? kBBarEpi1 : kBBarEpi0;
    float* vt = c.vt[grp];
    float* vt_w = vt + ((etid & 15u) >> 2) * 40u + (etid >> 4) * 4u + (etid & 3u);
    const float* vt_r = vt + n16 * kBVtStride + q * 4u;
    BTasks tasks(cx);
    #pragma unroll 1
    for (uint32_t ti = grp;; ti += 2) {
        const uint32_t t = tasks.get(ti);
        const bool task = t < kBNoTask;
        const uint32_t layer = t >> 28, m = task ? (t >> 8) & 0xFFFFu : 0u, j = t & 0xFFu;
        const uint32_t rows = c.tile_rows[m], a16 = (rows + 15u) >> 4, use = (ti >> 1) & 1u;
        bool ok = t != kBNoTask;
        if (task) {
            if (etid < rows) {
                const uint32_t f = c.rowf[c.tile_row0[m] + etid];
                c.ef[grp][etid] = static_cast<uint16_t>(f);
                if (layer == 0u) c.ew[grp][etid] = __uint_as_float(ld_cg_u32(tw + static_cast<size_t>(f) * kTwStride));
            }
            ok = cx.warp_wait(&c.tmem_full[grp], use, kErrWaitTmemFull);
            tc_fence_after();
        }
        // the group leaves together (an aborted launch, or the end of the tasks); also publishes ef and ew
        if (bar_red_or(bar, 128u, !ok)) return;
        if (!task) break;
        const uint32_t acc = c.tmem_base + ((ew * 32u) << 16) + grp * 128u;
        const uint32_t rec = F::rec(a16);
        uint8_t* img = p.buf + p.off_mid_tiles + F::image(p.k2, c.tile_a16[m], m) + static_cast<size_t>(j >> 2) * rec;
        #pragma unroll 1
        for (uint32_t ch = 0; ch < a16; ++ch) {
            uint32_t raw[kTileTokens];
            tmem_ld_32x32b_x16(acc + ch * 16u, raw);
            tmem_ld_wait();
            if (ch + 1u == a16) { tc_fence_before(); __syncwarp(); if ((etid & 31u) == 0u) mbar_arrive(&c.tmem_empty[grp]); }
            if (ch != 0u) bar_sync(bar, 128u);                              // (the reads of the chunk before are over)
            #pragma unroll
            for (uint32_t n = 0; n < kTileTokens; ++n) vt_w[n * kBVtStride] = __uint_as_float(raw[n]);
            bar_sync(bar, 128u);
            float a[16];
            #pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const float4 v = *reinterpret_cast<const float4*>(vt_r + i * 40u);
                a[4 * i] = v.x; a[4 * i + 1] = v.y; a[4 * i + 2] = v.z; a[4 * i + 3] = v.w;
            }
            const uint32_t n = ch * 16u + n16;
            const bool live = n < rows;
            if (layer == 0u) {
                float o[8];
                b_swiglu(p, a, live ? c.ew[grp][n] : 0.f, live, o);
                uint32_t sfw;
                b_requantise<kFmt>(p, o, live, sfw);
                if (live) {
                    if constexpr (kA8) {
                        uint8_t* at = img + ((j >> 1) & 1u) * a16 * 2048u + sw128_off(n, (j & 1u) * 4u + (q >> 1)) + (q & 1u) * 8u;
                        *reinterpret_cast<uint2*>(at) = make_uint2(cvt_e4m3x2(o[0], o[2]) | (cvt_e4m3x2(o[4], o[6]) << 16),
                                                                   cvt_e4m3x2(o[1], o[3]) | (cvt_e4m3x2(o[5], o[7]) << 16));    // (see widen8)
                    } else {
                        uint8_t* at = img + sw128_off(n, (j & 3u) * 2u + (q >> 2)) + (q & 3u) * 4u;
                        *reinterpret_cast<uint32_t*>(at) = cvt_e2m1x2(o[0], o[1]) | (cvt_e2m1x2(o[2], o[3]) << 8) |
                                                           (cvt_e2m1x2(o[4], o[5]) << 16) | (cvt_e2m1x2(o[6], o[7]) << 24);
                    }
                    if (q == 0u) {
                        uint8_t* sf = img + a16 * 2048u * F::kAtoms + plane_off(n);
                        if constexpr (kVec == 16) *reinterpret_cast<uint32_t*>(sf + (j & 3u) * 512u) = sfw;
                        else *reinterpret_cast<uint16_t*>(sf + ((j >> 1) & 1u) * 512u + (j & 1u) * 2u) = static_cast<uint16_t>(sfw);
                    }
                }
            } else {
                uint32_t w[8];
                #pragma unroll
                for (uint32_t i = 0; i < 8; ++i)
                    w[i] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(a[2 * i] * p.l2_scale))) |
                           (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(a[2 * i + 1] * p.l2_scale))) << 16);
                if (live) st_global_v8(p.buf + p.off_out + (static_cast<size_t>(c.ef[grp][n]) * p.H + j * 128u + q * 16u) * 2u, w);
            }
        }
        // one thread counts the finished task; its release covers the stores of the group, which the barrier orders before it
        bar_sync(bar, 128u);
        if (etid == 96u) {
            if (ti < 2u) cx.sm_phase(kSmFirstEpilogue);
            if (layer == 0u) {
                red_release_gpu_add(cx.counter(cx.par, kBCountTiles + kBMaxTiles + m), 1u);
                cx.sm_phase(kSmLastL1Epilogue);
            } else {
                red_release_gpu_add(cx.counter(cx.par, j), 1u);
            }
        }
    }
}

// ============================================================================================= combine
// Item i = column block * T + token: a half-warp adds the token's routes over 128 columns. SM b has the items b, b + G, ...;
// its warps take them two by two in that order: the combine warps when the SM has come to its first column task, the others
// when their role has ended.
__device__ void b_role_combine(const BCtx& cx, uint32_t lane) {
    const BParams& p = cx.p; BShared& c = cx.c;
    const uint32_t G = gridDim.x, nitems = static_cast<uint32_t>(p.T) * p.n2, half = lane >> 4, l16 = lane & 15u;
    const uint32_t M = c.M;
    uint32_t known = 0xFFFFFFFFu;                            // the column block this half-warp saw complete last
    // nothing is complete before this SM, like the others, has come to the tasks that go column block by column block (without live rows
    // there is nothing to wait for: 200 tokens, every slot masked, 9.66 us a pass behind the gate, 9.27 so)
    for (uint32_t spins = 0; M != 0u && *reinterpret_cast<volatile uint32_t*>(&c.comb_open) == 0u;) {
        __nanosleep(200);
        if (cx.give_up(spins, kErrWaitCombineFlag, 0u)) break;
    }
    __syncwarp();
    #pragma unroll 1
    for (;;) {
        uint32_t k = 0u;
        if (lane == 0) k = atomicAdd(&c.comb_next, 2u);
        k = __shfl_sync(0xffffffffu, k, 0);
        const uint32_t first = blockIdx.x + k * G;
        if (first >= nitems) break;
        const uint32_t i = first + half * G;
        const bool valid = i < nitems;
        const uint32_t col = udiv_small(valid ? i : first, p.T), tok = (valid ? i : first) - col * p.T;
        uint32_t mask = 0u;
        #pragma unroll 1
        for (int sl = 0; sl < p.topk; ++sl) mask |= (c.ex[tok * p.topk + sl] < kMaxLocalExperts ? 1u : 0u) << sl;
        bool ok = true;
        if (col != known && l16 == 0u) ok = cx.wait_count(cx.counter(cx.par, col), M, kErrWaitCombineFlag, tok);
        known = col;
        if (!__all_sync(0xffffffffu, ok)) return;
        __syncwarp();
        __threadfence();                                     // (the polling lanes' acquire, handed to the others)
        const uint8_t* src = p.buf + p.off_out + (static_cast<size_t>(tok) * p.topk * p.H + col * 128u + l16 * 8u) * 2u;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        #pragma unroll 1
        for (int s0 = 0; s0 < p.topk; s0 += 8) {
            uint4 v[8];
            #pragma unroll
            for (int u = 0; u < 8; ++u) {
                v[u] = make_uint4(0u, 0u, 0u, 0u);
                if ((mask >> (s0 + u)) & 1u) v[u] = ld_cg_v4(src + static_cast<size_t>(s0 + u) * p.H * 2u);
            }
            #pragma unroll
            for (int u = 0; u < 8; ++u) {
                acc[0] += __uint_as_float(v[u].x << 16); acc[1] += __uint_as_float(v[u].x & 0xFFFF0000u);
                acc[2] += __uint_as_float(v[u].y << 16); acc[3] += __uint_as_float(v[u].y & 0xFFFF0000u);
                acc[4] += __uint_as_float(v[u].z << 16); acc[5] += __uint_as_float(v[u].z & 0xFFFF0000u);
                acc[6] += __uint_as_float(v[u].w << 16); acc[7] += __uint_as_float(v[u].w & 0xFFFF0000u);
            }
        }
        uint4 o;
        uint32_t* ow = &o.x;
        #pragma unroll
        for (int q = 0; q < 4; ++q)
            ow[q] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(acc[2 * q]))) |
                    (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(acc[2 * q + 1]))) << 16);
        if (valid) *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.y) + (static_cast<size_t>(tok) * p.H + col * 128u + l16 * 8u) * 2u) = o;
        if (lane == 0 && k == 0u) cx.sm_phase(kSmFirstCombined);
        if (lane == 0) cx.sm_phase(kSmCombineDone);
    }
}

// ============================================================================================= routing
// The list of rows, for the epilogue: the run `r` of routing entries, one warp. An entry's place among the rows of its expert is the number
// of earlier entries that name it; 32 entries are a chain of about 560 cycles, bound by the ballots' arithmetic when
// all warps are at it. (So it is not in front of the first copy: that needs the counts alone.)
__device__ __forceinline__ void b_list_run(const BCtx& cx, uint32_t r, uint32_t seg_shift, uint32_t nent, uint32_t lane) {
    BShared& c = cx.c;
    const uint32_t lo = r << seg_shift, hi = min(lo + (1u << seg_shift), nent);
    uint16_t* cnt = c.run_cnt[r];
    reinterpret_cast<uint32_t*>(cnt)[lane] = 0u;
    __syncwarp();
    #pragma unroll 1
    for (uint32_t f0 = lo; f0 < hi; f0 += 32u) {
        const uint32_t f = f0 + lane, e = f < hi ? c.ex[f] : 0xFFu;
        // the lanes with the same expert: one ballot per bit (several times faster than a warp-wide match)
        uint32_t same = __ballot_sync(0xffffffffu, e < kMaxLocalExperts);
        #pragma unroll
        for (uint32_t b = 0; b < 6; ++b) {
            const uint32_t v = __ballot_sync(0xffffffffu, (e >> b) & 1u);
            same &= (e >> b) & 1u ? v : ~v;
        }
        const uint32_t below = same & ((1u << lane) - 1u);
        const uint32_t base = e < kMaxLocalExperts ? cnt[e] : 0u;
        __syncwarp();
        if (e < kMaxLocalExperts) {
            c.rowf[c.ebase[e] + c.wcnt[r][e] + base + __popc(below)] = static_cast<uint16_t>(f);
            if (below == 0u) cnt[e] = static_cast<uint16_t>(base + __popc(same));
        }
        __syncwarp();
    }
}
// entries before entry f in its run that name the same expert e (the whole warp)
__device__ __forceinline__ uint32_t b_rank_in_run(const BShared& c, uint32_t f, uint32_t e, uint32_t seg_shift, uint32_t lane) {
    uint32_t k = 0u;
    #pragma unroll 1
    for (uint32_t i = ((f >> seg_shift) << seg_shift) + lane; i - lane < f; i += 32u) k += __popc(__ballot_sync(0xffffffffu, i < f && c.ex[i] == e));
    return k;
}

// Sums over the runs, the experts' token tiles and the ring geometry (one warp; lane l takes the experts 2l and
// 2l + 1). Everything the SM does waits for it and its code runs once, from a cold instruction cache: few instructions.
template <int kFmt>
__device__ __forceinline__ void b_tiles(const BCtx& cx, uint32_t lane) {
    using F = BFmt<kFmt>;
    const BParams& p = cx.p; BShared& c = cx.c;
    uint32_t* w32 = reinterpret_cast<uint32_t*>(&c.wcnt[0][0]) + lane;
    uint32_t run = 0u, wv[kBRankWarps];                      // two 16-bit counts, at most 4096 each
    #pragma unroll
    for (uint32_t w = 0; w < kBRankWarps; ++w) wv[w] = w32[w * (kMaxLocalExperts / 2)];
    #pragma unroll
    for (uint32_t w = 0; w < kBRankWarps; ++w) { w32[w * (kMaxLocalExperts / 2)] = run; run += wv[w]; }
    const uint32_t lim = p.tile_limit;
    uint32_t cn[2] = {run & 0xFFFFu, run >> 16}, nt[2], rpt[2];
    #pragma unroll
    for (uint32_t h = 0; h < 2; ++h) { nt[h] = cn[h] != 0u ? 1u : 0u; rpt[h] = (cn[h] + 15u) & ~15u; }
    if (__any_sync(0xffffffffu, cn[0] > lim || cn[1] > lim)) {
        #pragma unroll 1
        for (uint32_t h = 0; h < 2; ++h) {                   // ceil(rows / limit) tiles of ceil(rows / tiles) rows, rounded up to 16
            const uint32_t n = h ? cn[1] : cn[0];
            uint32_t k = udiv_small(n + lim - 1u, lim), r = 0u;
            if (k != 0u) { r = (udiv_small(n + k - 1u, k) + 15u) & ~15u; k = udiv_small(n + r - 1u, r); }
            if (h) { nt[1] = k; rpt[1] = r; } else { nt[0] = k; rpt[0] = r; }
        }
    }
    // running sums over the experts of (rows, 16-row groups, tiles), packed 13 + 9 + 10 bits (all tiles of an expert but the
    // last are multiples of 16 rows)
    const uint32_t v0 = cn[0] | ((cn[0] + 15u) >> 4 << 13) | (nt[0] << 22), v1 = cn[1] | ((cn[1] + 15u) >> 4 << 13) | (nt[1] << 22);
    uint32_t incl = v0 + v1;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t a = __shfl_up_sync(0xffffffffu, incl, o); if (static_cast<int>(lane) >= o) incl += a; }
    const uint32_t all = __shfl_sync(0xffffffffu, incl, 31), M = all >> 22;
    const uint32_t max16 = __reduce_max_sync(0xffffffffu, rpt[0] > rpt[1] ? rpt[0] : rpt[1]) >> 4;
    #pragma unroll 1
    for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t e = 2u * lane + h, x = incl - v1 - (h ? 0u : v0), n = h ? cn[1] : cn[0], r = h ? rpt[1] : rpt[0];
        const uint32_t r0 = x & 0x1FFFu, a0 = (x >> 13) & 0x1FFu;
        uint32_t m = x >> 22;
        c.cnt[e] = n; c.ebase[e] = r0; c.etile[e] = m;
        #pragma unroll 1
        for (uint32_t lo = 0; lo < n; lo += r, ++m) {
            if (m >= kBMaxTiles) break;
            c.tile_e[m] = e;
            c.tile_row0[m] = r0 + lo;
            c.tile_rows[m] = n - lo < r ? n - lo : r;
            c.tile_a16[m] = a0 + (lo >> 4);
        }
    }
    if (lane == 0) {
        c.M = M; c.total = all & 0x1FFFu;
        if (M > kBMaxTiles) cx.fail(kErrTaskCapacity, M);
        // (a token that names an expert more than once: more rows than tokens x experts, for which there is no room)
        if ((all & 0x1FFFu) > p.cap_rows) cx.fail(kErrMetaCapacity, (all & 0x1FFFu) >> 4);
        c.start_ok = cx.aborted() ? 0u : 1u;                 // (decided once: every warp takes the same way from here)
        // Rings. Weights and records of equal depth: a record from the L2 takes about as long as a unit from HBM while the
        // weights stream. A stage holds two K units where four such stages fit (narrow tiles): the MMA warp's barrier waits
        // and loop cost more than its issue, and this halves them.
        const uint32_t rec = (max16 ? max16 : 1u) * 2048u * F::kAtoms + F::kPlanes * 512u;
        const uint32_t room = p.smem_ring, pair = p.unit_bytes + rec;
        const uint32_t spu = !F::kA8 && pair * 8u <= room ? 2u : 1u;
        uint32_t nr = udiv_small(room, pair * spu), nw = nr;
        if (F::kA8) {                                        // rings of their own; an even number of weight stages (see b_role_widen)
            nw = even_stages(udiv_small(room, pair), kBWStages);
            nw = nw < 4u ? 4u : nw;
            nr = udiv_small(room - nw * p.unit_bytes, rec);
        }
        nr = nr > kBRSlots ? kBRSlots : nr;
        if (!F::kA8) nw = nr;
        c.nr = nr; c.nw = nw; c.slot_bytes = rec * spu; c.spu = spu;
    }
}

// ============================================================================================= the kernel
template <int kFmt, bool kFe, bool kAsk>
__global__ void __launch_bounds__(BFmt<kFmt>::kThreadsAll, 1) batch_moe_kernel(const __grid_constant__ BParams p) {
    using F = BFmt<kFmt>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ BShared c;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~static_cast<uintptr_t>(1023u));
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, bid = blockIdx.x, G = gridDim.x;
    uint32_t* ctrl32 = reinterpret_cast<uint32_t*>(p.buf + p.off_ctrl);
    const uint32_t nent = static_cast<uint32_t>(p.T) * p.topk;
    const bool worker = warp >= kBServiceWarps && warp < kBServiceWarps + kBWorkWarps;
    const uint32_t ww = warp - kBServiceWarps;
    // ---- what needs nothing of the launches before this one: it overlaps the end of the previous kernel in the stream
    if (warp == 2) {
        if (lane < kBWStages) { mbar_init(&c.wfull[lane], 1); mbar_init(&c.wempty[lane], F::kA8 ? kBExpWarps / 2 : 1); }
        if (lane < kBRSlots) { mbar_init(&c.rfull[lane], F::kA8 ? 1 : 2); mbar_init(&c.rempty[lane], 1); }
        if (lane < 2) {
            mbar_init(&c.tmem_full[lane], 1); mbar_init(&c.tmem_empty[lane], 4);
            mbar_init(&c.xfull[lane], kBExpWarps / 2); mbar_init(&c.xempty[lane], 1);
        }
        c.task[lane] = 0u; c.task[lane + 32] = 0u;
        mbar_fence_init();
    }
    if (warp == 1) { tmem_alloc(&c.tmem_base, 512); tmem_relinquish(); tc_fence_before(); }
    if (warp < kBRankWarps) reinterpret_cast<uint32_t*>(c.wcnt[warp])[lane] = 0u;
    grid_dependency_wait();
    grid_launch_dependents();
    const unsigned long long t_first = globaltimer_ns();
    const uint32_t epoch = ld_volatile_u32(ctrl32 + kCtrlEpoch / 4 + bid);         // (tid 0 counts on after the barrier below)
    const uint32_t ntok = bid < static_cast<uint32_t>(p.T) ? udiv_small(p.T - 1u - bid, G) + 1u : 0u, nrows = ntok * p.topk;
    // a row in a warp's registers: 16 B chunks of the packed row and words of its scale bytes (hidden <= 4096)
    const uint32_t xq = p.x_row_bytes / 16u, nsf = p.x_sf_row_bytes / 4u;
    constexpr uint32_t kChunks = F::kA8 ? 8u : 4u, kWords = F::kVec == 16 ? 2u : 1u;
    constexpr uint32_t kAhead = F::kA8 ? 1u : 2u;                // rows a worker warp has in flight
    uint4 v[kAhead][kChunks];
    uint32_t vs[kAhead][kWords];
    auto load_row = [&](uint4 (&v)[kChunks], uint32_t (&vs)[kWords], uint32_t k) {
        if (k >= nrows) return;
        const uint32_t tok = bid + udiv_small(k, p.topk) * G;
        const uint8_t* xs = p.buf + p.off_x + static_cast<size_t>(tok) * p.x_row_bytes + lane * 16u;
        const uint8_t* sf = p.buf + p.off_x_sf + static_cast<size_t>(tok) * p.x_sf_row_bytes + lane * 4u;
        #pragma unroll
        for (uint32_t u = 0; u < kChunks; ++u) if (lane + u * 32u < xq) v[u] = ld_cg_v4(xs + u * 512u);
        #pragma unroll
        for (uint32_t u = 0; u < kWords; ++u) if (lane + u * 32u < nsf) vs[u] = ld_cg_u32(sf + u * 128u);
    };
    const BCtx cx(p, c, smem, globaltimer_ns() + p.timeout_ns, epoch & 1u);
    if constexpr (!kFe) {
        // ---- this SM's tokens (token mod G): the first rows of every worker warp are fetched before the routing is known
        if (worker) {
            #pragma unroll
            for (uint32_t a = 0; a < kAhead; ++a) load_row(v[a], vs[a], ww + a * kBWorkWarps);
        }
        // ---- the routing entries' experts into shared memory
        const long long* tk = reinterpret_cast<const long long*>(p.buf + p.off_topk_idx);
        #pragma unroll 4
        for (uint32_t f = tid; f < nent; f += F::kThreadsAll) {
            const long long e = tk[f];
            c.ex[f] = static_cast<uint8_t>(e < 0 ? 0xFF : (e < p.E ? static_cast<int>(e) : 0xFE));
        }
    }
    if (tid == 0) {
        c.abort_flag = 0u; c.comb_next = 0u; c.comb_open = 0u; c.wissued = 0u; c.rissued = 0u;
        // a run of 32, 64, 128 or 256 routing entries per counting warp
        const uint32_t per = (nent + kBRankWarps - 1u) / kBRankWarps;
        c.seg_shift = per <= 32u ? 5u : 32u - __clz(per - 1u);
        reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlSmEntry)[bid] = t_first;
        reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlSmPhase)[bid * kSmPhaseSlots + kSmEntry] = t_first;
        reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlSmWFirst)[bid] = ~0ull;
    }
    __syncthreads();
    tc_fence_after();
    if constexpr (kFe) {
        // ---- router frontend. All warps of all SMs work out partial logits (flagged records); SM (token mod G) then selects
        //      the token's experts as its records arrive and publishes the routing, while other warps quantise the token;
        //      every SM polls all routing records. No barrier between SMs, two exchanges through memory.
        const uint32_t flag = epoch + 1u, gw = warp * G + bid, nw = G * (F::kThreadsAll / 32);   // (consecutive items on different SMs)
        auto give_up = [&]() -> bool {
            if (cx.aborted()) return true;
            if (cx.expired()) { cx.fail(kErrWaitFrontend); return true; }
            return false;
        };
        // Items of one token where every warp gets one at most: all its loads are in flight at once up to hidden 3072, in two trips beyond (two
        // round trips less than with items of four tokens; 3 tokens 37.2 -> 35.3 us a pass, 24: 57.5 -> 55.3). Up to 24 items of four tokens per SM, one expert to an
        // item (150 tokens 72.0 -> 70.7); beyond, where the bytes count, blocks of experts (256: 79.2 -> 76.8 all in all). Two
        // more block sizes in between gained nothing: the launch pays for code that it jumps over.
        const uint32_t half_warps = kBRankWarps / 2, per = static_cast<uint32_t>(p.E) * kFeParts;
        if (per * p.T <= 16u * G) fe_logits_blocks<1, 6, 1>(p.fe, gw, nw, lane, flag);
        else if (per * ((p.T + 3u) / 4u) <= 24u * G) fe_logits_blocks<1, 3>(p.fe, gw, nw, lane, flag);
        else fe_logits_blocks<F::kA8 ? 2 : 4, 2>(p.fe, gw, nw, lane, flag);
        if (warp < half_warps) {
            #pragma unroll 1
            for (uint32_t k = warp; k < ntok; k += half_warps) {
                // the row is looked at here once more: the quantising warp would know 1.6 us
                // later (96 tokens of 3072, 128 experts: 77.3 -> 75.7 us a pass)
                const bool nz = fe_row_nonzero(p.fe.hidden + static_cast<size_t>(bid + k * G) * p.H, p.H, lane);
                if (!fe_select_token_regs<2>(p.fe, bid + k * G, nz, lane, flag, p.buf + p.off_routes, give_up)) break;
            }
        } else {
            // The other warps quantise this SM's tokens, a slice of 256 elements at a time. (A warp takes 5 to 7 us for a whole token, most of it divisions;
            // before its logits, as it once was, the records of its items came that much later: 256 tokens 86.0 -> 81.8 us, NVFP4.)
            const uint32_t nslice = static_cast<uint32_t>(p.H) / 256u, nq = F::kThreadsAll / 32 - half_warps;
            #pragma unroll 2
            for (uint32_t i = warp - half_warps; i < ntok * nslice; i += nq) {
                const uint32_t k = udiv_small(i, nslice), tok = bid + k * G;
                fe_quant_slice(p.fe.hidden + static_cast<size_t>(tok) * p.H, kFmt, p.fe.x_gs, p.buf + p.off_x + static_cast<size_t>(tok) * p.x_row_bytes,
                               p.buf + p.off_x_sf + static_cast<size_t>(tok) * p.x_sf_row_bytes, i - k * nslice, lane);
            }
        }
        #pragma unroll 1
        for (uint32_t f0 = tid; f0 < nent; f0 += 4u * F::kThreadsAll) {            // (four records per thread in flight)
            uint4 r[4];
            bool ok;
            uint32_t spins = 0;
            do {
                ok = true;
                #pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const uint32_t f = f0 + u * F::kThreadsAll;
                    if (f < nent) {
                        r[u] = ld_volatile_v4(p.buf + p.off_routes + static_cast<size_t>(f) * 16u);
                        ok = ok && r[u].y == flag && r[u].w == flag;
                    }
                }
            } while (!ok && !((++spins & 0x3Fu) == 0u && give_up()));
            #pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                const uint32_t f = f0 + u * F::kThreadsAll;
                if (f < nent) c.ex[f] = static_cast<uint8_t>(ok && r[u].x < static_cast<uint32_t>(p.E) ? r[u].x : 0xFFu);
            }
        }
        __syncthreads();
        if (bid == 0 && tid == 0) cx.stamp(kStampFrontend);
        if (worker) {
            #pragma unroll
            for (uint32_t a = 0; a < kAhead; ++a) load_row(v[a], vs[a], ww + a * kBWorkWarps);
        }
    }
    if (tid == 0) {
        ctrl32[kCtrlEpoch / 4 + bid] = epoch + 1u;
        cx.sm_phase(kSmPrologue);
        if (bid == 0) {
            ctrl32[kCtrlStatus / 4 + 1] = epoch + 1u;
            ctrl32[kCtrlStatus / 4 + 2] = 16u;                       // rows of an expert start on 16-row boundaries of the images
            ctrl32[kCtrlStatus / 4 + 3] = p.tile_limit;
            ctrl32[kCtrlStatus / 4 + 4] = kRanBatch;
            reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlStamps)[kStampEntry] = t_first;
            cx.stamp(kStampPrologue);
        }
    }
    // ---- how often each run of entries names each expert
    const uint32_t seg_shift = c.seg_shift;
    if (warp < kBRankWarps) {
        const uint32_t lo = warp << seg_shift, hi = min(lo + (1u << seg_shift), nent);
        #pragma unroll 1
        for (uint32_t f = lo + lane; f < hi; f += 32u) {
            const uint32_t e = c.ex[f];
            if (e < kMaxLocalExperts) atomicAdd(reinterpret_cast<uint32_t*>(c.wcnt[warp]) + (e >> 1), 1u << (16u * (e & 1u)));
            else if (e == 0xFEu) cx.fail(kErrWaitCombineFlag, 0xFFFFu);       // a route to an expert that does not exist
        }
    }
    __syncthreads();
    // ---- tiles. The warp that works them out is the weight loader (its stream starts when the worker warps have placed the SM's rows)
    if (warp == 0) {
        if (lane == 0) cx.sm_phase(kSmCountsKnown);
        b_tiles<kFmt>(cx, lane);
        __syncwarp();
        __threadfence_block();
        bar_arrive(kBBarTiles, F::kThreadsAll);
        if (lane == 0) { cx.sm_phase(kSmScheduled); if (bid == 0) cx.stamp(kStampScheduled); }
    } else {
        // The HBM has nothing to do until the rows are placed. While the tiles are worked out, warp 3 asks the first units of the weight tile `bid` into
        // the L2, if one of the first 128 entries names its expert: some SM's first task, this one's if no expert is empty. The loader adds as many when its
        // ring is full. (us a pass without and with both: 4 tokens 32.7, 31.6; 13 46.9, 45.6; 64 51.5, 50.5; 40 over 64 experts of 2048 x 1024 39.6, 37.5; 96
        // NVFP4 from hidden states, skewed, level. In front of the counting 64 take 50.6 and 200 tokens with every slot masked 9.3 instead of 9.2 (9.1
        // without). Longer reaches hold up the small loads of the start: 12 units here, 64 tokens 52.3 -> 53.0. Nor is there anything to gain where an SM has
        // less than two tiles: its ring holds them.)
        if (kAsk && warp == 3 && static_cast<uint32_t>(p.E) * p.n1 >= 2u * G) {
            const uint32_t e = udiv_small(bid, p.n1), left = 4u * lane < nent ? nent - 4u * lane : 0u;
            const uint32_t hit = __vcmpeq4(*reinterpret_cast<const uint32_t*>(c.ex + 4u * lane), e * 0x01010101u) & (left < 4u ? (1u << (8u * left)) - 1u : ~0u);
            if (__any_sync(0xffffffffu, hit != 0u) && lane == 0u)
                bulk_prefetch_l2(p.w1 + static_cast<size_t>(bid) * p.k1 * p.unit_bytes, (p.k1 < static_cast<int>(kBAhead) ? p.k1 : kBAhead) * p.unit_bytes);
        }
        bar_sync(kBBarTiles, F::kThreadsAll);
        if (tid == 96) cx.stamp_max(kStampLastScheduled);
    }

    const bool start = c.start_ok != 0u;
    if (warp == 3) {
        // the arrival counts of this launch's parity were cleared by the launch before it; clear the other set for the next one
        // (also when this launch has failed: the set holds the counts of the launch before)
        cx.clear_other(lane);
        if (bid == 0) {
            if (start) {
                #pragma unroll 1
                for (uint32_t e = lane; e < static_cast<uint32_t>(p.E) && p.stats != nullptr; e += 32) p.stats[e] += static_cast<int>(c.cnt[e]);
                // header line of the receive pool, for whoever inspects it afterwards
                if (lane == 0) st_ll_16B(p.buf + p.off_rx + static_cast<size_t>(cx.par) * p.rx_region, make_uint4(c.total, 0u, 0u, 0u), epoch + 1u);
            }
        }
    }
    if (worker && start) {
        // ---- copy the rows of this SM's tokens into the tiles' images, one warp per row; a warp's stores are released four
        //      rows at a time (a release waits for the stores before it: this SM's own weight stream begins behind them)
        uint32_t done_m[4], ndone = 0;
        #pragma unroll 1
        for (uint32_t k = ww; k < nrows; k += kBWorkWarps) {
            const uint32_t kt = udiv_small(k, p.topk), tok = bid + kt * G, f = tok * p.topk + k - kt * p.topk;
            const uint32_t e = c.ex[f];
            uint4 row[kChunks];
            uint32_t word[kWords];
            #pragma unroll
            for (uint32_t u = 0; u < kChunks; ++u) {
                row[u] = v[0][u];
                #pragma unroll
                for (uint32_t a = 1; a < kAhead; ++a) v[a - 1][u] = v[a][u];
            }
            #pragma unroll
            for (uint32_t u = 0; u < kWords; ++u) {
                word[u] = vs[0][u];
                #pragma unroll
                for (uint32_t a = 1; a < kAhead; ++a) vs[a - 1][u] = vs[a][u];
            }
            load_row(v[kAhead - 1u], vs[kAhead - 1u], k + kAhead * kBWorkWarps);
            if (e < kMaxLocalExperts) {
                // the expert's tile with this row
                const uint32_t pos = c.wcnt[f >> seg_shift][e] + b_rank_in_run(c, f, e, seg_shift, lane), eb = c.ebase[e];
                uint32_t m = c.etile[e];
                while (pos >= c.tile_row0[m] - eb + c.tile_rows[m]) ++m;
                const uint32_t n = pos - (c.tile_row0[m] - eb), a16 = (c.tile_rows[m] + 15u) >> 4, rec = F::rec(a16);
                uint8_t* img = p.buf + p.off_token_tiles + F::image(p.k1, c.tile_a16[m], m);
                // chunk u of a lane: 512 B further along the row, four 128 B atoms (with E4M3 two units of two atoms each, otherwise four units)
                const uint32_t at = lane >> 3;
                uint8_t* dst = img + (F::kA8 ? (at >> 1) * rec + (at & 1u) * a16 * 2048u : at * rec) + sw128_off(n, lane & 7u);
                #pragma unroll
                for (uint32_t u = 0; u < kChunks; ++u)
                    if (lane + u * 32u < xq) *reinterpret_cast<uint4*>(dst + u * (F::kA8 ? 2u : 4u) * rec) = F::kA8 ? even_odd(row[u]) : row[u];
                // scale word g: unit g / planes, plane g % planes
                #pragma unroll
                for (uint32_t u = 0; u < kWords; ++u) {
                    const uint32_t g = lane + u * 32u;
                    if (g < nsf) *reinterpret_cast<uint32_t*>(img + (g / F::kPlanes) * rec + a16 * 2048u * F::kAtoms + (g % F::kPlanes) * 512u + plane_off(n)) = word[u];
                }
                #pragma unroll
                for (uint32_t q = 0; q < 4; ++q) if (q == ndone) done_m[q] = m;
                ++ndone;
            }
            if (ndone == 4u || (ndone != 0u && k + kBWorkWarps >= nrows)) {
                __syncwarp();
                if (lane == 0) {
                    fence_acq_rel_gpu();             // (the reader's proxy fence after its acquire orders these stores with its bulk copies)
                    #pragma unroll
                    for (uint32_t q = 0; q < 4; ++q) if (q < ndone) atomicAdd(cx.counter(cx.par, kBCountTiles + done_m[q]), 1u);
                }
                ndone = 0u;
            }
        }
        bar_arrive(kBBarPlaced, 32u * (kBWorkWarps + 1));        // (the weight loader)
        if (lane == 0) cx.sm_phase(kSmRowsCached);
        // ---- the list of rows, for the epilogue
        #pragma unroll 1
        for (uint32_t r = ww; r < kBRankWarps; r += kBWorkWarps) b_list_run(cx, r, seg_shift, nent, lane);
        bar_sync(kBBarWork, kBWorkWarps * 32u);
        // ---- the rows' records in the receive pool (a row's place: the live entries before it), for whoever inspects the pool
        //      afterwards. With 4-bit tokens these warps only wait for the combine; with E4M3 tokens they are the widening group of
        //      the first unit, which waits for the records.
        if (warp >= kBServiceWarps + kBEpiWarps) {
            #pragma unroll 1
            for (uint32_t k = ww - kBEpiWarps; k < nrows; k += kBWorkWarps - kBEpiWarps) {
                const uint32_t kt = udiv_small(k, p.topk), tok = bid + kt * G, slot = k - kt * p.topk, f = tok * p.topk + slot;
                const uint32_t e = c.ex[f];
                if (e >= kMaxLocalExperts) continue;
                uint32_t li = 0u;
                #pragma unroll 1
                for (uint32_t i = lane * 4u; i < f; i += 128u) {
                    const uint32_t w = *reinterpret_cast<const uint32_t*>(c.ex + i);
                    #pragma unroll
                    for (uint32_t b = 0; b < 4; ++b) li += (i + b < f && ((w >> (8u * b)) & 0xFFu) < kMaxLocalExperts) ? 1u : 0u;
                }
                li = __reduce_add_sync(0xffffffffu, li);
                if (lane == 0)
                    st_ll_16B(p.buf + p.off_rx + static_cast<size_t>(cx.par) * p.rx_region + 32u + static_cast<size_t>(li) * 2u * p.rx_row_bytes + 2u * (p.rx_row_bytes - 16u),
                              make_uint4(e, tok, slot, kFe ? ld_cg_u32(p.buf + p.off_routes + static_cast<size_t>(f) * 16u + 8u)
                                                   : __float_as_uint(reinterpret_cast<const float*>(p.buf + p.off_topk_w)[f])), epoch + 1u);
            }
        }
    }

    // ---- roles
    if (start) {
        if (warp == 0) b_role_weights<F::kA8, kAsk>(cx, lane);
        else if (warp == 1) b_role_mma<kFmt>(cx, lane);
        else if (warp == 2) b_role_records<kFmt>(cx);
        else if (warp >= kBServiceWarps && warp < kBServiceWarps + kBEpiWarps)
            b_role_epilogue<kFmt, kFe>(cx, (warp - kBServiceWarps) >> 2, tid - 32u * kBServiceWarps - ((warp - kBServiceWarps) >> 2) * 128u);
        else if (warp >= kBServiceWarps + kBEpiWarps) {
            if constexpr (F::kA8) { const uint32_t x = tid - 32u * (kBServiceWarps + kBEpiWarps); b_role_widen(cx, x / kXGroupThreads, x % kXGroupThreads); }
        }
    }
    if (tid == 128) { cx.stamp_max(kStampLastTasksDone); cx.sm_phase(kSmTasksDone); if (bid == 0) cx.stamp(kStampTasksDone); }
    if (!cx.aborted()) b_role_combine(cx, lane);
    // ---- exit: an aborted SM lets the copies in flight land (bounded waits) before its shared memory goes away
    // (both loaders count into the stages' barriers: a stage that only one of them has filled never completes, so the
    // wait is also bounded in time)
    if (cx.aborted() && (warp == 0 || warp == 2)) {
        const bool w = warp == 0;
        const uint32_t issued = *reinterpret_cast<volatile uint32_t*>(w ? &c.wissued : &c.rissued), nst = w ? c.nw : c.nr;
        uint64_t* bars = w && F::kA8 ? c.wfull : c.rfull;
        #pragma unroll 1
        for (uint32_t k = issued > nst ? issued - nst : 0u; k < issued; ++k)
            for (uint32_t spin = 0; spin < 2000u && !mbar_try_wait(&bars[k % nst], (k / nst) & 1u); ++spin) { }
        for (uint32_t spin = 0; spin < 2000u; ++spin) __nanosleep(100);          // (copies of some 10 KB: microseconds at most)
    }
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(c.tmem_base, 512); }
    if (tid == 0) { if (bid == 0) cx.stamp(kStampExit); cx.stamp_max(kStampLastExit); cx.sm_phase(kSmExit); }
}

}  // namespace mm
