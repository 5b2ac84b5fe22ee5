// The layer on one rank with at most 16 routing entries (decode), as one persistent sm_100a kernel of its own.
//
// The launch is a chain of short steps around 50 MB of weights (8 us of HBM time for one token and eight experts), so what
// counts is the number of steps and what one costs:
//   * Every SM reads the routing entries and sorts them itself (one warp, registers), starts its weight stream right away,
//     and builds ONE token tile of all 16 rows in shared memory (rows grouped by expert), which every task multiplies with:
//     D[128 weight rows x 16 rows]; a task's epilogue looks at its expert's columns.
//   * L1 weight tiles are dealt round-robin; the remainder tiles are cut along K between fixed groups of SMs, so that every SM
//     streams the same number of units. The parts come first; the group's first SM adds the others' sums in SM order.
//   * What one SM hands to another (parts, intermediate rows, expert outputs) are flagged 8-byte words {data, launch number}
//     that the consumer polls: one trip through the L2, no fence, no counter. All SMs gather all intermediate rows (a few KB)
//     into the L2 tasks' token tile while the L2 weights are already in the ring.
//   * From hidden states: the router's partial logits are spread over the SMs as flagged records, then every SM selects for and
//     quantises the (one or two) tokens by itself: one exchange instead of two.
//   * Little code: what runs once per launch is fetched cold, and long unrolled pieces cost more than they save.
// Bound: latency. One token over eight experts of the benchmark's layer: 18.4 us a pass, of which the weight stream is about half.
#pragma once
#include "mm_batch.cuh"

namespace mm {

constexpr uint32_t kDEntries = 16;                 // routing entries (= rows) of a launch at most
constexpr int kDEpiWarps = 8;                      // warps 4..11: build the token tiles, two epilogue groups
constexpr int kDThreads = 32 * (4 + kDEpiWarps);
constexpr int kDThreadsA8 = kDThreads + 32 * kBExpWarps;     // E4M3 tokens: widening warps 12..19
constexpr int kDStages = 12;
constexpr uint32_t kDBarGroups = 5, kDBarRouted = 6;
// tensor-memory columns with E4M3 tokens: behind the two accumulators the scales of the weights and of the tokens (8 each) and the widened units (64 each).
// Four units: the widening runs ahead of the MMAs, which take two at a turn (two tokens 28.3 -> 27.9 us a pass against two units, one at a turn).
// In the batch kernel, whose accumulators leave room for four too, that gained nothing (100 tokens 68.4, 69.1).
constexpr uint32_t kDWide = 4, kDTmScaleW = 64, kDTmScaleX = kDTmScaleW + kDWide * 8, kDTmWide = 128;

struct DShared {
    uint64_t wfull[kDStages], wempty[kDStages];
    uint64_t tmem_full[2], tmem_empty[2], xfull[kDWide], xempty[kDWide], tile_full[2];
    uint32_t tmem_base, abort_flag, comb_next, wissued, M, nlive, live_mask, start_ok;
    uint32_t split_t, split_range, split_first, split_parts;      // this SM's part of a remainder tile: tile, first unit | end unit << 8, first SM of the group, parts (0: none)
    uint32_t exp_e[kDEntries], exp_c0[kDEntries], exp_n[kDEntries];    // active experts, ascending: id, first column, rows
    alignas(16) uint32_t ent_e[kDEntries]; float ent_w[kDEntries];   // per routing entry: expert (>= 64: none), weight
    uint32_t ent_col[kDEntries];                                    // column of the entry's row in the token tile
    uint32_t col_f[kDEntries], col_mid[kDEntries]; float col_w[kDEntries];   // per column: entry, row of the intermediate pool, weight
    float vt[2][kTileTokens * kBVtStride];
};

struct DCtx : BCore {
    DShared& c;
    __device__ __forceinline__ DCtx(const BParams& p_, DShared& c_, uint8_t* smem_, uint64_t deadline_, uint32_t par_)
        : BCore{p_, &c_.abort_flag, smem_, deadline_, par_}, c(c_) {}
};

template <int kFmt> struct DFmt : BFmt<kFmt> {
    static constexpr int kThreads = BFmt<kFmt>::kA8 ? kDThreadsA8 : kDThreads;
    static constexpr uint32_t kBuilders = BFmt<kFmt>::kA8 ? kDEpiWarps + kBExpWarps : kDEpiWarps;    // warps from 4 on that build the first token tile
    static constexpr uint32_t kTmemColumns = BFmt<kFmt>::kA8 ? 512u : 128u;
    static constexpr uint32_t kRec = 2048u * BFmt<kFmt>::kAtoms + BFmt<kFmt>::kPlanes * 512u;     // one K unit of the 16-row tile
};

// task `ti` of this SM: its part of a remainder L1 tile, its whole L1 tiles, its L2 tiles
struct DTask { uint32_t layer, a, j, ub, ue, parts; bool valid; };
struct DTasks {
    const DCtx& cx;
    uint32_t has_split, my1, r1;
    __device__ __forceinline__ explicit DTasks(const DCtx& c_) : cx(c_) {
        const uint32_t NT1 = c_.c.M * c_.p.n1, G = gridDim.x;
        r1 = NT1 - udiv_small(NT1, G) * G;
        has_split = c_.c.split_parts != 0u ? 1u : 0u;
        my1 = r1 + blockIdx.x < NT1 ? udiv_small(NT1 - 1u - r1 - blockIdx.x, G) + 1u : 0u;
    }
    __device__ __forceinline__ DTask get(uint32_t ti) const {
        DTask t;
        const uint32_t G = gridDim.x;
        t.layer = 0u; t.ub = 0u; t.ue = cx.p.k1; t.parts = 1u; t.valid = true;
        uint32_t x;
        if (ti < has_split) { x = cx.c.split_t; t.ub = cx.c.split_range & 0xFFu; t.ue = cx.c.split_range >> 8; t.parts = cx.c.split_parts; }
        else if (ti < has_split + my1) x = r1 + blockIdx.x + (ti - has_split) * G;
        else {
            x = blockIdx.x + (ti - has_split - my1) * G;
            t.layer = 1u; t.ue = cx.p.k2;
            t.valid = x < cx.c.M * cx.p.n2;
        }
        const uint32_t n = t.layer ? cx.p.n2 : cx.p.n1;
        t.a = t.valid ? udiv_small(x, n) : 0u;
        t.j = x - t.a * n;
        return t;
    }
};

// `first` is called once: when the first unit has been asked for, or (false) on an SM without any.
template <typename First>
__device__ __forceinline__ void d_role_weights(const DCtx& cx, uint32_t nw, uint8_t* ring, First first) {
    const BParams& p = cx.p; DShared& c = cx.c;
    const uint64_t policy = l2_evict_first_policy();
    uint32_t it = 0, s = 0, ph = 0;
    DTasks tasks(cx);
    #pragma unroll 1
    for (uint32_t ti = 0;; ++ti) {
        const DTask t = tasks.get(ti);
        if (!t.valid) break;
        const uint8_t* src = (t.layer ? p.w2 : p.w1) +
            ((static_cast<size_t>(c.exp_e[t.a]) * (t.layer ? p.n2 : p.n1) + t.j) * (t.layer ? p.k2 : p.k1) + t.ub) * p.unit_bytes;
        #pragma unroll 1
        for (uint32_t u = t.ub; u < t.ue; ++u, ++it, src += p.unit_bytes) {
            if (!cx.warp_wait(&c.wempty[s], ph ^ 1u, kErrWaitEmpty)) return;
            if (elect_one()) {
                mbar_arrive_expect_tx(&c.wfull[s], p.unit_bytes);
                bulk_g2s_hint(ring + static_cast<size_t>(s) * p.unit_bytes, src, p.unit_bytes, &c.wfull[s], policy);
                c.wissued = it + 1u;
            }
            __syncwarp();
            if (it == 0u) first(true);
            if (++s == nw) { s = 0; ph ^= 1u; }
        }
    }
    if (it == 0u) first(false);
}

template <int kFmt>
__device__ void d_role_mma(const DCtx& cx, uint32_t lane, uint32_t nw_, uint32_t ring_off) {
    using F = DFmt<kFmt>;
    constexpr bool kA8 = F::kA8;
    constexpr uint32_t kPlanes = F::kPlanes, kStepK = kA8 ? 32u : 64u;
    constexpr uint32_t kIdesc = kA8 ? idesc_block_scaled(kFmtF8E2M1, kFmtF8E4M3, 128u, kTileTokens, 1u)
                                    : idesc_block_scaled(kFmtMxf4E2M1, kFmtMxf4E2M1, 128u, kTileTokens, kFmt == 1 ? 0u : 1u);
    const BParams& p = cx.p; DShared& c = cx.c;
    // (operands broadcast from lane 0: uniform registers, see the batch kernel's issuer)
    const uint32_t nw = b_uniform(nw_), tm = b_uniform(c.tmem_base);
    const uint32_t s0 = b_uniform(smem_u32(cx.smem)), ring0 = s0 + b_uniform(ring_off);
    uint32_t it = 0, s = 0, ph = 0;
    bool have1 = false, have2 = false;
    DTasks tasks(cx);
    #pragma unroll 1
    for (uint32_t ti = 0;; ++ti) {
        const DTask t = tasks.get(ti);
        if (!b_uniform(t.valid ? 1u : 0u)) break;
        const uint32_t layer = b_uniform(t.layer), ub = b_uniform(t.ub), ue = b_uniform(t.ue);
        const uint32_t acc = ti & 1u, use = (ti >> 1) & 1u, d = tm + acc * 16u;
        if (!cx.warp_wait(&c.tmem_empty[acc], use ^ 1u, kErrWaitTmemEmpty)) return;
        if (layer == 0u && !have1) { if (!cx.warp_wait(&c.tile_full[0], 0u, kErrWaitActsFull)) return; have1 = true; }
        if (layer != 0u && !have2) { if (!cx.warp_wait(&c.tile_full[1], 0u, kErrWaitL1Done)) return; have2 = true; }
        tc_fence_after();
        // A stage that is there already goes out in the same turn: a turn is a barrier wait, a fence, an election and a reconvergence beside
        // the issue, 540 to 640 cycles for a unit that the tensor pipe has in 200 (one token 20.6 -> 20.4 us a pass, two 27.2
        // -> 26.7; four stages a turn no better).
        #pragma unroll 1
        for (uint32_t u = ub; u < ue;) {
            if (!cx.warp_wait(kA8 ? &c.xfull[it % kDWide] : &c.wfull[s], kA8 ? (it / kDWide) & 1u : ph, kErrWaitFull)) return;
            const uint32_t s1 = s + 1u == nw ? 0u : s + 1u;
            const bool next = u + 1u < ue && (kA8 ? mbar_test(&c.xfull[(it + 1u) % kDWide], ((it + 1u) / kDWide) & 1u) : mbar_test(&c.wfull[s1], s1 == 0u ? ph ^ 1u : ph));
            const uint32_t n = __all_sync(0xffffffffu, next) ? 2u : 1u;
            tc_fence_after();
            if (lane == 0 && it == 0u) cx.sm_phase(kSmFirstLanded);
            if (elect_one()) {
                #pragma unroll 1
                for (uint32_t b = 0; b < n; ++b) {
                    const uint32_t slot = b == 0u ? s : s1, i = it + b, wsm = ring0 + slot * p.unit_bytes, tok = s0 + (u + b) * F::kRec;
                    const uint64_t adesc = smem_desc(wsm, 1024u, kLayoutSw128), bdesc = smem_desc(tok, 1024u, kLayoutSw128);
                    const uint64_t asf = smem_desc(wsm + kUnitWBytes, 128u, kLayoutNone);
                    const uint64_t bsf = smem_desc(tok + 2048u * F::kAtoms, 128u, kLayoutNone);
                    const uint32_t sfa = kA8 ? tm + kDTmScaleW + (i % kDWide) * 8u : tm + 32u + (i & 1u) * 32u, sfb = kA8 ? tm + kDTmScaleX + (i % kDWide) * 8u : sfa + 16u;
                    const uint32_t wide = tm + kDTmWide + (i % kDWide) * 64u;
                    #pragma unroll
                    for (uint32_t pl = 0; pl < kPlanes; ++pl) {
                        if constexpr (!kA8) utccp_32x128b_warpx4(sfa + pl * 4u, asf + pl * 32u);
                        utccp_32x128b_warpx4(sfb + pl * 4u, bsf + pl * 32u);
                    }
                    #pragma unroll
                    for (uint32_t ks = 0; ks < kUnitK / kStepK; ++ks) {
                        const uint32_t pl = (ks * kStepK) / (4u * F::kVec), sf_id = ((ks * kStepK) % (4u * F::kVec)) / F::kVec;
                        const uint64_t ad = adesc + (ks & 3u) * 2u;
                        const uint64_t bd = bdesc + (ks & 3u) * 2u + (kA8 ? (ks >> 2) * (2048u >> 4) : 0u);
                        const uint32_t idesc = idesc_with_sf(kIdesc, sf_id, sf_id), accum = (u + b != ub || ks != 0u) ? 1u : 0u;
                        if constexpr (kA8) umma_mxf8f6f4_ta(d, wide + ks * 8u, bd, idesc, sfa + pl * 4u, sfb + pl * 4u, accum);
                        else if constexpr (kFmt == 0) umma_mxf4_block32(d, ad, bd, idesc, sfa + pl * 4u, sfb + pl * 4u, accum);
                        else umma_nvf4_block16(d, ad, bd, idesc, sfa + pl * 4u, sfb + pl * 4u, accum);
                    }
                    tc_commit(kA8 ? &c.xempty[i % kDWide] : &c.wempty[slot]);
                }
            }
            __syncwarp();
            u += n; it += n; s += n;
            if (s >= nw) { s -= nw; ph ^= 1u; }
        }
        if (elect_one()) tc_commit(&c.tmem_full[acc]);
        __syncwarp();
    }
    if (lane == 0 && it != 0u) cx.stamp_max(kStampLastWeight);
}

// The widening warps' loop (E4M3 tokens, see b_role_widen) over this kernel's tasks; the ring is even here too.
__device__ void d_role_widen(const DCtx& cx, uint32_t grp, uint32_t xtid, uint32_t nw, const uint8_t* ring) {
    const BParams& p = cx.p; DShared& c = cx.c;
    const uint32_t lane = xtid & 31u;
    const uint32_t tm = c.tmem_base + ((xtid & 96u) << 16);
    uint32_t it = 0, s = 0, ph = 0;
    DTasks tasks(cx);
    #pragma unroll 1
    for (uint32_t ti = 0;; ++ti) {
        const DTask t = tasks.get(ti);
        if (!t.valid) break;
        #pragma unroll 1
        for (uint32_t u = t.ub; u < t.ue; ++u, ++it) {
            if ((it & 1u) == grp) {
                if (!cx.warp_wait(&c.wfull[s], ph, kErrWaitFull)) return;
                BWiden w;
                w.load(ring + static_cast<size_t>(s) * p.unit_bytes, xtid);
                __syncwarp();
                if (lane == 0) mbar_arrive(&c.wempty[s]);
                const uint32_t x = it % kDWide;                  // (always one of this group's)
                if (!cx.warp_wait(&c.xempty[x], ((it / kDWide) & 1u) ^ 1u, kErrWaitEmpty)) return;
                tc_fence_after();
                w.store(tm + kDTmWide + x * 64u, tm + kDTmScaleW + x * 8u);
                __syncwarp();
                if (lane == 0) mbar_arrive(&c.xfull[x]);
            }
            if (++s == nw) { s = 0; ph ^= 1u; }
        }
    }
}

// Intermediate rows of all experts -> the token tile of the L2 tasks (both epilogue groups, after the SM's last L1 task: its
// MMAs on the tokens' tile, whose place this one takes, are over). Payload in 8-byte pieces (one 16 B load of two flagged words), then the scale words.
template <int kFmt>
__device__ __forceinline__ bool d_gather(const DCtx& cx, uint8_t* tile, uint32_t gtid) {
    using F = DFmt<kFmt>;
    const BParams& p = cx.p; DShared& c = cx.c;
    constexpr uint32_t kThreads = kDEpiWarps * 32, kFly = 3;
    const uint32_t flag = *reinterpret_cast<volatile uint32_t*>(&c.start_ok), pieces = p.mid_row_bytes / 8u, n = c.nlive * pieces;   // (start_ok holds the launch's flag)
    uint32_t spins = 0;
    #pragma unroll 1
    for (uint32_t i0 = gtid; i0 < n; i0 += kThreads * kFly) {
        uint4 v[kFly];
        bool ok;
        const uint8_t* src[kFly];
        #pragma unroll
        for (uint32_t u = 0; u < kFly; ++u) {
            const uint32_t i = i0 + u * kThreads, col = udiv_small(i < n ? i : 0u, pieces), pc = (i < n ? i : 0u) - col * pieces;
            src[u] = p.buf + p.off_mid + static_cast<size_t>(c.col_mid[col]) * 2u * p.mid_row_bytes + pc * 16u;
            v[u] = make_uint4(0u, flag ^ 1u, 0u, flag ^ 1u);
        }
        do {                                             // (only the missing ones again: polls of all of them slowed the last L1 tasks and the stream, 21.4 -> 20.6 us for one token)
            #pragma unroll
            for (uint32_t u = 0; u < kFly; ++u) if (i0 + u * kThreads < n && (v[u].y != flag || v[u].w != flag)) v[u] = ld_volatile_v4(src[u]);
            ok = true;
            #pragma unroll
            for (uint32_t u = 0; u < kFly; ++u) ok = ok && (i0 + u * kThreads >= n || (v[u].y == flag && v[u].w == flag));
            if (!ok && cx.give_up(spins, kErrWaitL1Done, 0u)) return false;
        } while (!ok);
        #pragma unroll
        for (uint32_t u = 0; u < kFly; ++u) {
            const uint32_t i = i0 + u * kThreads;
            if (i < n) {
                const uint32_t col = udiv_small(i, pieces), pc = i - col * pieces, ci = pc >> 1, at = ci >> 3;       // 16 B chunk, 128 B atom of the row
                uint8_t* dst = tile + (F::kA8 ? (at >> 1) * F::kRec + (at & 1u) * 2048u : at * F::kRec) + sw128_off(col, ci & 7u) + (pc & 1u) * 8u;
                *reinterpret_cast<uint2*>(dst) = F::kA8 ? even_odd(v[u].x, v[u].z) : make_uint2(v[u].x, v[u].z);
            }
        }
    }
    #pragma unroll 1
    for (uint32_t i = gtid; i < c.nlive * p.n1; i += kThreads) {
        const uint32_t col = udiv_small(i, p.n1), j = i - col * p.n1;
        const uint8_t* src = p.buf + p.off_mid_sf + (static_cast<size_t>(c.col_mid[col]) * p.n1 + j) * 8u;
        uint2 q = ld_volatile_v2(src);
        while (q.y != flag) {
            if (cx.give_up(spins, kErrWaitL1Done, 0u)) return false;
            q = ld_volatile_v2(src);
        }
        uint8_t* sf = tile + (j >> 2) * F::kRec + 2048u * F::kAtoms + plane_off(col);
        if constexpr (F::kVec == 16) *reinterpret_cast<uint32_t*>(sf + (j & 3u) * 512u) = q.x;
        else *reinterpret_cast<uint16_t*>(sf + ((j >> 1) & 1u) * 512u + (j & 1u) * 2u) = static_cast<uint16_t>(q.x);
    }
    return true;
}

template <int kFmt>
__device__ void d_role_epilogue(const DCtx& cx, uint32_t grp, uint32_t etid, uint8_t* tile, uint32_t flag) {
    using F = DFmt<kFmt>;
    constexpr bool kA8 = F::kA8;
    constexpr int kVec = F::kVec;
    const BParams& p = cx.p; DShared& c = cx.c;
    const uint32_t ew = etid >> 5, q = etid & 7u, n = etid >> 3, bar = grp ? kBBarEpi1 : kBBarEpi0;
    float* vt = c.vt[grp];
    float* vt_w = vt + ((etid & 15u) >> 2) * 40u + (etid >> 4) * 4u + (etid & 3u);
    const float* vt_r = vt + n * kBVtStride + q * 4u;
    DTasks tasks(cx);
    bool gathered = false, bad = false;
    #pragma unroll 1
    for (uint32_t ti = grp;; ti += 2) {
        const DTask t = tasks.get(ti);
        // The second token tile, when this group meets its first L2 task (or has no further task, or has failed): the other group does the same.
        // (One place for it: the code of the gather is fetched once per launch, mostly cold.)
        if ((bad || !t.valid || t.layer != 0u) && !gathered) {
            gathered = true;
            // (both groups are past their L1 tasks: nothing reads the first tile any more; they leave together if one has failed)
            if (bar_red_or(kDBarGroups, kDEpiWarps * 32u, bad)) return;
            const bool ok = d_gather<kFmt>(cx, tile, grp * 128u + etid);
            fence_proxy_async_smem();
            const bool all_ok = __all_sync(0xffffffffu, ok);
            if ((etid & 31u) == 0u && all_ok) mbar_arrive(&c.tile_full[1]);
            if (grp == 0u && etid == 0u) cx.sm_phase(kSmFirstL2Staged);
            if (bar_red_or(bar, 128u, !all_ok)) return;
        }
        if (bad || !t.valid) break;
        const uint32_t use = (ti >> 1) & 1u, c0 = c.exp_c0[t.a], nv = c.exp_n[t.a];
        const bool ok = cx.warp_wait(&c.tmem_full[grp], use, kErrWaitTmemFull);
        tc_fence_after();
        uint32_t raw[kTileTokens];
        if (ok) {
            tmem_ld_32x32b_x16(c.tmem_base + ((ew * 32u) << 16) + grp * 16u, raw);
            tmem_ld_wait();
            tc_fence_before();
        }
        __syncwarp();
        if ((etid & 31u) == 0u) mbar_arrive(&c.tmem_empty[grp]);
        if (bar_red_or(bar, 128u, !ok)) { bad = true; continue; }
        #pragma unroll
        for (uint32_t i = 0; i < kTileTokens; ++i) vt_w[i * kBVtStride] = __uint_as_float(raw[i]);
        if (ti < 2u && etid == 0u) cx.sm_phase(kSmFirstMmaDone);
        if (t.parts > 1u) {
            // A part of a remainder tile: [part SM][row of the expert][weight row] flagged fp32 words; the group's first SM adds.
            const uint32_t first = c.split_first;
            auto part_word = [&](uint32_t sm, uint32_t i) { return p.buf + p.off_parts + ((static_cast<size_t>(sm) * kDEntries + i) * kTileRows + etid) * 8u; };
            if (blockIdx.x != first) {
                #pragma unroll 1
                for (uint32_t i = 0; i < nv; ++i) st_volatile_v2(part_word(blockIdx.x, i), __float_as_uint(vt_w[(c0 + i) * kBVtStride]), flag);
                continue;                                            // (each thread wrote and read its own words of vt)
            }
            bool got = true;
            uint32_t spins = 0;
            #pragma unroll 1
            for (uint32_t i = 0; i < nv && got; ++i) {
                float sum = 0.f + vt_w[(c0 + i) * kBVtStride];
                #pragma unroll 1
                for (uint32_t p0 = 1; p0 < t.parts && got; p0 += 8) {        // eight parts' words in flight, added in SM order
                    uint2 w[8];
                    bool all;
                    do {
                        all = true;
                        #pragma unroll
                        for (uint32_t u = 0; u < 8; ++u)
                            if (p0 + u < t.parts) { w[u] = ld_volatile_v2(part_word(first + p0 + u, i)); all = all && w[u].y == flag; }
                        if (!all && cx.give_up(spins, kErrWaitL1Done, 1u)) got = false;
                    } while (!all && got);
                    #pragma unroll
                    for (uint32_t u = 0; u < 8; ++u) if (p0 + u < t.parts) sum += __uint_as_float(w[u].x);
                }
                vt_w[(c0 + i) * kBVtStride] = sum;
            }
            if (bar_red_or(bar, 128u, !got)) { bad = true; continue; }
        } else bar_sync(bar, 128u);
        float a[16];
        #pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(vt_r + i * 40u);
            a[4 * i] = v.x; a[4 * i + 1] = v.y; a[4 * i + 2] = v.z; a[4 * i + 3] = v.w;
        }
        const bool live = n - c0 < nv;
        if (t.layer == 0u) {
            float o[8];
            uint32_t sfw;
            b_swiglu(p, a, live ? c.col_w[n] : 0.f, live, o);
            b_requantise<kFmt>(p, o, live, sfw);
            if (live) {
                const size_t row = c.col_mid[n];
                uint8_t* dst = p.buf + p.off_mid + row * 2u * p.mid_row_bytes + (t.j * 8u + q) * (kA8 ? 16u : 8u);
                if constexpr (kA8) {
                    const uint32_t w0 = cvt_e4m3x2(o[0], o[1]) | (cvt_e4m3x2(o[2], o[3]) << 16), w1 = cvt_e4m3x2(o[4], o[5]) | (cvt_e4m3x2(o[6], o[7]) << 16);
                    st_ll_half(dst, make_uint4(w0, w1, 0u, 0u), flag, 0u);
                } else {
                    st_volatile_v2(dst, cvt_e2m1x2(o[0], o[1]) | (cvt_e2m1x2(o[2], o[3]) << 8) | (cvt_e2m1x2(o[4], o[5]) << 16) | (cvt_e2m1x2(o[6], o[7]) << 24), flag);
                }
                if (q == 0u) st_volatile_v2(p.buf + p.off_mid_sf + (row * p.n1 + t.j) * 8u, kVec == 16 ? sfw : sfw & 0xFFFFu, flag);
            }
            if (etid == 0u) cx.sm_phase(kSmLastL1Epilogue);
        } else if (live) {
            uint32_t w[8];
            #pragma unroll
            for (uint32_t i = 0; i < 8; ++i)
                w[i] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(a[2 * i] * p.l2_scale))) |
                       (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(a[2 * i + 1] * p.l2_scale))) << 16);
            uint8_t* dst = p.buf + p.off_comb + (static_cast<size_t>(c.col_f[n]) * p.H + t.j * 128u + q * 16u) * 4u;
            const uint32_t lo[8] = {w[0], flag, w[1], flag, w[2], flag, w[3], flag}, hi[8] = {w[4], flag, w[5], flag, w[6], flag, w[7], flag};
            st_global_v8(dst, lo);
            st_global_v8(dst + 32, hi);
        }
        if (ti < 2u && etid == 0u) cx.sm_phase(kSmFirstEpilogue);
        bar_sync(bar, 128u);                                         // (the reads of vt are over)
    }
}

// Items (token, eight columns). A lane polls one route of its item, 1 to 8 neighbouring lanes (a power of two, at most the routes) an
// item; when their flagged words are there every lane of the item has them by shuffles and adds them in slot order. (A lane that polled all routes
// of its item, 16 loads at a time, saw the last words 2.5 us after they were stored, 4 at worst: one token 20.5 -> 18.3 us a pass, two E4M3
// tokens 30.6 -> 28.0, two of four routes over a small layer 12.2 -> 11.1.)
__device__ void d_role_combine(const DCtx& cx, uint32_t flag, uint32_t lane) {
    const BParams& p = cx.p; DShared& c = cx.c;
    const uint32_t G = gridDim.x, per = p.H / 8u, nitems = static_cast<uint32_t>(p.T) * per;
    const uint32_t shift = p.topk >= 8 ? 3u : (p.topk >= 4 ? 2u : (p.topk >= 2 ? 1u : 0u)), L = 1u << shift, sub = lane & (L - 1u);
    uint32_t spins = 0;
    #pragma unroll 1
    for (;;) {
        uint32_t k = 0u;
        if (lane == 0u) k = atomicAdd(&c.comb_next, 32u >> shift);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (blockIdx.x + k * G >= nitems) return;
        const uint32_t idx = blockIdx.x + (k + (lane >> shift)) * G;
        const bool valid = idx < nitems;
        const uint32_t tok = udiv_small(valid ? idx : 0u, per), ch = (valid ? idx : 0u) - tok * per;
        const uint32_t mask = valid ? (c.live_mask >> (tok * p.topk)) & ((1u << p.topk) - 1u) : 0u;
        const uint8_t* base = p.buf + p.off_comb + (static_cast<size_t>(tok) * p.topk * p.H + ch * 8u) * 4u;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        #pragma unroll 1
        for (uint32_t s0 = 0; s0 < static_cast<uint32_t>(p.topk); s0 += L) {
            const bool mine = ((mask >> (s0 + sub)) & 1u) != 0u;
            const uint8_t* src = base + static_cast<size_t>(s0 + sub) * p.H * 4u;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            bool ok = !mine;
            for (;;) {
                if (!ok) {
                    const uint4 a = ld_volatile_v4(src), b = ld_volatile_v4(src + 16);
                    ok = ll_valid(a, b, flag);
                    v = ll_data(a, b);
                }
                if (__all_sync(0xffffffffu, ok)) break;
                if (__any_sync(0xffffffffu, !ok && cx.give_up(spins, kErrWaitCombineFlag, tok))) return;
            }
            #pragma unroll 1
            for (uint32_t s = 0; s < L; ++s) {
                const uint32_t from = (lane & ~(L - 1u)) + s;
                const uint32_t w[4] = {__shfl_sync(0xffffffffu, v.x, from), __shfl_sync(0xffffffffu, v.y, from),
                                       __shfl_sync(0xffffffffu, v.z, from), __shfl_sync(0xffffffffu, v.w, from)};
                #pragma unroll
                for (int i = 0; i < 4; ++i) { acc[2 * i] += __uint_as_float(w[i] << 16); acc[2 * i + 1] += __uint_as_float(w[i] & 0xFFFF0000u); }
            }
        }
        uint4 o;
        uint32_t* ow = &o.x;
        #pragma unroll
        for (int i = 0; i < 4; ++i)
            ow[i] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(acc[2 * i]))) |
                    (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(acc[2 * i + 1]))) << 16);
        if (valid && sub == 0u) *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.y) + (static_cast<size_t>(tok) * p.H + ch * 8u) * 2u) = o;
        if (lane == 0u) {
            if (k == 0u) cx.sm_phase(kSmFirstCombined);
            cx.sm_phase(kSmCombineDone);
        }
    }
}

// Sorts the routing entries by (expert, entry) and derives this SM's part of a remainder tile (one warp; lane i holds entry i).
__device__ __forceinline__ void d_route(const DCtx& cx, uint32_t e, float w, uint32_t n, uint32_t lane) {
    const BParams& p = cx.p; DShared& c = cx.c;
    const bool live = lane < n && e < kMaxLocalExperts;
    if (__any_sync(0xffffffffu, lane < n && e == 0xFEu)) { if (lane == 0) cx.fail(kErrWaitCombineFlag, 0xFFFFu); }   // a route to an expert that does not exist
    if (static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, live))) > p.cap_rows) { if (lane == 0) cx.fail(kErrMetaCapacity, 0u); }     // (more rows than the receive pool has room for)
    const uint32_t key = live ? e : 0xFFu;
    if (lane < kDEntries) c.ent_e[lane] = key;
    __syncwarp();
    // every lane compares its entry with all of them: plain arithmetic on four 16-byte reads (votes and shuffles, one of each per entry, took 0.5 us, and
    // 3 to 5 us in the E4M3 kernel from hidden states)
    uint32_t keys[kDEntries];
    #pragma unroll
    for (uint32_t i = 0; i < kDEntries; i += 4) {
        const uint4 q = *reinterpret_cast<const uint4*>(c.ent_e + i);
        keys[i] = q.x; keys[i + 1] = q.y; keys[i + 2] = q.z; keys[i + 3] = q.w;
    }
    uint32_t below = 0u, pos = 0u, rows = 0u, group = 0u;            // rows of smaller experts, earlier rows of this one, all of its rows; smaller experts
    #pragma unroll
    for (uint32_t i = 0; i < kDEntries; ++i) {
        below += keys[i] < key ? 1u : 0u;
        rows += keys[i] == key ? 1u : 0u;
        pos += (keys[i] == key && i < lane) ? 1u : 0u;
    }
    const uint32_t live_mask = __ballot_sync(0xffffffffu, live), firsts = __ballot_sync(0xffffffffu, live && pos == 0u), M = __popc(firsts);
    #pragma unroll
    for (uint32_t i = 0; i < kDEntries; ++i) group += (keys[i] < key && ((firsts >> i) & 1u) != 0u) ? 1u : 0u;
    if (live) {
        const uint32_t col = below + pos;
        c.ent_col[lane] = col;
        c.col_f[col] = lane; c.col_mid[col] = group * kTileTokens + pos; c.col_w[col] = w;
        if (pos == 0u) { c.exp_e[group] = e; c.exp_c0[group] = below; c.exp_n[group] = rows; }
    }
    const uint32_t G = gridDim.x, bid = blockIdx.x, NT1 = M * p.n1, r = NT1 - udiv_small(NT1, G) * G, k = p.k1;
    if (lane == 0) {
        c.M = M; c.nlive = __popc(live_mask); c.live_mask = live_mask;
        c.split_parts = 0u;
        if (r != 0u) {
            // the first r tiles are the remainder: tile t is shared by the SMs [ceil(t G / r), ceil((t + 1) G / r))
            const uint32_t t = udiv_small(bid * r, G), gs = udiv_small(t * G + r - 1u, r), ge = udiv_small((t + 1u) * G + r - 1u, r);
            const uint32_t S = ge - gs, li = bid - gs, base = udiv_small(k, S), extra = k - base * S;
            const uint32_t ub = li * base + (li < extra ? li : extra), ue = ub + base + (li < extra ? 1u : 0u);
            if (ue > ub) { c.split_t = t; c.split_range = ub | (ue << 8); c.split_first = gs; c.split_parts = S < k ? S : k; }
        }
    }
}

template <int kFmt, bool kFe>
__global__ void __launch_bounds__(DFmt<kFmt>::kThreads, 1) decode_moe_kernel(const __grid_constant__ BParams p) {
    using F = DFmt<kFmt>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ DShared c;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~static_cast<uintptr_t>(1023u));
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, bid = blockIdx.x, G = gridDim.x;
    uint32_t* ctrl32 = reinterpret_cast<uint32_t*>(p.buf + p.off_ctrl);
    const uint32_t n = static_cast<uint32_t>(p.T) * p.topk;
    // shared memory: token tile (the intermediate rows' tile takes the place of the tokens'), weight ring
    const uint32_t ring_off = (p.k1 > p.k2 ? p.k1 : p.k2) * F::kRec;
    uint32_t nw = udiv_small(p.smem_ring - ring_off, p.unit_bytes);
    nw = F::kA8 ? even_stages(nw, kDStages) : (nw > kDStages ? kDStages : nw);
    // ---- what needs nothing of the launches before this one: it overlaps the end of the previous kernel in the stream
    if (warp == 2) {
        if (lane < kDStages) { mbar_init(&c.wfull[lane], 1); mbar_init(&c.wempty[lane], F::kA8 ? kBExpWarps / 2 : 1); }
        if (lane < 2) {
            mbar_init(&c.tmem_full[lane], 1); mbar_init(&c.tmem_empty[lane], 4);
            mbar_init(&c.tile_full[lane], lane == 0 ? F::kBuilders : kDEpiWarps);
        }
        if (lane < kDWide) { mbar_init(&c.xfull[lane], kBExpWarps / 2); mbar_init(&c.xempty[lane], 1); }
        mbar_fence_init();
        if (lane == 0) { c.abort_flag = 0u; c.comb_next = 0u; c.wissued = 0u; c.start_ok = 0u; }
    }
    if (warp == 1) { tmem_alloc(&c.tmem_base, F::kTmemColumns); tmem_relinquish(); tc_fence_before(); }
    __syncthreads();
    tc_fence_after();
    grid_dependency_wait();
    grid_launch_dependents();
    const unsigned long long t_first = globaltimer_ns();
    const uint32_t epoch = ld_volatile_u32(ctrl32 + kCtrlEpoch / 4 + bid), flag = epoch + 1u;      // (warp 3 counts on, off the critical path)
    const DCtx cx(p, c, smem, globaltimer_ns() + p.timeout_ns, epoch & 1u);
    constexpr uint32_t kEW = 4;                                       // the first of the warps that build the token tile
    const bool builder = warp >= kEW && warp < kEW + F::kBuilders;
    constexpr uint32_t kPerWarp = kDEntries / F::kBuilders;           // entries a builder warp writes: 2, with E4M3 tokens 1
    // Rows of entries bw (and bw + 8) in registers before the routing is known: the 16 B chunks of the packed row and its scale
    // bytes (lane, lane + 32, ...). From hidden states the tokens are quantised into shared memory first, where the accumulators go later.
    constexpr uint32_t kChunks = F::kA8 ? 9u : 5u;
    const uint32_t xq = p.x_row_bytes / 16u, per_row = xq + p.x_sf_row_bytes / 16u;
    uint4 v[kPerWarp][kChunks];
    uint8_t* const quantised = reinterpret_cast<uint8_t*>(c.vt);      // the tokens' rows, each the packed row and its scale bytes
    const uint32_t qbytes = p.x_row_bytes + p.x_sf_row_bytes;
    uint32_t e = 0xFFu;
    float w = 0.f;
    if constexpr (!kFe) {
        if (warp == 0 && lane < n) {
            const long long ex = reinterpret_cast<const long long*>(p.buf + p.off_topk_idx)[lane];
            w = reinterpret_cast<const float*>(p.buf + p.off_topk_w)[lane];
            e = ex < 0 ? 0xFFu : (ex < p.E ? static_cast<uint32_t>(ex) : 0xFEu);
        }
        if (builder) {
            #pragma unroll
            for (uint32_t a = 0; a < kPerWarp; ++a) {
                const uint32_t f = warp - kEW + a * F::kBuilders;
                if (f < n) {
                    const uint32_t tok = udiv_small(f, p.topk);
                    const uint8_t* xs = p.buf + p.off_x + static_cast<size_t>(tok) * p.x_row_bytes;
                    const uint8_t* sf = p.buf + p.off_x_sf + static_cast<size_t>(tok) * p.x_sf_row_bytes;
                    #pragma unroll
                    for (uint32_t u = 0; u < kChunks; ++u) {
                        const uint32_t ci = lane + u * 32;
                        if (ci < per_row) v[a][u] = ld_cg_v4(ci < xq ? xs + ci * 16u : sf + (ci - xq) * 16u);
                    }
                }
            }
        }
    } else {
        // ---- router frontend: partial logits spread over the SMs; selection and quantisation on every SM. An item is one token's, with all its
        //      loads in flight up to hidden 3072, in two trips beyond (one token 27.2 -> 26.2 us a pass against items of four tokens in two trips, two with E4M3 38.9 -> 36.8)
        fe_logits_blocks<1, 6, 1>(p.fe, warp * G + bid, G * (F::kThreads / 32), lane, flag);
        if (builder) {
            // A slice of 256 elements to a warp at a time, two in flight. (Every warp used to quantise the tokens of its entries, the same token in eight
            // warps, out of registers: 75 to 150 KB of unrolled code. Two tokens 33.0 -> 30.9 us a pass, NVFP4 45.7 -> 31.4, one 27.5 -> 24.1.)
            const uint32_t nslice = static_cast<uint32_t>(p.k1);
            #pragma unroll 2
            for (uint32_t i = warp - kEW; i < static_cast<uint32_t>(p.T) * nslice; i += F::kBuilders) {
                const uint32_t tok = i >= nslice ? 1u : 0u, slice = i - tok * nslice;       // (two tokens at most)
                const __nv_bfloat16* xrow = p.fe.hidden + static_cast<size_t>(tok) * p.H;
                fe_quant_slice(xrow, kFmt, p.fe.x_gs, quantised + tok * qbytes, quantised + tok * qbytes + p.x_row_bytes, slice, lane,
                               bid == (tok < G ? tok : 0u), p.buf + p.off_x + static_cast<size_t>(tok) * p.x_row_bytes, p.buf + p.off_x_sf + static_cast<size_t>(tok) * p.x_sf_row_bytes);
            }
        }
        // (warp 1, which has nothing to do yet, runs the selection once on whatever records lie there and drops the result: the
        // SM then has the code in its instruction cache when the records arrive)
        if (warp >= 1u && warp <= 3u) {
            auto give_up = [&]() -> bool {
                if (cx.aborted()) return true;
                if (cx.expired()) { cx.fail(kErrWaitFrontend); return true; }
                return false;
            };
            const bool dry = warp == 1u;
            const uint32_t tok = dry ? 0u : warp - 2u;
            if (tok < static_cast<uint32_t>(p.T)) {
                const bool nz = fe_row_nonzero(p.fe.hidden + static_cast<size_t>(tok) * p.H, p.H, lane);
                uint32_t ce; float cw;
                const bool ok = fe_select_token_regs<2>(p.fe, tok, nz, lane, dry ? 0u : flag, nullptr, give_up, !dry && bid == (tok < G ? tok : 0u), &ce, &cw);   // (one SM writes the token's routing views)
                if (lane < 8u && !dry) { c.ent_e[tok * 8u + lane] = ok ? ce : 0xFFu; c.ent_w[tok * 8u + lane] = ok ? cw : 0.f; }
            }
        }
        __syncthreads();
        if (bid == 0 && tid == 0) cx.stamp(kStampFrontend);
        if (warp == 0 && lane < n) { e = c.ent_e[lane]; w = c.ent_w[lane]; e = e < static_cast<uint32_t>(p.E) ? e : 0xFFu; }
    }
    // ---- routing. The warp that sorts the entries is the weight loader: it does not wait for the others
    if (warp == 0) {
        d_route(cx, e, w, n, lane);
        __syncwarp();
        if (lane == 0) c.start_ok = cx.aborted() ? 0u : flag;        // (decided once: every warp takes the same way from here)
        __threadfence_block();
        __syncwarp();
        // The others hear of the routing when the stream has begun, so that their first instructions, which come from the L2, do not hold up the
        // loader's (one token 22.0 -> 21.4 us a pass, two 28.2 -> 27.6). With E4M3 tokens the tile takes longer than
        // the first unit, and the others start first (two tokens 31.7 us, the other way round 32.9).
        // (The times go to memory when the whole stream has been asked for.)
        const bool go = *reinterpret_cast<volatile uint32_t*>(&c.start_ok) != 0u;
        unsigned long long t_routed = 0ull, t_first = ~0ull;          // (~0: no weights on this SM)
        if (F::kA8 || !go) { t_routed = globaltimer_ns(); bar_arrive(kDBarRouted, F::kThreads); }
        if (go) d_role_weights(cx, nw, smem + ring_off, [&](bool any) {
            const unsigned long long t = globaltimer_ns();
            if (any) t_first = t;
            if constexpr (!F::kA8) { t_routed = t; bar_arrive(kDBarRouted, F::kThreads); }
        });
        if (lane == 0) {
            cx.sm_phase(kSmScheduled, t_routed); cx.stamp_max(kStampLastScheduled, t_routed); if (bid == 0) cx.stamp(kStampScheduled, t_routed);
            reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlSmWFirst)[bid] = t_first;
            if (t_first != ~0ull) cx.sm_phase(kSmFirstIssue, t_first);
        }
    } else bar_sync(kDBarRouted, F::kThreads);
    const bool start = *reinterpret_cast<volatile uint32_t*>(&c.start_ok) != 0u;
    if (start) {
        if (warp == 1) {
            d_role_mma<kFmt>(cx, lane, nw, ring_off);
        } else if (builder) {
            // ---- the token tile
            #pragma unroll
            for (uint32_t a = 0; a < kPerWarp; ++a) {
                const uint32_t f = warp - kEW + a * F::kBuilders;
                if (f < n && ((c.live_mask >> f) & 1u) != 0u) {
                    const uint32_t col = c.ent_col[f];
                    if constexpr (kFe) {
                        const uint32_t tok = f >> 3;                  // (eight routes per token)
                        #pragma unroll
                        for (uint32_t u = 0; u < kChunks; ++u)
                            if (lane + u * 32u < per_row) v[a][u] = *reinterpret_cast<const uint4*>(quantised + tok * qbytes + (lane + u * 32u) * 16u);
                    }
                    #pragma unroll
                    for (uint32_t u = 0; u < kChunks; ++u) {
                        const uint32_t ci = lane + u * 32;
                        if (ci < xq) {
                            const uint32_t at = ci >> 3;
                            *reinterpret_cast<uint4*>(smem + (F::kA8 ? (at >> 1) * F::kRec + (at & 1u) * 2048u : at * F::kRec) + sw128_off(col, ci & 7u)) = F::kA8 ? even_odd(v[a][u]) : v[a][u];
                        } else if (ci < per_row) {
                            const uint32_t g = (ci - xq) * 4u;
                            const uint32_t wv[4] = {v[a][u].x, v[a][u].y, v[a][u].z, v[a][u].w};
                            #pragma unroll
                            for (uint32_t k = 0; k < 4; ++k)
                                *reinterpret_cast<uint32_t*>(smem + ((g + k) / F::kPlanes) * F::kRec + 2048u * F::kAtoms + ((g + k) % F::kPlanes) * 512u + plane_off(col)) = wv[k];
                        }
                    }
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&c.tile_full[0]); cx.sm_phase(kSmRowsCached); }
            if (warp < kEW + kDEpiWarps) d_role_epilogue<kFmt>(cx, (warp - kEW) >> 2, (tid - 32u * kEW) & 127u, smem, flag);
            else if constexpr (F::kA8) { const uint32_t x = tid - 32u * (kEW + kDEpiWarps); d_role_widen(cx, x / kXGroupThreads, x % kXGroupThreads, nw, smem + ring_off); }
        }
    }
    // ---- off the critical path: launch number, counters, stamps, and what others may inspect afterwards
    if (warp == 3) {
        if (lane == 0) {
            ctrl32[kCtrlEpoch / 4 + bid] = epoch + 1u;
            reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlSmEntry)[bid] = t_first;
            reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlSmPhase)[bid * kSmPhaseSlots + kSmEntry] = t_first;
            if (bid == 0) {
                ctrl32[kCtrlStatus / 4 + 1] = epoch + 1u; ctrl32[kCtrlStatus / 4 + 2] = 0u; ctrl32[kCtrlStatus / 4 + 3] = 0u;
                ctrl32[kCtrlStatus / 4 + 4] = kRanDecode;
                reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlStamps)[kStampEntry] = t_first;
                reinterpret_cast<unsigned long long*>(p.buf + p.off_ctrl + kCtrlStamps)[kStampPrologue] = t_first;   // (set-up precedes the first stamp)
            }
        }
        // the batch kernel's arrival counts of the other parity (also when this launch has failed)
        cx.clear_other(lane);
        if (bid == 0 && start) {
            if (p.stats != nullptr && lane < c.M) p.stats[c.exp_e[lane]] += static_cast<int>(c.exp_n[lane]);
            uint8_t* region = p.buf + p.off_rx + static_cast<size_t>(cx.par) * p.rx_region;
            if (lane == 0) st_ll_16B(region, make_uint4(c.nlive, 0u, 0u, 0u), flag);
            if (lane < n && ((c.live_mask >> lane) & 1u) != 0u) {
                const uint32_t li = __popc(c.live_mask & ((1u << lane) - 1u)), tok = udiv_small(lane, p.topk);
                st_ll_16B(region + 32u + static_cast<size_t>(li) * 2u * p.rx_row_bytes + 2u * (p.rx_row_bytes - 16u),
                          make_uint4(c.ent_e[lane], tok, lane - tok * p.topk, __float_as_uint(c.col_w[c.ent_col[lane]])), flag);
            }
        }
    }
    if (tid == 128) { cx.stamp_max(kStampLastTasksDone); cx.sm_phase(kSmTasksDone); if (bid == 0) cx.stamp(kStampTasksDone); }
    // (two warps have nothing else to do: they begin when this SM has all intermediate rows, until then their polls would only take from what the stream
    // and the hand-over can get)
    if (start && (warp == 2 || warp == 3)) cx.warp_wait(&c.tile_full[1], 0u, kErrWaitL1Done);
    if (start) d_role_combine(cx, flag, lane);
    // ---- exit: an aborted SM lets the copies in flight land (bounded waits) before its shared memory goes away
    if (cx.aborted() && warp == 0) {
        const uint32_t issued = *reinterpret_cast<volatile uint32_t*>(&c.wissued);
        #pragma unroll 1
        for (uint32_t k = issued > nw ? issued - nw : 0u; k < issued; ++k)
            for (uint32_t spin = 0; spin < 2000u && !mbar_try_wait(&c.wfull[k % nw], (k / nw) & 1u); ++spin) { }
        for (uint32_t spin = 0; spin < 2000u; ++spin) __nanosleep(100);
    }
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(c.tmem_base, F::kTmemColumns); }
    if (tid == 0) { if (bid == 0) cx.stamp(kStampExit); cx.stamp_max(kStampLastExit); cx.sm_phase(kSmExit); }
}

}  // namespace mm
