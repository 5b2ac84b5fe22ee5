// Router frontend: bf16 router GEMM (fp32 accumulate, one bf16 rounding), top-8 selection with the
// (score descending, expert id ascending) order, routing weights, and token quantisation into the layer's input views.
//
// Reduction order of a logit (fixed, so that a CPU restatement can reproduce it bit for bit): K is cut into two halves;
// inside a half, lane l of a warp owns the 8-element chunks l, l + 32, l + 64, ... and runs one fused multiply-add chain
// over them in order; the 32 partial sums are combined by a butterfly (xor 16, 8, 4, 2, 1); the two halves are added
// (first + second) in fp32 and the sum is rounded to bf16 once. A half is one warp's work with all its loads in flight
// at once: one memory round trip per logit.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cstdint>
#include "mm_ptx.cuh"
#include "mm_frontend_route.h"

namespace mm {

struct FeParams {
    const __nv_bfloat16* hidden; const __nv_bfloat16* router_w; const float* bias;
    float* logits;
    uint8_t* x; uint8_t* x_sf; long long* topk_idx; float* topk_w;
    int T, H, E, topk, score_mode, fmt, x_row_bytes, x_sf_row_bytes;
    float x_gs;
    int cluster_tokens;                      // tokens of a cluster (`frontend_cluster_kernel` alone)
};

__device__ __forceinline__ void unpack_bf16x8(const uint4& v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    #pragma unroll
    for (int i = 0; i < 4; ++i) { f[2 * i] = __uint_as_float(w[i] << 16); f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u); }
}

constexpr uint32_t kFeParts = 2;
constexpr int kFeMaxFusedTokens = 256;       // tokens per rank the single-kernel path takes (its logit records live in the buffer)

// Partial logits live in the workspace as 16 B records per (token, expert): {first half, flag, second half, flag}; each
// half is written by its warp with one 8-byte store, so a reader that finds `flag` in a half also has its value.
// One warp per (expert, half of K, block of up to 4 tokens); `warp` of `nwarps` warps cooperate. This function and
// `fe_select_token` serve the multi-rank kernel: its dispatching SMs select for all tokens of the rank among up to 1024
// experts from shared memory, within that kernel's registers. The one-rank kernels and the stand-alone frontend have
// `fe_logits_blocks` and `fe_select_token_regs`; what those would give among several ranks has not been measured.
__device__ __forceinline__ void fe_logits_items(const FeParams& q, uint32_t warp, uint32_t nwarps, uint32_t lane, uint32_t flag) {
    const uint32_t tblocks = (q.T + 3) / 4, nchunk = q.H / 8, half = (nchunk + kFeParts - 1) / kFeParts;
    const uint32_t nitems = static_cast<uint32_t>(q.E) * kFeParts * tblocks;
    for (uint32_t item = warp; item < nitems; item += nwarps) {
        const uint32_t part = item % kFeParts, e = (item / kFeParts) % q.E, t0 = (item / (kFeParts * q.E)) * 4;
        const uint32_t nt = min(4u, static_cast<uint32_t>(q.T) - t0);
        const uint32_t c_lo = part * half, c_hi = min(nchunk, c_lo + half);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        const uint4* wrow = reinterpret_cast<const uint4*>(q.router_w + static_cast<size_t>(e) * q.H);
        // six chunks per lane are fetched before the first multiply-add (a half of K = 3072 is exactly that: one memory
        // round trip); the multiply-adds then run in the same order as a chunk-by-chunk loop would
        constexpr uint32_t kAhead = 6;
        #pragma unroll 1
        for (uint32_t ch0 = c_lo + lane; ch0 < c_hi; ch0 += 32 * kAhead) {
            uint4 wq[kAhead], xq[4][kAhead];
            #pragma unroll
            for (uint32_t b = 0; b < kAhead; ++b) {
                const uint32_t ch = ch0 + 32 * b;
                if (ch < c_hi) {
                    wq[b] = __ldg(wrow + ch);
                    #pragma unroll
                    for (uint32_t t = 0; t < 4; ++t)
                        if (t < nt) xq[t][b] = __ldg(reinterpret_cast<const uint4*>(q.hidden + static_cast<size_t>(t0 + t) * q.H) + ch);
                }
            }
            #pragma unroll
            for (uint32_t b = 0; b < kAhead; ++b) {
                if (ch0 + 32 * b < c_hi) {
                    float w[8];
                    unpack_bf16x8(wq[b], w);
                    #pragma unroll
                    for (uint32_t t = 0; t < 4; ++t) {
                        if (t < nt) {
                            float x[8];
                            unpack_bf16x8(xq[t][b], x);
                            #pragma unroll
                            for (int k = 0; k < 8; ++k) acc[t] = fmaf(x[k], w[k], acc[t]);
                        }
                    }
                }
            }
        }
        #pragma unroll
        for (uint32_t t = 0; t < 4; ++t) {
            #pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
            if (lane == 0 && t < nt)
                st_volatile_v2(reinterpret_cast<uint8_t*>(q.logits) + (static_cast<size_t>(t0 + t) * q.E + e) * 16u + part * 8u,
                               __float_as_uint(acc[t]), flag);
        }
    }
}

// The same partial logits (the same sums in the same order) with blocks of kEb experts x kTb tokens per warp and kAhead chunks
// per lane in flight: per multiply-add a block of 4 x 4 reads 0.5 operand chunks instead of 1.25, which is the time of a large
// batch; a small one needs every (expert, half) as an item of its own to have enough of them. `fe_expert_block` draws the stand-alone frontend's line at four items per SM.
template <int kEb, int kAhead, int kTb = 4>
__device__ __forceinline__ void fe_logits_blocks(const FeParams& q, uint32_t warp, uint32_t nwarps, uint32_t lane, uint32_t flag) {
    const uint32_t tblocks = (q.T + kTb - 1) / kTb, eblocks = (q.E + kEb - 1) / kEb, nchunk = q.H / 8, half = (nchunk + kFeParts - 1) / kFeParts;
    const uint32_t nitems = eblocks * kFeParts * tblocks;
    #pragma unroll 1
    for (uint32_t item = warp; item < nitems; item += nwarps) {
        const uint32_t part = item % kFeParts, r = item / kFeParts, tb = udiv_small(r, eblocks), e0 = (r - tb * eblocks) * kEb, t0 = tb * kTb;
        const uint32_t nt = min(static_cast<uint32_t>(kTb), static_cast<uint32_t>(q.T) - t0), ne = min(static_cast<uint32_t>(kEb), static_cast<uint32_t>(q.E) - e0);
        const uint32_t c_lo = part * half, c_hi = min(nchunk, c_lo + half);
        float acc[kEb][kTb];
        #pragma unroll
        for (int e = 0; e < kEb; ++e) {
            #pragma unroll
            for (int t = 0; t < kTb; ++t) acc[e][t] = 0.f;
        }
        // (rows beyond the last expert or token repeat the last one: their sums are not stored)
        const uint4 *wrow[kEb], *xrow[kTb];
        #pragma unroll
        for (uint32_t e = 0; e < kEb; ++e) wrow[e] = reinterpret_cast<const uint4*>(q.router_w + static_cast<size_t>(e0 + (e < ne ? e : ne - 1u)) * q.H);
        #pragma unroll
        for (uint32_t t = 0; t < kTb; ++t) xrow[t] = reinterpret_cast<const uint4*>(q.hidden + static_cast<size_t>(t0 + (t < nt ? t : nt - 1u)) * q.H);
        #pragma unroll 1
        for (uint32_t ch0 = c_lo + lane; ch0 < c_hi; ch0 += 32 * kAhead) {
            uint4 wq[kEb][kAhead], xq[kTb][kAhead];
            #pragma unroll
            for (uint32_t b = 0; b < kAhead; ++b) {
                const uint32_t ch = ch0 + 32 * b;
                if (ch < c_hi) {
                    #pragma unroll
                    for (uint32_t e = 0; e < kEb; ++e) wq[e][b] = __ldg(wrow[e] + ch);
                    #pragma unroll
                    for (uint32_t t = 0; t < kTb; ++t) if (t < nt) xq[t][b] = __ldg(xrow[t] + ch);
                }
            }
            #pragma unroll
            for (uint32_t b = 0; b < kAhead; ++b) {
                if (ch0 + 32 * b < c_hi) {
                    #pragma unroll
                    for (uint32_t t = 0; t < kTb; ++t) {
                        if (t < nt) {
                            float x[8];
                            unpack_bf16x8(xq[t][b], x);
                            #pragma unroll
                            for (uint32_t e = 0; e < kEb; ++e) {
                                float w[8];
                                unpack_bf16x8(wq[e][b], w);
                                #pragma unroll
                                for (int k = 0; k < 8; ++k) acc[e][t] = fmaf(x[k], w[k], acc[e][t]);
                            }
                        }
                    }
                }
            }
        }
        #pragma unroll
        for (uint32_t e = 0; e < kEb; ++e) {
            #pragma unroll
            for (uint32_t t = 0; t < kTb; ++t) {
                #pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[e][t] += __shfl_xor_sync(0xffffffffu, acc[e][t], o);
                if (lane == 0 && t < nt && e < ne)
                    st_volatile_v2(reinterpret_cast<uint8_t*>(q.logits) + (static_cast<size_t>(t0 + t) * q.E + e0 + e) * 16u + part * 8u,
                                   __float_as_uint(acc[e][t]), flag);
            }
        }
    }
}
__device__ __forceinline__ uint32_t fe_expert_block(const FeParams& q, uint32_t grid) {
    const uint32_t per = static_cast<uint32_t>(q.E) * kFeParts * ((q.T + 3) / 4);     // items of one expert each
    return per >= 16u * grid ? 4u : (per >= 8u * grid ? 2u : 1u);
}

// the logit from its two halves
__device__ __forceinline__ float fe_logit(float first, float second) { return bf16_round(first + second) + 0.0f; }
// logit of (token t, expert e) from its two halves; `flag` != 0: poll until both halves carry it (`ok` = false if `give_up`
// says so first)
template <typename GiveUp>
__device__ __forceinline__ float fe_read_logit(const FeParams& q, uint32_t t, uint32_t e, uint32_t flag, bool& ok, GiveUp give_up) {
    const uint8_t* src = reinterpret_cast<const uint8_t*>(q.logits) + (static_cast<size_t>(t) * q.E + e) * 16u;
    uint32_t spins = 0;
    for (;;) {
        const uint4 v = ld_volatile_v4(src);
        if (flag == 0u || (v.y == flag && v.w == flag)) return fe_logit(__uint_as_float(v.x), __uint_as_float(v.z));
        if ((++spins & 0x3Fu) == 0u && give_up()) { ok = false; return 0.f; }
    }
}

__device__ __forceinline__ uint32_t orderable_f32(float v) {
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
// orderable score of an expert, 0: not selectable
__device__ __forceinline__ uint32_t fe_key(const FeParams& q, float v, float bias) {
    const float s = (q.score_mode == 1 ? (1.0f / (1.0f + expf(-v))) + bias : v) + 0.0f;
    return s != -INFINITY ? orderable_f32(s) : 0u;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, v, o);
        v = other > v ? other : v;
    }
    return v;
}

// Eight consecutive elements per lane -> 4 bytes of E2M1 codes (formats 0, 1; in .x) or 8 bytes of E4M3 (format 2), and the
// byte of the lane's scale block, which two (format 1) or four neighbouring lanes share. Every lane of the warp calls it.
__device__ __forceinline__ uint2 fe_quant8(const uint4& raw, int fmt, float x_gs, bool& nonzero, uint32_t& sf_byte) {
    float x[8];
    unpack_bf16x8(raw, x);
    float local = 0.f;
    #pragma unroll
    for (int j = 0; j < 8; ++j) {
        nonzero |= x[j] != 0.f;
        if (fmt == 1) x[j] = __fdiv_rn(x[j], x_gs);
        local = fmaxf(local, fabsf(x[j]));
    }
    local = fmaxf(local, __shfl_xor_sync(0xffffffffu, local, 1));
    if (fmt != 1) local = fmaxf(local, __shfl_xor_sync(0xffffffffu, local, 2));
    const float v = fmt == 2 ? fmaxf(local, 1.0e-4f) * (1.0f / 448.0f) : fmaxf(local, 1.0e-30f) * (1.0f / 6.0f);
    float sf;
    if (fmt == 1) {
        sf_byte = cvt_e4m3x2(v, 0.f) & 0xFFu;
        if (sf_byte == 0u) sf_byte = 1u;
        sf = e4m3_to_float(sf_byte);
    } else {
        sf_byte = ceil_pow2_exp(v);
        sf = __uint_as_float(sf_byte << 23);
    }
    const float inv = 1.0f / sf;
    uint2 bytes = make_uint2(0u, 0u);
    if (fmt == 2) {
        bytes.x = cvt_e4m3x2(x[0] * inv, x[1] * inv) | (cvt_e4m3x2(x[2] * inv, x[3] * inv) << 16);
        bytes.y = cvt_e4m3x2(x[4] * inv, x[5] * inv) | (cvt_e4m3x2(x[6] * inv, x[7] * inv) << 16);
    } else {
        #pragma unroll
        for (int j = 0; j < 4; ++j) bytes.x |= cvt_e2m1x2(x[2 * j] * inv, x[2 * j + 1] * inv) << (8 * j);
    }
    return bytes;
}

// One warp quantises token row `xrow` (bf16 [H]) to packed E2M1 (formats 0, 1) or E4M3 bytes (format 2) + scale bytes;
// returns whether any element is non-zero. With `pool_row` != nullptr the same bytes are also stored there as a row of
// the receive pool (packed row, then the scale bytes; every 4 data bytes followed by `flag`): the dispatch of the fused
// frontend writes the peer's pool straight from the registers instead of re-reading the views it has just written.
__device__ __forceinline__ bool fe_quant_token(const __nv_bfloat16* xrow, int H, int fmt, float x_gs,
                                               uint8_t* qrow, uint8_t* sfrow, uint32_t lane,
                                               uint8_t* pool_row = nullptr, uint32_t flag = 0u, uint32_t x_row_bytes = 0u) {
    const int vec = fmt == 1 ? 16 : 32, lanes_per_group = vec / 8;
    bool nonzero = false;
    uint4 ahead[4];                                              // (four slices of the row in flight)
    #pragma unroll 4
    for (int k0 = lane * 8; k0 < H; k0 += 256) {
        if (((k0 >> 8) & 3) == 0) {
            #pragma unroll
            for (int b = 0; b < 4; ++b) if (k0 + 256 * b < H) ahead[b] = *reinterpret_cast<const uint4*>(xrow + k0 + 256 * b);
        }
        const int slice = (k0 >> 8) & 3;
        uint32_t sf_byte;
        const uint2 bytes = fe_quant8(slice == 0 ? ahead[0] : (slice == 1 ? ahead[1] : (slice == 2 ? ahead[2] : ahead[3])), fmt, x_gs, nonzero, sf_byte);
        if ((lane % lanes_per_group) == 0) sfrow[k0 / vec] = static_cast<uint8_t>(sf_byte);
        const int it = k0 >> 8;                                  // which 256-element slice of the row
        if (fmt == 2) {
            *reinterpret_cast<uint2*>(qrow + k0) = bytes;
            if (pool_row != nullptr) {
                asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" :: "l"(pool_row + 2 * k0), "r"(bytes.x), "r"(flag), "r"(bytes.y), "r"(flag) : "memory");
            }
        } else {
            *reinterpret_cast<uint32_t*>(qrow + k0 / 2) = bytes.x;
            if (pool_row != nullptr) st_volatile_v2(pool_row + k0, bytes.x, flag);         // 2 * (k0 / 2)
        }
        if (pool_row != nullptr) {
            // four scale bytes make one word: every lane of a group holds its group's byte; the first lane of four groups stores
            const int span = 4 * lanes_per_group;               // lanes that share one scale word
            const uint32_t base_lane = lane & ~static_cast<uint32_t>(span - 1);
            uint32_t word = 0u;
            #pragma unroll
            for (int b = 0; b < 4; ++b) word |= __shfl_sync(0xffffffffu, sf_byte, base_lane + b * lanes_per_group) << (8 * b);
            if ((lane & static_cast<uint32_t>(span - 1)) == 0u) {
                const uint32_t sf_off = static_cast<uint32_t>(it) * (256u / vec) + (lane / span) * 4u;     // byte offset inside the row's scale bytes
                st_volatile_v2(pool_row + 2u * (x_row_bytes + sf_off), word, flag);
            }
        }
    }
    return __any_sync(0xffffffffu, nonzero);
}

// One warp quantises the 256 elements `slice` of a token row; with `also` the bytes go to a second row too.
__device__ __forceinline__ void fe_quant_slice(const __nv_bfloat16* xrow, int fmt, float x_gs, uint8_t* qrow, uint8_t* sfrow, uint32_t slice, uint32_t lane,
                                               bool also = false, uint8_t* qrow2 = nullptr, uint8_t* sfrow2 = nullptr) {
    const uint32_t k0 = slice * 256u + lane * 8u, vec = fmt == 1 ? 16u : 32u;
    bool nonzero = false;
    uint32_t sf_byte;
    const uint2 bytes = fe_quant8(*reinterpret_cast<const uint4*>(xrow + k0), fmt, x_gs, nonzero, sf_byte);
    auto put = [&](uint8_t* q, uint8_t* sf) {
        if (lane % (vec / 8u) == 0u) sf[k0 / vec] = static_cast<uint8_t>(sf_byte);
        if (fmt == 2) *reinterpret_cast<uint2*>(q + k0) = bytes;
        else *reinterpret_cast<uint32_t*>(q + k0 / 2u) = bytes.x;
    };
    put(qrow, sfrow);
    if (also) put(qrow2, sfrow2);
}

// One warp: is any element of the bf16 row non-zero?
__device__ __forceinline__ bool fe_row_nonzero(const __nv_bfloat16* xrow, int H, uint32_t lane) {
    // all loads of the row are issued before the first is used (one memory round trip, not one per 256 elements); the
    // row then sits in this SM's L1 for the quantisation pass that follows with the same lane mapping
    uint32_t any = 0u;
    #pragma unroll
    for (int i = 0; i < 16; ++i) {                        // H <= 4096
        const int k0 = lane * 8 + i * 256;
        if (k0 < H) {
            const uint4 v = *reinterpret_cast<const uint4*>(xrow + k0);
            any |= v.x | v.y | v.z | v.w;
        }
    }
    const bool nz = (any & 0x7FFF7FFFu) != 0u;
    return __any_sync(0xffffffffu, nz);
}

// One warp selects the top-8 experts of token t from its logits (other SMs wrote them; `flag` != 0: they may still be on
// their way and are polled) and writes topk_idx / topk_weights. `sc` is a per-warp scratch of 2 E floats in shared
// memory (scores, then the plain logits). Returns false if `give_up` ended a poll.
template <typename GiveUp>
__device__ __forceinline__ bool fe_select_token(const FeParams& q, uint32_t t, float* sc, bool nonzero, uint32_t lane, uint32_t flag, GiveUp give_up) {
    float* lgv = sc + q.E;
    bool ok = true;
    // the token's logit records, eight per lane in flight at a time (one memory round trip per 256 experts when they have
    // all arrived); a record that is not complete yet is polled on its own afterwards
    for (int e0 = lane; e0 < q.E; e0 += 32 * 8) {
        uint4 rec[8];
        #pragma unroll
        for (int b = 0; b < 8; ++b) {
            const int e = e0 + 32 * b;
            if (e < q.E) rec[b] = ld_volatile_v4(reinterpret_cast<const uint8_t*>(q.logits) + (static_cast<size_t>(t) * q.E + e) * 16u);
        }
        #pragma unroll
        for (int b = 0; b < 8; ++b) {
            const int e = e0 + 32 * b;
            if (e >= q.E) continue;
            float v;
            if (flag == 0u || (rec[b].y == flag && rec[b].w == flag)) v = bf16_round(__uint_as_float(rec[b].x) + __uint_as_float(rec[b].z)) + 0.0f;
            else v = fe_read_logit(q, t, static_cast<uint32_t>(e), flag, ok, give_up);
            lgv[e] = v;
            sc[e] = q.score_mode == 1 ? (1.0f / (1.0f + expf(-v))) + q.bias[e] : v;
        }
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    __syncwarp();
    // eight rounds of a warp-wide maximum over 64-bit keys (score, then smaller expert id)
    unsigned long long chosen = 0ull;
    for (int k = 0; k < 8; ++k) {
        unsigned long long best = 0ull;
        for (int e = lane; e < q.E; e += 32) {
            const float s = sc[e];
            if (s == -INFINITY) continue;
            const unsigned long long key = (static_cast<unsigned long long>(orderable_f32(s + 0.0f)) << 32) | (0xFFFFFFFFu - static_cast<uint32_t>(e));
            best = key > best ? key : best;
        }
        best = warp_max_u64(best);
        // no candidate left (fewer than eight selectable experts: every remaining score is -inf): the slot stays empty
        const bool found = best != 0ull;
        const uint32_t e_best = 0xFFFFFFFFu - static_cast<uint32_t>(best & 0xFFFFFFFFull);
        if (found && lane == 0) sc[e_best] = -INFINITY;
        if (static_cast<int>(lane) == k) chosen = found ? e_best : 0xFFFFFFFFull;
        __syncwarp();
    }
    const bool empty_slot = lane < 8 && chosen == 0xFFFFFFFFull;
    const int e_sel = empty_slot ? 0 : static_cast<int>(chosen);
    const float v_sel = lane < 8 && !empty_slot ? lgv[e_sel] : -INFINITY;
    float wgt;
    if (q.score_mode == 1) {
        const float s = lane < 8 ? 1.0f / (1.0f + expf(-v_sel)) : 0.f;
        float sum = 0.f;
        #pragma unroll
        for (int k = 0; k < 8; ++k) sum += __shfl_sync(0xffffffffu, s, k);
        wgt = s / sum;
    } else {
        float mx = v_sel;
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float ex = lane < 8 ? expf(v_sel - mx) : 0.f;
        float sum = 0.f;
        #pragma unroll
        for (int k = 0; k < 8; ++k) sum += __shfl_sync(0xffffffffu, ex, k);
        wgt = ex / sum;
    }
    if (lane < 8) {
        q.topk_idx[static_cast<size_t>(t) * 8 + lane] = nonzero && !empty_slot ? e_sel : -1;
        q.topk_w[static_cast<size_t>(t) * 8 + lane] = nonzero && !empty_slot ? wgt : 0.f;
    }
    return true;
}

// The top-8 of one token from its logits and score keys, kPer experts per lane (lane, lane + 32, ...): see `fe_select_token_regs`.
template <int kPer>
__device__ __forceinline__ void fe_choose(const FeParams& q, uint32_t t, bool nonzero, uint32_t lane, uint32_t flag, uint8_t* records, const float (&lg)[kPer],
                                          uint32_t (&key)[kPer], bool publish = true, uint32_t* e_out = nullptr, float* w_out = nullptr) {
    uint32_t top = 0u, top_h = 0u;                                // this lane's best score and the first of its experts that has it
    float top_v = 0.f;
    auto rescan = [&]() {
        top = 0u;
        #pragma unroll
        for (uint32_t h = 0; h < kPer; ++h) if (key[h] > top) { top = key[h]; top_h = h; top_v = lg[h]; }
    };
    rescan();
    uint32_t chosen = 0xFFFFFFFFu;
    float v_sel = -INFINITY;
    #pragma unroll 1
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t best = __reduce_max_sync(0xffffffffu, top);
        const uint32_t e = __reduce_min_sync(0xffffffffu, best != 0u && top == best ? lane + 32u * top_h : 0xFFFFFFFFu);
        const float v = __shfl_sync(0xffffffffu, top_v, e & 31u);
        if (e != 0xFFFFFFFFu) {
            if (lane == k) { chosen = e; v_sel = v; }
            if ((e & 31u) == lane) {
                #pragma unroll
                for (uint32_t h = 0; h < kPer; ++h) if (h == (e >> 5)) key[h] = 0u;
                rescan();
            }
        }
        __syncwarp();
    }
    const bool empty_slot = chosen == 0xFFFFFFFFu;
    float wgt;
    if (q.score_mode == 1) {
        const float s = lane < 8 ? 1.0f / (1.0f + expf(-v_sel)) : 0.f;
        float sum = 0.f;
        #pragma unroll
        for (int k = 0; k < 8; ++k) sum += __shfl_sync(0xffffffffu, s, k);
        wgt = s / sum;
    } else {
        float mx = v_sel;
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float ex = lane < 8 ? expf(v_sel - mx) : 0.f;
        float sum = 0.f;
        #pragma unroll
        for (int k = 0; k < 8; ++k) sum += __shfl_sync(0xffffffffu, ex, k);
        wgt = ex / sum;
    }
    if (lane < 8) {
        const bool live = nonzero && !empty_slot;
        const float w = live ? wgt : 0.f;
        if (records != nullptr && publish)
            asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};"
                     :: "l"(records + (static_cast<size_t>(t) * 8u + lane) * 16u), "r"(live ? chosen : 0xFFFFFFFFu), "r"(flag), "r"(__float_as_uint(w)), "r"(flag) : "memory");
        if (e_out != nullptr) { *e_out = live ? chosen : 0xFFFFFFFFu; *w_out = w; }
        if (publish) {
            q.topk_idx[static_cast<size_t>(t) * 8 + lane] = live ? static_cast<long long>(chosen) : -1ll;
            q.topk_w[static_cast<size_t>(t) * 8 + lane] = w;
        }
    }
}

// One warp selects the top-8 of token t among at most 32 kPer experts, kPer per lane, in registers: the same keys, weights
// and order of additions as `fe_select_token` (maximum of the scores, then the smallest expert with it, eight times); a lane
// keeps its best score at hand, so that a round is two warp reductions and a rescan by one lane. The routing goes into
// topk_idx / topk_weights and, with `records`, as flagged 16 B records {expert (~0: none), flag, weight, flag} to where the
// launch's other SMs poll it; `e_out` / `w_out` get lane k's route k (`publish` false: only those). `flag` 0: the logits are complete. Returns false if `give_up` ended a poll.
template <int kPer, typename GiveUp>
__device__ __forceinline__ bool fe_select_token_regs(const FeParams& q, uint32_t t, bool nonzero, uint32_t lane, uint32_t flag, uint8_t* records, GiveUp give_up,
                                                     bool publish = true, uint32_t* e_out = nullptr, float* w_out = nullptr) {
    bool ok = true;
    float lg[kPer];
    uint32_t key[kPer];                                           // orderable score, 0: not selectable
    constexpr int kFly = kPer < 8 ? kPer : 4;                     // records in flight
    float bias[kPer];                                             // (fetched before the records are awaited: the load may come from HBM)
    #pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const uint32_t e = lane + 32u * h;
        bias[h] = q.score_mode == 1 && e < static_cast<uint32_t>(q.E) ? __ldg(q.bias + e) : 0.f;
    }
    #pragma unroll
    for (int h0 = 0; h0 < kPer; h0 += kFly) {
        uint4 rec[kFly];
        #pragma unroll
        for (int h = 0; h < kFly; ++h) {
            const uint32_t e = lane + 32u * (h0 + h);
            if (e < static_cast<uint32_t>(q.E)) rec[h] = ld_volatile_v4(reinterpret_cast<const uint8_t*>(q.logits) + (static_cast<size_t>(t) * q.E + e) * 16u);
        }
        #pragma unroll
        for (int h = 0; h < kFly; ++h) {
            const uint32_t e = lane + 32u * (h0 + h);
            lg[h0 + h] = 0.f; key[h0 + h] = 0u;
            if (e < static_cast<uint32_t>(q.E)) {
                float v;
                if (flag == 0u || (rec[h].y == flag && rec[h].w == flag)) v = fe_logit(__uint_as_float(rec[h].x), __uint_as_float(rec[h].z));
                else v = fe_read_logit(q, t, e, flag, ok, give_up);
                lg[h0 + h] = v;
                key[h0 + h] = fe_key(q, v, bias[h0 + h]);
            }
        }
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    fe_choose<kPer>(q, t, nonzero, lane, flag, records, lg, key, publish, e_out, w_out);
    return true;
}

// The stand-alone frontend, two launches. First the partial logits and, by the last warps of the grid, the tokens'
// quantisation (it needs no logits); then one warp per token for the selection. The second launch starts early and waits on
// the device, so its launch latency is hidden behind the first.
constexpr int kFeThreads = 512;
__global__ void __launch_bounds__(kFeThreads, 1) frontend_logits_kernel(const __grid_constant__ FeParams q) {
    const uint32_t lane = threadIdx.x & 31u, nwarps = gridDim.x * (kFeThreads / 32), w = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;   // (consecutive items on different SMs)
    grid_dependency_wait();
    grid_launch_dependents();
    #pragma unroll 1
    for (uint32_t t = nwarps - 1u - w; t < static_cast<uint32_t>(q.T); t += nwarps)
        fe_quant_token(q.hidden + static_cast<size_t>(t) * q.H, q.H, q.fmt, q.x_gs, q.x + static_cast<size_t>(t) * q.x_row_bytes,
                       q.x_sf + static_cast<size_t>(t) * q.x_sf_row_bytes, lane);
    const uint32_t eb = fe_expert_block(q, gridDim.x);
    if (eb == 1u) fe_logits_blocks<1, 3>(q, w, nwarps, lane, 1u);
    else if (eb == 2u) fe_logits_blocks<2, 2>(q, w, nwarps, lane, 1u);
    else fe_logits_blocks<4, 2>(q, w, nwarps, lane, 1u);
}

template <int kPer>
__global__ void __launch_bounds__(32) frontend_select_kernel(const __grid_constant__ FeParams q) {
    const uint32_t lane = threadIdx.x, t = blockIdx.x;
    grid_dependency_wait();
    grid_launch_dependents();
    const bool nonzero = fe_row_nonzero(q.hidden + static_cast<size_t>(t) * q.H, q.H, lane);
    fe_select_token_regs<kPer>(q, t, nonzero, lane, 0u, nullptr, [] { return false; });
}

// The same for a few tokens, in one launch. A cluster of CTAs takes one or two tokens through all three steps, so that the partial
// logits meet in shared memory instead of in a second launch: CTA r works out the experts [r E / C, (r + 1) E / C) and sends each
// sum to the CTA that selects for the token (token i of the cluster: CTA i), whose other warps quantise it; behind one cluster
// barrier those select. The sums are those of `fe_logits_blocks`, in the same order, and go to the workspace too, for whoever inspects it.
// Bound: latency, of the weights' trip (147 KB to a CTA with 384 experts of 3072) and of the selection. 1 token over 48 experts of 3072 4.2 us, 8 over 384 9.1.
constexpr int kFcThreads = 512;
constexpr int kFcTokens = 2;                 // tokens of a cluster at most

// kPer: experts per lane of the selecting warp; kChunks: 16 B chunks of half a row per lane (hidden <= 512 kChunks); kExperts: experts of a warp in flight
template <int kPer, int kChunks, int kExperts>
__global__ void __launch_bounds__(kFcThreads, 1) frontend_cluster_kernel(const __grid_constant__ FeParams q) {
    __shared__ uint4 xs[kFcTokens][kChunks * 64];
    __shared__ float parts[kFeParts][kPer * 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, rank = cluster_rank(), C = cluster_size();
    const uint32_t t0 = udiv_small(blockIdx.x, C) * q.cluster_tokens, nt = min(static_cast<uint32_t>(q.cluster_tokens), static_cast<uint32_t>(q.T) - t0);
    cluster_arrive();                        // (nobody writes into a CTA that has not started)
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t nchunk = q.H / 8, half = (nchunk + kFeParts - 1) / kFeParts, part = warp & 1u;
    const uint32_t c_lo = part * half + lane, c_hi = min(nchunk, part * half + half);
    const uint32_t e_lo = udiv_small(rank * q.E, C) + (warp >> 1), e_hi = udiv_small((rank + 1u) * q.E, C);
    constexpr uint32_t kStride = kFcThreads / 32 / kFeParts;
    #pragma unroll 1
    for (uint32_t e0 = e_lo;; e0 += kStride * kExperts) {
        uint4 w[kExperts][kChunks];
        #pragma unroll
        for (uint32_t k = 0; k < kExperts; ++k) {
            #pragma unroll
            for (uint32_t b = 0; b < kChunks; ++b) {
                const uint32_t e = e0 + k * kStride, ch = c_lo + 32u * b;
                if (e < e_hi && ch < c_hi) w[k][b] = __ldg(reinterpret_cast<const uint4*>(q.router_w + static_cast<size_t>(e) * q.H) + ch);
            }
        }
        if (e0 == e_lo) {                    // the tokens, behind the first weights' requests
            const uint4* src = reinterpret_cast<const uint4*>(q.hidden + static_cast<size_t>(t0) * q.H);
            for (uint32_t t = 0; t < nt; ++t)
                for (uint32_t i = tid; i < nchunk; i += kFcThreads) xs[t][i] = __ldg(src + t * nchunk + i);
            __syncthreads();
            cluster_wait();
        }
        if (e0 >= e_hi) break;
        #pragma unroll 1
        for (uint32_t t = 0; t < nt; ++t) {
            float acc[kExperts];
            #pragma unroll
            for (uint32_t k = 0; k < kExperts; ++k) acc[k] = 0.f;
            #pragma unroll
            for (uint32_t b = 0; b < kChunks; ++b) {
                if (c_lo + 32u * b < c_hi) {
                    float x[8];
                    unpack_bf16x8(xs[t][c_lo + 32u * b], x);
                    #pragma unroll
                    for (uint32_t k = 0; k < kExperts; ++k) {
                        float f[8];
                        unpack_bf16x8(w[k][b], f);       // (an expert beyond the last one: whatever was there, its sum is not stored)
                        #pragma unroll
                        for (int i = 0; i < 8; ++i) acc[k] = fmaf(x[i], f[i], acc[k]);
                    }
                }
            }
            #pragma unroll
            for (uint32_t k = 0; k < kExperts; ++k) {
                #pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
            }
            #pragma unroll
            for (uint32_t k = 0; k < kExperts; ++k) {
                const uint32_t e = e0 + k * kStride;
                if (lane == k && e < e_hi) {
                    st_cluster_f32(&parts[part][e], t, acc[k]);
                    st_volatile_v2(reinterpret_cast<uint8_t*>(q.logits) + (static_cast<size_t>(t0 + t) * q.E + e) * 16u + part * 8u, __float_as_uint(acc[k]), 1u);
                }
            }
        }
    }
    __syncwarp();
    cluster_arrive();
    const uint32_t t = t0 + rank;
    const __nv_bfloat16* row = reinterpret_cast<const __nv_bfloat16*>(xs[rank < nt ? rank : 0u]);
    bool nz = false;
    if (rank < nt && warp == 0u) nz = fe_row_nonzero(row, q.H, lane);
    if (rank < nt && warp != 0u) {           // (one warp for the whole token took 2 to 6 us, longer than the selection: 1 token over 48 experts of 3072 6.05 -> 4.2, NVFP4 8.3 -> 4.3)
        #pragma unroll 1
        for (uint32_t i = warp - 1u; i < static_cast<uint32_t>(q.H) / 256u; i += kFcThreads / 32 - 1)
            fe_quant_slice(row, q.fmt, q.x_gs, q.x + static_cast<size_t>(t) * q.x_row_bytes, q.x_sf + static_cast<size_t>(t) * q.x_sf_row_bytes, i, lane);
    }
    __syncwarp();
    cluster_wait();                          // (the last access to another CTA's shared memory lies before it)
    if (rank < nt && warp == 0u) {
        float lg[kPer];
        uint32_t key[kPer];
        #pragma unroll
        for (uint32_t h = 0; h < kPer; ++h) {
            const uint32_t e = lane + 32u * h;
            lg[h] = 0.f; key[h] = 0u;
            if (e < static_cast<uint32_t>(q.E)) {
                lg[h] = fe_logit(parts[0][e], parts[1][e]);
                key[h] = fe_key(q, lg[h], q.score_mode == 1 ? __ldg(q.bias + e) : 0.f);
            }
        }
        fe_choose<kPer>(q, t, nz, lane, 0u, nullptr, lg, key);
    }
}

}  // namespace mm
