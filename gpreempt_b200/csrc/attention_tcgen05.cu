// Multi-head self-attention on the tcgen05 tensor cores for the single-plane (bf16 / fp16)
// models: softmax(Q K^T / sqrt(d)) V with head dimension 64, no mask, sequences up to 512.
//
// Stands in for the batch_matmul + softmax + batch_matmul kernels TVM generates for the
// reference's BERT workload (scripts/compile/compile-bert.py:33-91; replayed by
// src/executor.cpp:157-162).  One tile = (batch item, head, block of 128 queries), claimed through
// the block-level preemption loop (scripts/compile/convert_to_blp.py:39-70).
//
// Two warpgroups share a tile's queries and take its blocks of 64 keys in turn, each with an online
// softmax of its own; their two partial results are merged at the end.  Per block: S = Q K^T as one
// 128x64x64 product into tensor memory; every thread owns one query row (its TMEM lane), reads the 64
// scores once, exponentiates them and writes the probabilities as a 16-bit A operand into shared
// memory (128-byte swizzled, as TMA would); P V is a 128x64x64 product accumulated in tensor memory,
// whose B operand is the value tile as it lies in HBM (rows are keys): the descriptor names it
// MN-major, so no transposed copy of the values exists.  The accumulated output is rescaled whenever a row's
// maximum has grown, so that the largest probability of a block is 1 and exact in 16 bits, and the normaliser
// sums the probabilities as rounded, so that an error they share cancels.  (Letting the exponent's
// reference lag behind the maximum by up to 2^8, as published attention kernels do, rounds the largest
// probability too.  Distance from 64 bits of rows that one key dominates, fp16: 2.32e-4 of the norm with
// the lag, 2.08e-4 without, 2.07e-4 with the rounded sum as well, where rounding the result is 2.06e-4; a layer
// of BERT-base s512 b32: 72, 77 and 78 us.)
//
// The scores of the next block are computed as soon as this block's have left tensor memory for
// registers (two key buffers), under this block's softmax; the values of the next block arrive
// under its exponentials (one value buffer: the next values are fetched when P V is complete).
//
// What bounds it: the special-function unit has 128 x 64 exponentials a block (512 cycles at 16 an SM
// and cycle, 22 us a layer of BERT-base s512 b32), everything else is latency between the two products;
// two CTAs of two independent warpgroups per SM overlap each other's, to ~30 % of that unit's rate.
// BERT-base s512 b32, a layer: one warpgroup of 128 keys a block with the output folded into registers
// and a transposing kernel in front took 89 + 16 us; scores and context issued in line, 82; by one warp of each
// group, 73.5; by two, with the next tile claimed under the last block of this one and its queries and first
// keys fetched under the merge, 70.  (Tried, at the same time or slower: a warp of its own for copies and
// products, two buffers of values, the next tile claimed under the merge without fetching anything of it.)
// The first two warps of a warpgroup issue TMA and MMA; every wait is bounded, and a wait that gives up raises
// a flag that ends all others, so the threads of a CTA pass the same barriers and leave together.
//
// A tile takes ~14 us at 512 keys with two CTAs per SM, so the word is read in every block of keys as
// well as between tiles: on a raised word both warpgroups leave at the end of a softmax, the CTA waits for
// its copies and products in flight, notes the tile and returns; launched again it recomputes that tile first
// (a redo costs at most a tile and keeps the instruction sequence, so results stay the same bits).  From the
// first look at the raised word to the last CTA's exit: p99 7.7 us, 13.7 when a claimed tile always completed.
#include "layers.cuh"
#include "sm100.cuh"

#include <type_traits>

namespace gpx {

using namespace sm100;

constexpr int kFaThreads = 256;
constexpr int kFaQ = 128, kFaKeys = 64, kFaD = 64;
constexpr uint32_t kFaQBytes = kFaQ * kFaD * 2;     // 16 KiB
constexpr uint32_t kFaKBytes = kFaKeys * kFaD * 2;  // 8 KiB, keys or values of a block
constexpr uint32_t kFaPBytes = kFaQ * kFaKeys * 2;  // 16 KiB
// per warpgroup: two K, V, P; both: Q, slack, control
constexpr uint32_t kFaGroupBytes = 3 * kFaKBytes + kFaPBytes;
constexpr uint32_t kFaSmem = kFaQBytes + 2 * kFaGroupBytes + 1024 + 2304;
constexpr uint32_t kFaTmemCols = 256;  // per warpgroup: S 64 columns, output 64 columns
constexpr unsigned long long kFaWaitLimitNs = 2000000000ull;

struct FaControl {
    unsigned long long bar_q;
    unsigned long long bar_s[2], bar_o[2], bar_v[2];  // per warpgroup
    unsigned long long bar_k[2][2];
    uint32_t tmem_base;
    int tile;
    int next;         // the tile after this one, if it was claimed under this one
    int abort_flag;
    int stop;         // the word was seen raised inside the tile
    int leave[2][2];  // [warpgroup][step parity] what its first thread made of that: the same for all of them
    int gave_up;      // a warpgroup has left the tile unfinished
    float ml[2][kFaQ][2];  // row maximum and normaliser of each warpgroup
};
static_assert(sizeof(FaControl) <= 2304, "control block outgrew its shared-memory budget");

// 2^x, the hardware approximation (relative error ~2^-22; -inf gives 0).
__device__ __forceinline__ float fa_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The largest of three (one instruction on this architecture).
__device__ __forceinline__ float fa_max3(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}

template <bool HALF>
__global__ void __launch_bounds__(kFaThreads, 2)
attention_tc_kernel(const __grid_constant__ AttnParams p, BlpArgs blp) {
    constexpr int FMT = HALF ? PF_F16 : PF_BF16;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    unsigned char *smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    FaControl *ctl = reinterpret_cast<FaControl *>(smem + kFaQBytes + 2 * kFaGroupBytes);
    volatile int *abort_flag = &ctl->abort_flag;
    const int tid = threadIdx.x;
    const int wg = __shfl_sync(0xffffffffu, tid >> 7, 0);  // warpgroup
    const int row = tid & 127;
    // The first warp of a warpgroup fetches keys and issues scores, the second fetches values and issues contexts: each
    // is ~500 cycles a block on top of the softmax, which all four warps wait for.
    const int wq = __shfl_sync(0xffffffffu, row >> 5, 0);
    const bool elected = elect_one(), warp0 = wq == 0, issuer = elected && warp0, issuer_v = elected && wq == 1;
    unsigned char *mine = smem + kFaQBytes + wg * kFaGroupBytes;
    const uint32_t sQ = smem_u32(smem), sK = smem_u32(mine), sV = sK + 2 * kFaKBytes, sP = sK + 3 * kFaKBytes;
    unsigned char *pV = mine + 2 * kFaKBytes, *pP = mine + 3 * kFaKBytes;

    if (tid == 0) {
        mbar_init(smem_u32(&ctl->bar_q), 1);
        for (int g = 0; g < 2; ++g) {
            mbar_init(smem_u32(&ctl->bar_s[g]), 1);
            mbar_init(smem_u32(&ctl->bar_o[g]), 1);
            mbar_init(smem_u32(&ctl->bar_v[g]), 1);
            mbar_init(smem_u32(&ctl->bar_k[g][0]), 1);
            mbar_init(smem_u32(&ctl->bar_k[g][1]), 1);
        }
        ctl->abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (tid < 32) tmem_alloc(smem_u32(&ctl->tmem_base), kFaTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    pdl_wait();  // the prologue above overlapped the predecessor's tail
    pdl_launch_dependents();
    if (tid == 0) trace_begin(blp);
    const uint32_t tmem_base = ctl->tmem_base;
    const uint32_t t_s = tmem_base + wg * 128, t_o = t_s + 64;          // as the products address them
    const uint32_t lane_off = (uint32_t)((row >> 5) * 32) << 16;        // as this warp's loads do
    constexpr uint32_t idesc = HALF ? make_idesc_f16_f32(kFaQ, 64) : make_idesc_bf16_f32(kFaQ, 64);
    constexpr uint32_t idesc_o = idesc | (1u << 16);  // B is MN-major: value rows are keys
    auto fail = [&](int code) {
        *abort_flag = 1;
        if (p.error && atomicCAS(p.error, 0, code) == 0) p.error[1] = blp.kernel_id * 1000 + (int)blockIdx.x;
    };
    auto wait = [&](unsigned long long *bar, uint32_t phase, int code) {
        if (!mbar_wait(smem_u32(bar), phase, abort_flag, kFaWaitLimitNs)) fail(code);
    };
    auto group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + wg) : "memory"); };

    const int qblocks = (p.S + kFaQ - 1) / kFaQ;
    const int nkb = (p.S + kFaKeys - 1) / kFaKeys;
    const int steps = (nkb - wg + 1) / 2;  // blocks wg, wg + 2, ... of this warpgroup
    const float scale_log2 = p.scale * 1.4426950408889634f;  // scores are exponentiated base 2
    uint32_t ph_q = 0, ph_s = 0, ph_o = 0, ph_v = 0, ph_k = 0;  // (ph_k: bit b for key buffer b)
    // A preemptible launch gives an unfinished tile up when the word goes up: the CTA notes it (two CTAs
    // share a slot) and takes it first when it is launched again.
    int *const given_up = blp.preempted && p.slots
                              ? (blockIdx.x & 1 ? &p.slots[blockIdx.x >> 1].k_done : &p.slots[blockIdx.x >> 1].next_iter) : nullptr;
    int pending = given_up && tid == 0 ? *given_up - 1 : -1;
    auto stop_here = [&]() {
        if (blp.trace) atomicMin(blp.trace + 2, globaltimer_ns());
        atomicCAS(blp.stop_index, -1, blp.kernel_id);
    };
    struct At {
        int qb, head, b, col0, key_row0;
    };
    auto at_tile = [&](int tile) {
        At a;
        a.qb = tile % qblocks;
        a.head = (tile / qblocks) % p.heads;
        a.b = tile / (qblocks * p.heads);
        a.col0 = a.head * kFaD, a.key_row0 = a.b * p.S;
        return a;
    };
    auto fetch = [&](const At &a, uint32_t dst, const void *map, unsigned long long *bar, int step) {
        mbar_arrive_expect_tx(smem_u32(bar), kFaKBytes);
        tma_load_2d(dst, map, smem_u32(bar), a.col0, a.key_row0 + (2 * step + wg) * kFaKeys);
    };
    // queries, and this warpgroup's first keys, of a tile
    auto fetch_first = [&](const At &a) {
        if (tid == 0) {
            mbar_arrive_expect_tx(smem_u32(&ctl->bar_q), kFaQBytes);
            tma_load_2d(sQ, &p.tq, smem_u32(&ctl->bar_q), a.col0, a.key_row0 + a.qb * kFaQ);
        }
        if (issuer && steps > 0) {
            fetch(a, sK, &p.tk, &ctl->bar_k[wg][0], 0);
            if (steps > 1) fetch(a, sK + kFaKBytes, &p.tk, &ctl->bar_k[wg][1], 1);
        }
    };
    // The next tile is claimed under the last block of this one (its word and its cursor are on their way under the
    // exponentials and behind them), when this one can no longer be given up, and its queries and first keys are
    // fetched under the merge.
    const bool claims = tid == 96;
    const bool more = blp.total_tiles > (int)gridDim.x;  // (with a CTA for every tile each runs one)
    int next = -1, iter = 0;
    for (;; ++iter) {
        const bool fetched = next >= 0;
        if (tid == 0) {
            int t = -1;
            if (*abort_flag || next == -2) {  // (-2: the last tile has been claimed)
            } else if (fetched) {
                t = next;
            } else if (pending < 0) {
                t = blp_claim(blp, iter);
            } else if (load_word(blp.preempted) != 0) {
                stop_here();  // (the note stays)
            } else {
                t = pending;
                pending = -1;
                *given_up = 0;
            }
            ctl->tile = t;
            ctl->next = -1;
            ctl->stop = ctl->gave_up = 0;
        }
        __syncthreads();
        const int tile = ctl->tile;
        if (tile < 0) break;
        next = -1;
        const At at = at_tile(tile);
        const int b = at.b, q0 = at.qb * kFaQ, col0 = at.col0;
        if (!fetched) fetch_first(at);
        if (issuer_v && steps > 0) fetch(at, sV, &p.tv, &ctl->bar_v[wg], 0);
        // S = Q K^T of block j (warp 0; the lane that issues it)
        auto scores = [&](int j) {
            const int kb = j & 1;
            wait(&ctl->bar_k[wg][kb], (ph_k >> kb) & 1, 402);
            ph_k ^= 1u << kb;
            tc_fence_after_sync();
            if (issuer && !*abort_flag) {
                const uint64_t dq = make_smem_desc_sw128(sQ), dk = make_smem_desc_sw128(sK + kb * kFaKBytes);
#pragma unroll
                for (int k = 0; k < kFaD / 16; ++k) mma_f16_ss(t_s, dq + 2 * k, dk + 2 * k, idesc, k > 0 ? 1u : 0u);
                mma_commit(smem_u32(&ctl->bar_s[wg]));
            }
            __syncwarp();
        };
        float m = -INFINITY, l = 0.f;
        __syncwarp();
        if (steps > 0 && warp0) {
            wait(&ctl->bar_q, ph_q, 401);
            scores(0);
        }
        ph_q ^= 1;
        bool left = false;
        for (int j = 0; j < steps; ++j) {
            wait(&ctl->bar_s[wg], ph_s, 403);
            ph_s ^= 1;
            tc_fence_after_sync();
            const bool may_leave = given_up && j + 1 < steps;
            const bool ask = claims && more && j + 1 == steps;
            int word = 0;  // looked at when the softmax, which hides the read, is through
            if ((may_leave && tid == 0) || (ask && blp.preempted)) word = load_word(blp.preempted);
            if (issuer && j + 2 < steps && !*abort_flag) fetch(at, sK + (j & 1) * kFaKBytes, &p.tk, &ctl->bar_k[wg][j & 1], j + 2);  // S is done with the keys
            uint32_t v[64];
            {
                uint32_t a[32], c[32];
                __syncwarp();
                tmem_ld_32x32(t_s + lane_off, a);
                tmem_ld_32x32(t_s + lane_off + 32, c);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = a[i], v[32 + i] = c[i];
            }
            if (j + 1 < steps) {
                // The scores are in registers: the next block's products run under this block's softmax.
                tc_fence_before_sync();
                group_sync();
                if (warp0) scores(j + 1);
            }
            const int key0 = (2 * j + wg) * kFaKeys;
            const int keys = p.S - key0 < kFaKeys ? p.S - key0 : kFaKeys;
            if (keys < kFaKeys) {
#pragma unroll
                for (int i = 0; i < 64; ++i)
                    if (i >= keys) v[i] = 0xff800000u;  // -inf
            }
            // (of the raw scores: the scale is positive)
            float bmax = fa_max3(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]));
            float bmax2 = fa_max3(__uint_as_float(v[3]), __uint_as_float(v[4]), __uint_as_float(v[5]));
#pragma unroll
            for (int i = 6; i < 62; i += 4) {
                bmax = fa_max3(bmax, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
                bmax2 = fa_max3(bmax2, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
            }
            bmax = fa_max3(fmaxf(bmax, bmax2), __uint_as_float(v[62]), __uint_as_float(v[63]));
            const float m_new = fmaxf(m, bmax * scale_log2);
            // P V of the block before: its probabilities and values are free, its output is complete
            if (j > 0) {
                wait(&ctl->bar_o[wg], ph_o, 404);
                ph_o ^= 1;
                if (issuer_v && !*abort_flag) fetch(at, sV, &p.tv, &ctl->bar_v[wg], j);
            } else {
                m = m_new;
            }
            if (__any_sync(0xffffffffu, m_new > m)) {
                const float alpha = fa_ex2(m - m_new);
                tc_fence_after_sync();
#pragma unroll
                for (int c = 0; c < kFaD; c += 16) {
                    uint32_t o[16];
                    tmem_ld_32x16(t_o + lane_off + c, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                    tmem_st_32x16(t_o + lane_off + c, o);
                }
                tmem_st_wait();
                l *= alpha;
                m = m_new;
            }
            const int r8 = row & 7;
            unsigned char *prow = pP + (row >> 3) * 1024 + r8 * 128;
            float lsum[4] = {0.f, 0.f, 0.f, 0.f};
            const float2 sc2 = make_float2(scale_log2, scale_log2), neg_m = make_float2(-m, -m);
#pragma unroll
            for (int c = 0; c < 64; c += 8) {
                uint32_t pk[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 x = fma2(make_float2(__uint_as_float(v[c + 2 * i]), __uint_as_float(v[c + 2 * i + 1])), sc2, neg_m);
                    pk[i] = pf_pack2(fa_ex2(x.x), fa_ex2(x.y), FMT);
                    const float2 e = pf_unpack2(pk[i], FMT);
                    lsum[i] += e.x + e.y;
                }
                // eight keys = one 16-byte piece of this row, at piece index XOR (row mod 8)
                *reinterpret_cast<uint4 *>(prow + (((c >> 3) ^ r8) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            }
            l += (lsum[0] + lsum[1]) + (lsum[2] + lsum[3]);
            if (ask) {
                // (with the word up nothing is claimed here; the claim at the top of the loop records the stop point)
                if (!blp.preempted)
                    next = (int)blockIdx.x + (iter + 1) * (int)gridDim.x;
                else if (word == 0)
                    next = atomicAdd(blp.executed, 1);
            }
            if (keys < kFaKeys) {
                // Rows past the sequence belong to the next batch item: their probabilities are zero, and
                // so must they be (zero times an infinity is not).
                wait(&ctl->bar_v[wg], ph_v, 405);
                for (int e = row; e < (kFaKeys - keys) * 8; e += 128)
                    *reinterpret_cast<uint4 *>(pV + (keys + (e >> 3)) * 128 + (e & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
            fence_proxy_async();  // the probabilities were written by ordinary stores, the MMA reads them
            tc_fence_before_sync();
            if (may_leave && row == 0) {
                if (word != 0) *(volatile int *)&ctl->stop = 1;
                ctl->leave[wg][j & 1] = *(volatile int *)&ctl->stop;
            }
            group_sync();
            if (may_leave && ctl->leave[wg][j & 1]) {
                // what is still on its way lands first: these values, the next scores, the keys after them
                wait(&ctl->bar_v[wg], ph_v, 407);
                wait(&ctl->bar_s[wg], ph_s, 407);
                if (warp0 && j + 2 < steps) wait(&ctl->bar_k[wg][j & 1], (ph_k >> (j & 1)) & 1, 407);
                if (row == 0) ctl->gave_up = 1;
                left = true;
                break;
            }
            if (wq == 1) {
                wait(&ctl->bar_v[wg], ph_v, 405);
                tc_fence_after_sync();
                if (issuer_v && !*abort_flag) {
                    const uint64_t dp = make_smem_desc_sw128(sP);
                    // Value tile: 64 keys x 128 bytes, 128-byte swizzle.  As an MN-major operand eight keys
                    // are 1024 bytes apart from the next eight, and the 64 output columns are one swizzle
                    // atom wide; a step of sixteen keys is 2048 bytes (128 in the descriptor's units).
                    const uint64_t dv = make_smem_desc_sw128(sV) | ((uint64_t)(1024 >> 4) << 16);
#pragma unroll
                    for (int k = 0; k < kFaKeys / 16; ++k)
                        mma_f16_ss(t_o, dp + 2 * k, dv + 128 * k, idesc_o, (j > 0 || k > 0) ? 1u : 0u);
                    mma_commit(smem_u32(&ctl->bar_o[wg]));
                }
                __syncwarp();
            }
            ph_v ^= 1;
        }
        if (steps > 0 && !left) {
            wait(&ctl->bar_o[wg], ph_o, 406);
            ph_o ^= 1;
        }
        tc_fence_after_sync();
        __syncwarp();
        // ---- merge: warpgroup g finishes columns 32 g .. 32 g + 31, the other 32 go through shared memory
        // (this warpgroup's V tile and half its P tile, free by now: [column][row] floats)
        float keep[32];
        if (!left) {
            uint32_t o[32];
            float *give = reinterpret_cast<float *>(pV);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (steps > 0) {
                    tmem_ld_32x32(t_o + lane_off + 32 * half, o);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = 0u;
                }
                if (half == wg) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) keep[i] = __uint_as_float(o[i]);
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) give[i * kFaQ + row] = __uint_as_float(o[i]);
                }
            }
            ctl->ml[wg][row][0] = m;
            ctl->ml[wg][row][1] = l;
            if (claims && next != -1) ctl->next = next < blp.total_tiles ? next : -2;
        }
        tc_fence_before_sync();
        __syncthreads();
        next = ctl->next;
        if (next >= 0 && !*abort_flag) fetch_first(at_tile(next));
        if (ctl->gave_up) {
            if (tid == 0) {
                *given_up = tile + 1;
                stop_here();
            }
            break;
        }
        if (q0 + row < p.S) {
            const float m0 = ctl->ml[0][row][0], m1 = ctl->ml[1][row][0];
            const float mm = fmaxf(m0, m1);
            const float a0 = fa_ex2(m0 - mm), a1 = fa_ex2(m1 - mm);
            const float inv = 1.0f / (ctl->ml[0][row][1] * a0 + ctl->ml[1][row][1] * a1);
            const float f_mine = (wg == 0 ? a0 : a1) * inv, f_other = (wg == 0 ? a1 : a0) * inv;
            const float *take = reinterpret_cast<const float *>(smem + kFaQBytes + (wg ^ 1) * kFaGroupBytes + 2 * kFaKBytes);
            uint32_t w[16];
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                const float x = fmaf(take[i * kFaQ + row], f_other, keep[i] * f_mine);
                const float y = fmaf(take[(i + 1) * kFaQ + row], f_other, keep[i + 1] * f_mine);
                w[i >> 1] = pf_pack2(x, y, FMT);
            }
            bf16_bits *dst = p.out_hi + ((size_t)b * p.S + q0 + row) * p.ld_out + col0 + 32 * wg;
            st_sector(dst, w);
            st_sector(dst + 16, w + 8);
        }
        fence_proxy_async();  // TMA writes the next tile's operands where ordinary accesses were made
        __syncthreads();
        if (*abort_flag) {
            for (int spin = 0; spin < 64; ++spin) __nanosleep(1000);  // copies in flight land before the CTA ends
            break;
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (tid < 32) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kFaTmemCols);
    }
    if (tid == 0) trace_end(blp, iter);
}

cudaError_t attention_tc_prepare() {
    cudaError_t e = cudaFuncSetAttribute(attention_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFaSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(attention_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFaSmem);
}

int attention_tc_threads() { return kFaThreads; }

cudaError_t attention_tc_launch(const AttnParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    return launch_layer(p.fmt == PF_F16 ? attention_tc_kernel<true> : attention_tc_kernel<false>, grid, kFaThreads, kFaSmem, s, p, blp);
}

}  // namespace gpx
