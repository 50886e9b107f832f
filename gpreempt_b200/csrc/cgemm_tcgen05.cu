// Convolution as a row-shifted GEMM on the tcgen05 tensor cores, fp32 accuracy from split-bf16
// operands, K-block-granular preemption.
//
// Stands in for the TVM-generated fused conv2d(+bias)(+add)(+relu) kernels the reference
// replays (src/executor.cpp:157-162).  Activations and weights are stored as two bf16 planes
// (x ~= hi + lo); one fp32 product is three tensor-core products hi*hi + hi*lo + lo*hi
// accumulated in fp32 in tensor memory, which keeps 16 mantissa bits per operand and meets the
// 1e-4 parity bound of the fp32 configuration at a third of the bf16 tensor rate.
//
// GEMM view: rows are stored pixels of the input (see act_layout.h), a filter tap is a constant
// row shift, so the A operand of every K block is a plain 2-D TMA tile [128 rows][64 channels]
// at row (m0 + shift[tap]); rows outside the tensor are zero-filled by TMA.  B is the weight
// matrix [Cout][taps*Cin].  Rows that are not real output pixels (image borders of the padded
// layouts) are computed and dropped by the epilogue.
//
// Single-plane models (bf16 / fp16 storage) use the same kernel with one product per K step and
// twice as many ring stages.
//
// CTA roles, ring, messages and the preempt / spill / resume protocol are those of
// gemm_tcgen05.cu, with two accumulator buffers in tensor memory so that the epilogue of one
// tile overlaps the K loop of the next.  The epilogue adds the bias, applies the activation,
// splits the fp32 result into the plane format and writes each row into the consumer's layout
// with 256-bit stores.  The residual of a 1x1 convolution on plain rows is added by the tensor
// core itself: extra K blocks whose A operand is the residual tile and whose B operand is a
// 64x64 identity tile kept in shared memory; other residuals are added by the epilogue.
#include "layers.cuh"
#include "sm100.cuh"

#include <cuda_bf16.h>
#include <type_traits>

namespace gpx {

using namespace sm100;

constexpr int kCBM = 128, kCBK = 64, kCUmmaK = 16;
// Warp 0 feeds TMA, warp 1 issues MMAs, warps from 2 on are the epilogue, the last warp polls the preempt
// word: kEpiParts epilogue warps per TMEM lane quarter, each taking an equal share of the columns,
// so that enough independent TMEM loads, conversions and stores are in flight while a tile is drained
// (the epilogue, not the tensor pipe, bounds the small-K layers).
constexpr int kCAffGroup = 128;  // threads of a group that maps an A operand; groups take K blocks in turn
constexpr int kCAffMaxC = kCgemmMaxAffineC;
constexpr unsigned long long kCWaitLimitNs = 2000000000ull;


struct CgemmControlSize {
    unsigned char bytes[2560];  // room for CgemmControl (checked below)
};

// BN: columns of an output tile.  TWO: two-plane operands (float32 models), three products per K step;
// otherwise one 16-bit plane and one product.
// CL: the CTAs of a cluster share the K range of a 64-column tile and reduce it among themselves
// (latency-critical launches, one tile a CTA); the sixteen epilogue warps halve the chain of
// instructions behind the products, which is what such a launch waits for.
template <int BN, bool TWO, bool AFF, bool CL>
struct CgemmCfg {
    static constexpr int kEpiParts = BN == 256 || (CL && !AFF) ? 4 : 2;  // epilogue warps per TMEM lane quarter
    static constexpr int kEpiThreads = 128 * kEpiParts;
    static constexpr int kPollWarp = 2 + kEpiThreads / 32;
    static constexpr int kAffGroups = !AFF ? 0 : (!TWO && !CL ? 3 : 2);
    static constexpr int kThreads = 64 + kEpiThreads + 32 + kAffGroups * kCAffGroup;
    static constexpr uint32_t kPlanes = TWO ? 2 : 1;
    static constexpr uint32_t kABytes = kCBM * kCBK * 2;        // one plane of A: 16 KiB
    static constexpr uint32_t kWBytes = BN * kCBK * 2;          // one plane of W
    static constexpr uint32_t kKbBytes = kPlanes * (kABytes + kWBytes);  // operands of one K block
    static constexpr uint32_t kWOff = kPlanes * kABytes;        // W (hi) tile inside a K block
    // K blocks a ring stage holds at most.  The round of one stage (barrier waits, message, commit) costs
    // either role ~300 cycles; a 64- or 128-column product of one plane takes 128 or 256, so two
    // of them share a round, unless the affine map sets the pace (VGG-16's 64-column layer at batch 16: 168 -> 121 us).
    static constexpr int kKps = (!TWO && !AFF && BN <= 128) ? 2 : 1;
    static constexpr uint32_t kStageBytes = kKps * kKbBytes;
    static constexpr int kStages = (int)((192u * 1024u) / kStageBytes);  // 3 to 8
    // ring stages the landing area of a cluster reduction takes (128 rows of BN floats)
    static constexpr int kLandStages = CL ? (int)((kCBM * BN * 4 + kStageBytes - 1) / kStageBytes) : 0;
    static constexpr int kRing = kStages - kLandStages;  // stages in use as the ring where there is one
    // ring + alignment slack + 64x64 identity tile + control block
    static constexpr uint32_t kIdentBytes = 64 * kCBK * 2;
    static constexpr size_t kSmem =
        (size_t)kStages * kStageBytes + 1024 + kIdentBytes + sizeof(CgemmControlSize) + (AFF ? 2 * kCAffMaxC * sizeof(float) : 0);
    // Accumulator columns of one tile: hi*hi and both cross terms for two-plane operands, one sum
    // otherwise; two tiles' worth of them in tensor memory, so that the epilogue of one tile overlaps
    // the K loop of the next.
    static constexpr int kBufCols = (int)kPlanes * BN;
    // The mapped A operand of a stage goes to tensor memory (32 columns) where the accumulators leave room: two planes
    // do not, and a latency-critical launch of three or four K blocks a CTA gains nothing (DenseNet-201 b1 bf16 1 061 us, 1 067).
    static constexpr int kACols = 2 * kBufCols;
    static constexpr bool kTmemA = AFF && !TWO && !CL && kACols + 32 * kStages <= 512;
    static constexpr int kTmemCols = kTmemA ? 512 : 2 * kBufCols;
    static_assert(kTmemCols <= 512 && kStages <= 8, "tile does not fit");
    static_assert(kRing >= 3 && (!CL || BN == 64), "no ring left beside the landing area");
};

// Message of a ring stage: CMSG_DATA + number of K blocks, CMSG_RES + index of the residual block, or
// the word was seen raised.  (The end of a CTA's schedule needs no message: every role counts tiles.)
enum : int { CMSG_STOP = 1, CMSG_DATA = 4, CMSG_RES = 16 };
enum : int { CEPI_COMPLETE = 0, CEPI_PARTIAL = 1, CEPI_EXIT = 2 };

struct CgemmControl {
    unsigned long long full[8];
    unsigned long long empty[8];
    unsigned long long ready[8];       // the A tile of a stage has been through its affine map
    unsigned long long landed;         // cluster reduction: every peer's partial rows have arrived
    unsigned long long tmem_full[2];   // one per accumulator buffer
    unsigned long long tmem_empty[2];
    uint32_t tmem_base;
    int stage_msg[8];
    int epi_kind[2];
    int epi_k_done[2];
    int epi_go[2];
    int raised;      // the word was up when this CTA started
    int word_up;     // the polling warp has seen the word raised
    int poll_done;   // the producer is through: the polling warp returns
    int abort_flag;
    alignas(16) float bias_s[2][256];  // bias of the tile each accumulator buffer holds, staged by the epilogue
};

static_assert(sizeof(CgemmControl) <= sizeof(CgemmControlSize), "control block outgrew its shared-memory budget");

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&p);
}
// 256-bit global load (32-byte aligned): one whole sector per lane.
__device__ __forceinline__ void ld_global_v8(const void *ptr, uint32_t *r) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "l"(ptr));
}
__device__ __forceinline__ float bf16_lo_to_f32(uint32_t packed) { return __uint_as_float(packed << 16); }
__device__ __forceinline__ float bf16_hi_to_f32(uint32_t packed) {
    return __uint_as_float(packed & 0xffff0000u);
}

// Phase timers of a development build (-DGPX_CGEMM_TIMING): clock64 deltas summed over CTAs into a
// device array that gpx_debug_cgemm_timing reads.  Compiled out otherwise.
#ifdef GPX_CGEMM_TIMING
__device__ unsigned long long g_cgemm_timing[32];
#define TCK(var) long long var = clock64()
#define TADD(slot, val) atomicAdd(&g_cgemm_timing[slot], (unsigned long long)(val))
#else
#define TCK(var)
#define TADD(slot, val)
#endif

template <int BN, bool TWO, bool AFF, bool CL>
__global__ void __launch_bounds__(CgemmCfg<BN, TWO, AFF, CL>::kThreads, 1)
cgemm_tcgen05_kernel(const __grid_constant__ CgemmParams p, BlpArgs blp) {
    using Cfg = CgemmCfg<BN, TWO, AFF, CL>;
    constexpr int kStages = Cfg::kStages;
    constexpr int kBufCols = Cfg::kBufCols;
    TCK(t_start);
    // The prologue below (barriers, tensor memory, descriptor prefetch) touches nothing a
    // predecessor kernel writes, so it runs while that kernel drains; pdl_wait() comes after it.
    extern __shared__ unsigned char smem_raw[];
    uint32_t raw_addr = smem_u32(smem_raw);
    uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
    unsigned char *smem = smem_raw + pad;
    // The identity tile follows the ring (1024-byte aligned, as its swizzled layout needs).
    constexpr uint32_t ident_off = kStages * Cfg::kStageBytes;
    CgemmControl *ctl = reinterpret_cast<CgemmControl *>(smem + ident_off + Cfg::kIdentBytes);
    const uint32_t smem_base = smem_u32(smem);
    volatile int *abort_flag = &ctl->abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    // A tile is (row block, column block, K split); splits of one output block are adjacent so
    // they run at the same time.  With k_splits == 1 a tile covers the whole K range.
    const int total_tiles = p.tiles_m * p.tiles_n * p.k_splits;
    const int all_kb = p.taps * p.cin_blocks;
    struct TileAt {
        int m_blk, n_blk, split, kb_base, main_kb;
    };
    auto tile_at = [&](int tile) {
        TileAt t;
        const int otile = p.k_splits == 1 ? tile : fast_div(tile, p.k_splits, p.inv_k_splits);
        t.split = tile - otile * p.k_splits;
        // Column tiles vary fastest: CTAs that run together share the same A rows.
        t.m_blk = p.tiles_n == 1 ? otile : fast_div(otile, p.tiles_n, p.inv_tiles_n);
        t.n_blk = otile - t.m_blk * p.tiles_n;
        t.kb_base = t.split * p.kb_per_split;
        const int left = all_kb - t.kb_base;
        t.main_kb = left < p.kb_per_split ? left : p.kb_per_split;
        return t;
    };
    const bool resumable = !CL && blp.preempted != nullptr;
    // (with one split nothing lands, and the ring has all stages: VGG-16 of two images, whose layers of 28x28 pixels are 120
    // tiles of 72 K blocks, float32 544 us with one stage fewer, 534 with all; bf16 332 and 329)
    const int nst = CL && p.k_splits == 1 ? Cfg::kStages : Cfg::kRing;

    CgemmSlot *slot = p.slots + blockIdx.x;
    float *spill = p.spill + (size_t)blockIdx.x * kCgemmSpillFloats;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&ctl->full[s]), 1);
            mbar_init(smem_u32(&ctl->empty[s]), 1);
            if (AFF) mbar_init(smem_u32(&ctl->ready[s]), kCAffGroup / 32);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&ctl->tmem_full[b]), 2);
            mbar_init(smem_u32(&ctl->tmem_empty[b]), 1);
            ctl->epi_kind[b] = CEPI_COMPLETE;
            ctl->epi_k_done[b] = 0;
        }
        if (CL) {
            // a row of the share this CTA finishes comes from each of the other CTAs, if it is a row of the GEMM,
            // and from this CTA's own epilogue warps
            const int share = kCBM / p.k_splits;
            const int rows = p.m_rows - tile_at(blockIdx.x).m_blk * kCBM - (int)cluster_ctarank() * share;
            mbar_init(smem_u32(&ctl->landed), 1 + Cfg::kEpiThreads / 32);
            if (rows > 0 && p.k_splits > 1)
                mbar_arrive_expect_tx(smem_u32(&ctl->landed), (uint32_t)((rows < share ? rows : share) * (p.k_splits - 1) * BN * 4));
            else
                mbar_arrive(smem_u32(&ctl->landed));
        }
        ctl->abort_flag = 0;
        ctl->epi_go[0] = ctl->epi_go[1] = 0;
        ctl->raised = 0;
        ctl->word_up = 0;
        ctl->poll_done = 0;
        fence_barrier_init();
        fence_proxy_async();
        prefetch_tensormap(&p.a_hi);
        prefetch_tensormap(&p.w_hi);
        if (TWO) {
            prefetch_tensormap(&p.a_lo);
            prefetch_tensormap(&p.w_lo);
        }
    }
    // scale and shift of every input channel (parameters: no kernel writes them), zero past the last
    float *aff_s = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(ctl) + sizeof(CgemmControlSize));
    if (AFF)
        for (int c = threadIdx.x; c < p.cin_blocks * kCBK; c += Cfg::kThreads) {
            aff_s[c] = c < p.aff_c ? __ldg(p.aff_scale + c) : 0.f;
            aff_s[kCAffMaxC + c] = c < p.aff_c ? __ldg(p.aff_shift + c) : 0.f;
        }
    if (warp == 1) tmem_alloc(smem_u32(&ctl->tmem_base), Cfg::kTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = ctl->tmem_base;
    if (CL) cluster_arrive();  // this CTA runs: its shared memory may be written to

    // A non-preemptible launch knows its first tile without reading the cursor, and parameters are
    // never written by a kernel: its producer warp fetches the weight tiles of the first ring
    // stages before it waits for the predecessor, so that their latency overlaps the
    // predecessor's tail (batch-1 forwards are chains of such latencies).  The other roles go to their
    // places before the predecessor has finished too: only activations (the producer's A tiles, the
    // epilogue's residual and its stores) wait for it.  Every thread of a preemptible launch waits here.
    const bool early_weights = !resumable && (int)blockIdx.x < total_tiles;
    int prearmed = 0;  // K blocks whose barrier is armed and whose weight loads are in flight
    constexpr int KPS = Cfg::kKps;
    TileAt first_tile{};
    int tap0 = 0, cb0 = 0;  // filter tap and channel block of its first K block
    if (early_weights) first_tile = tile_at(blockIdx.x);
    const bool issuer = elect_one();
    if (early_weights && warp == 0) {
        prearmed = first_tile.main_kb < nst * KPS ? first_tile.main_kb : nst * KPS;
        tap0 = p.taps == 1 ? 0 : fast_div(first_tile.kb_base, p.cin_blocks, p.inv_cin_blocks);
        cb0 = first_tile.kb_base - tap0 * p.cin_blocks;
        int cb = cb0, w_tap = tap0 * p.cin, st = 0;
        for (int kb = 0; kb < prearmed; ++st) {
            const uint32_t bar = smem_u32(&ctl->full[st]);
            const int n = prearmed - kb < KPS ? prearmed - kb : KPS;
            if (issuer) {
                const uint32_t ident_bytes = (p.res_kb && kb == 0) ? Cfg::kIdentBytes : 0u;
                ctl->stage_msg[st] = CMSG_DATA + n;
                mbar_arrive_expect_tx(bar, n * Cfg::kKbBytes + ident_bytes);
                if (ident_bytes) tma_load_2d(smem_base + ident_off, &p.ident, bar, 0, 0);
            }
#pragma unroll
            for (int j = 0; j < KPS; ++j) {
                if (j > 0 && j >= n) break;
                const uint32_t dst = smem_base + st * Cfg::kStageBytes + j * Cfg::kKbBytes;
                if (issuer) {
                    tma_load_2d(dst + Cfg::kWOff, &p.w_hi, bar, w_tap + cb * kCBK, first_tile.n_blk * BN);
                    if (TWO) tma_load_2d(dst + Cfg::kWOff + Cfg::kWBytes, &p.w_lo, bar, w_tap + cb * kCBK, first_tile.n_blk * BN);
                }
                if (++cb == p.cin_blocks) {
                    cb = 0;
                    w_tap += p.cin;
                }
            }
            kb += n;
        }
        __syncwarp();
    }
    if (!CL || warp == 0) {
        pdl_wait();  // from here on the predecessor's results (and this executor's slots) are visible
        pdl_launch_dependents();
    }
    TCK(t_begin);

    // A non-preemptible launch never stops early, so it neither reads nor writes the cursor.
    const int first_iter = resumable ? slot->next_iter : 0;
    const int first_k = resumable ? slot->k_done : 0;
    const int slot_grid = resumable ? slot->grid : 0;

    // A kernel that starts while the word is raised (it was queued behind the stop point) leaves
    // at once: the cursor is unchanged, the stop point is recorded if this CTA still has work
    // (kernel_transform_be.py:10-12).
    if (resumable) {
        if (threadIdx.x == 0) {
            const int raised = load_word(blp.preempted);
            if (raised) {
                if ((int)blockIdx.x + first_iter * (int)gridDim.x < total_tiles && blp.stop_index)
                    atomicCAS(blp.stop_index, -1, blp.kernel_id);
                if (blp.trace) {
                    unsigned long long t = globaltimer_ns();
                    atomicMin(blp.trace + 0, t);
                    atomicMin(blp.trace + 2, t);
                    atomicMax(blp.trace + 1, t);
                }
            }
            ctl->raised = raised;
        }
        tc_fence_before_sync();
        __syncthreads();
        if (ctl->raised) {
            if (warp == 1) {
                tc_fence_after_sync();
                tmem_dealloc(tmem_base, Cfg::kTmemCols);
            }
            return;
        }
    }
    if (threadIdx.x == 0) trace_begin(blp);
#ifdef GPX_CGEMM_TIMING
    if (threadIdx.x == 0) TADD(14, clock64() - t_start);
#endif

    const bool grid_ok = slot_grid == 0 || slot_grid == (int)gridDim.x;
    auto fail = [&](int code) {
        ctl->abort_flag = 1;
        if (atomicCAS(p.error, 0, code) == 0) p.error[1] = blp.kernel_id * 1000 + (int)blockIdx.x;
    };

    if (!grid_ok) {
        if (threadIdx.x == 0) fail(900);
    } else if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        // The whole warp walks the schedule and one elected lane issues: warp-uniform control flow
        // keeps coordinates, addresses and barriers on the uniform datapath, where the TMA instruction
        // reads them.  (tap, channel block) advance by counting; dividing by cin_blocks for every K
        // block, on a lone thread, was a third of the ~780 cycles a K block cost here before.
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        // The identity tile travels with the first stage this CTA fills.
        uint32_t ident_bytes = (p.res_kb && prearmed == 0) ? Cfg::kIdentBytes : 0u;
        const volatile int *word_up = &ctl->word_up;
        TCK(t_prod0);
#ifdef GPX_CGEMM_TIMING
        long long prod_wait = 0;
#endif
        int kb = first_k;
        int tap = tap0, cb = cb0;
        if (prearmed) {
            // The weights of these stages are already on their way: only activations are missing.
            const int row0 = first_tile.m_blk * kCBM;
            int a_row = row0 + p.tap_shift[tap];
            for (; kb < prearmed; ++stage) {
                const uint32_t bar = smem_u32(&ctl->full[stage]);
                const int n = prearmed - kb < KPS ? prearmed - kb : KPS;
#pragma unroll
                for (int j = 0; j < KPS; ++j) {
                    if (j > 0 && j >= n) break;
                    const uint32_t dst = smem_base + stage * Cfg::kStageBytes + j * Cfg::kKbBytes;
                    if (issuer) {
                        tma_load_2d(dst, &p.a_hi, bar, cb * kCBK, a_row);
                        if (TWO) tma_load_2d(dst + Cfg::kABytes, &p.a_lo, bar, cb * kCBK, a_row);
                    }
                    if (++cb == p.cin_blocks) {
                        cb = 0;
                        if (++tap < p.taps) a_row = row0 + p.tap_shift[tap];
                    }
                }
                kb += n;
            }
            __syncwarp();
            if (stage == nst) {
                stage = 0;
                phase ^= 1;
            }
        }
        for (int it = first_iter; ok; ++it, kb = 0) {
            const int tile = blockIdx.x + it * gridDim.x;
            if (tile >= total_tiles) break;
            const TileAt t = tile_at(tile);
            const int num_kb = t.main_kb + p.res_kb;  // the residual rides along as extra K blocks
            const int row0 = t.m_blk * kCBM, w_row = t.n_blk * BN;
            if (it > first_iter || !prearmed) {
                const int kb_abs = t.kb_base + kb;
                tap = p.taps == 1 ? 0 : fast_div(kb_abs, p.cin_blocks, p.inv_cin_blocks);
                cb = kb_abs - tap * p.cin_blocks;
            }
            int a_row = row0 + p.tap_shift[tap < p.taps ? tap : 0];
            int w_tap = tap * p.cin;
            while (kb < num_kb) {
                const uint32_t bar = smem_u32(&ctl->full[stage]);
                const uint32_t dst = smem_base + stage * Cfg::kStageBytes;
                TCK(t_w0);
                // (looked at before the wait, which hides it: what follows the wait delays the ring)
                const bool stop = resumable && __any_sync(0xffffffffu, *word_up);
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->empty[stage]), phase ^ 1, abort_flag, kCWaitLimitNs))) {
                    if (lane == 0) fail(101);
                    ok = false;
                    break;
                }
                if (stop) {
                    if (issuer) {
                        ctl->stage_msg[stage] = CMSG_STOP;
                        mbar_arrive(bar);
                        if (blp.trace) atomicMin(blp.trace + 2, globaltimer_ns());
                    }
                    if (AFF) {
                        // each group of the affine map looks at its own stages only: one message for each
                        for (int g = 1; g < Cfg::kAffGroups; ++g) {
                            if (++stage == nst) {
                                stage = 0;
                                phase ^= 1;
                            }
                            if (!mbar_wait(smem_u32(&ctl->empty[stage]), phase ^ 1, abort_flag, kCWaitLimitNs)) break;
                            if (issuer) {
                                ctl->stage_msg[stage] = CMSG_STOP;
                                mbar_arrive(smem_u32(&ctl->full[stage]));
                            }
                        }
                    }
                    ok = false;
                    break;
                }
#ifdef GPX_CGEMM_TIMING
                prod_wait += clock64() - t_w0;
#endif
                if (kb >= t.main_kb) {
                    // Residual block: A = 64 channels of the residual rows of this tile; the W
                    // operand is the 64x64 identity that stays in shared memory, applied to the
                    // matching 64 accumulator columns, so the tensor core adds the residual.
                    const int rb = kb - t.main_kb;
                    if (issuer) {
                        ctl->stage_msg[stage] = CMSG_RES + rb;
                        mbar_arrive_expect_tx(bar, Cfg::kPlanes * Cfg::kABytes + ident_bytes);
                        tma_load_2d(dst, &p.r_hi, bar, w_row + rb * kCBK, row0);
                        if (TWO) tma_load_2d(dst + Cfg::kABytes, &p.r_lo, bar, w_row + rb * kCBK, row0);
                        if (ident_bytes) tma_load_2d(smem_base + ident_off, &p.ident, bar, 0, 0);
                    }
                    ++kb;
                } else {
                    const int n = t.main_kb - kb < KPS ? t.main_kb - kb : KPS;
                    if (issuer && ident_bytes) tma_load_2d(smem_base + ident_off, &p.ident, bar, 0, 0);
#pragma unroll
                    for (int j = 0; j < KPS; ++j) {
                        if (j > 0 && j >= n) break;
                        const uint32_t d = dst + j * Cfg::kKbBytes;
                        if (issuer) {
                            tma_load_2d(d, &p.a_hi, bar, cb * kCBK, a_row);
                            tma_load_2d(d + Cfg::kWOff, &p.w_hi, bar, w_tap + cb * kCBK, w_row);
                            if (TWO) {
                                tma_load_2d(d + Cfg::kABytes, &p.a_lo, bar, cb * kCBK, a_row);
                                tma_load_2d(d + Cfg::kWOff + Cfg::kWBytes, &p.w_lo, bar, w_tap + cb * kCBK, w_row);
                            }
                        }
                        if (++cb == p.cin_blocks) {
                            cb = 0;
                            w_tap += p.cin;
                            if (++tap < p.taps) a_row = row0 + p.tap_shift[tap];
                        }
                    }
                    if (issuer) {  // (the bytes may be announced after the loads: the arrival still holds the phase)
                        ctl->stage_msg[stage] = CMSG_DATA + n;
                        mbar_arrive_expect_tx(bar, n * Cfg::kKbBytes + ident_bytes);
                    }
                    kb += n;
                }
                __syncwarp();
                ident_bytes = 0;
                if (++stage == nst) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
#ifdef GPX_CGEMM_TIMING
        if (lane == 0) {
            TADD(0, prod_wait);
            TADD(1, clock64() - t_prod0);
        }
#endif
        if (lane == 0) *(volatile int *)&ctl->poll_done = 1;
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        // Warp-uniform like the producer, one elected lane issues the tensor-core instructions.
        constexpr uint32_t idesc_bf16 = make_idesc_bf16_f32(kCBM, BN), idesc_f16 = make_idesc_f16_f32(kCBM, BN);
        constexpr int kWide = TWO ? 2 * BN : BN;
        constexpr uint32_t idesc_wide = make_idesc_bf16_f32(kCBM, kWide);
        const uint32_t idesc = (!TWO && p.fmt == PF_F16) ? idesc_f16 : idesc_bf16;
        const uint32_t idesc64 = (!TWO && p.fmt == PF_F16) ? make_idesc_f16_f32(kCBM, 64) : make_idesc_bf16_f32(kCBM, 64);
        const uint64_t eye = make_smem_desc_sw128(smem_base + ident_off);
        const uint64_t ring = make_smem_desc_sw128(smem_base);
        const int res_kb = p.res_kb;
        int stage = 0;
        uint32_t phase = 0;
        int kb = first_k;
        TCK(t_mma0);
#ifdef GPX_CGEMM_TIMING
        long long mma_wait_full = 0, mma_wait_tmem = 0, mma_kb = 0;
#endif
        uint32_t seg = 0;
        for (int tile = blockIdx.x + first_iter * gridDim.x; tile < total_tiles; tile += gridDim.x, ++seg, kb = 0) {
            const int buf = (int)(seg & 1);
            const uint32_t acc0 = tmem_base + buf * kBufCols;
            const int num_kb = tile_at(tile).main_kb + res_kb;
            TCK(t_e0);
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->tmem_empty[buf]), (seg >> 1) & 1, abort_flag, kCWaitLimitNs))) {
                if (lane == 0) fail(202);
                break;
            }
#ifdef GPX_CGEMM_TIMING
            mma_wait_tmem += clock64() - t_e0;
#endif
            tc_fence_after_sync();
            int end = CEPI_COMPLETE;
            while (kb < num_kb) {
                TCK(t_f0);
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->full[stage]), phase, abort_flag, kCWaitLimitNs))) {
                    if (lane == 0) fail(201);
                    end = -1;
                    break;
                }
#ifdef GPX_CGEMM_TIMING
                mma_wait_full += clock64() - t_f0;
                ++mma_kb;
#endif
                tc_fence_after_sync();
                const int msg = __shfl_sync(0xffffffffu, ctl->stage_msg[stage], 0);
                if (msg == CMSG_STOP) {
                    end = CEPI_PARTIAL;
                    break;
                }
                const int n = msg >= CMSG_RES ? 1 : msg - CMSG_DATA;  // K blocks in this stage
                if (AFF) {
                    if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->ready[stage]), phase, abort_flag, kCWaitLimitNs))) {
                        if (lane == 0) fail(203);
                        end = -1;
                        break;
                    }
                    tc_fence_after_sync();
                }
                // descriptor addresses are in 16-byte units
                const uint64_t a0 = ring + (uint64_t)(stage * (Cfg::kStageBytes >> 4));
                if (issuer) {
                    if (msg >= CMSG_RES) {
                        // residual x identity on 64 accumulator columns: the hi plane into the hi*hi
                        // accumulator, the lo plane into the cross-term accumulator (exact products,
                        // added like any other)
                        const uint32_t col = (uint32_t)(msg - CMSG_RES) * 64;
#pragma unroll
                        for (int k = 0; k < kCBK / kCUmmaK; ++k) {
                            mma_f16_ss(acc0 + col, a0 + 2 * k, eye + 2 * k, idesc64, 1u);
                            if (TWO) mma_f16_ss(acc0 + BN + col, a0 + (Cfg::kABytes >> 4) + 2 * k, eye + 2 * k, idesc64, 1u);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < KPS; ++j) {
                            if (j > 0 && j >= n) break;
                            const uint64_t a_hi = a0 + j * (Cfg::kKbBytes >> 4);
                            const uint64_t a_lo = a_hi + (Cfg::kABytes >> 4);
                            const uint64_t w_hi = a_hi + (Cfg::kWOff >> 4);
                            const uint32_t acc = (j > 0 || kb > 0) ? 1u : 0u;
                            if (TWO) {
                                // fp32 product from three bf16 products: hi*hi in one accumulator, both
                                // cross terms in the other.  The tensor core truncates when it adds into
                                // the fp32 accumulator, a bias that grows with the length of the
                                // accumulation chain; keeping the small cross terms apart keeps them
                                // clear of it.  The W_lo tile follows the W_hi tile in the stage and
                                // the two accumulators are adjacent columns, so A_hi x [W_hi; W_lo] is
                                // ONE instruction of width 2*BN, which reads the A_hi tile once.  The
                                // order is fixed, so a resumed tile replays exactly the instruction
                                // sequence of an uninterrupted one.
#pragma unroll
                                for (int k = 0; k < kCBK / kCUmmaK; ++k) {
                                    mma_f16_ss(acc0, a_hi + 2 * k, w_hi + 2 * k, idesc_wide, k > 0 ? 1u : acc);
                                    mma_f16_ss(acc0 + BN, a_lo + 2 * k, w_hi + 2 * k, idesc, 1u);
                                }
                            } else if constexpr (Cfg::kTmemA) {
                                const uint32_t a_cols = tmem_base + Cfg::kACols + 32 * stage;
#pragma unroll
                                for (int k = 0; k < kCBK / kCUmmaK; ++k)
                                    mma_f16_ts(acc0, a_cols + 8 * k, w_hi + 2 * k, idesc, k > 0 ? 1u : acc);
                            } else {
#pragma unroll
                                for (int k = 0; k < kCBK / kCUmmaK; ++k)
                                    mma_f16_ss(acc0, a_hi + 2 * k, w_hi + 2 * k, idesc, k > 0 ? 1u : acc);
                            }
                        }
                    }
                    mma_commit(smem_u32(&ctl->empty[stage]));
                }
                kb += n;
                __syncwarp();
                if (++stage == nst) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            if (end < 0) break;
            if (issuer) {
                ctl->epi_kind[buf] = end;
                ctl->epi_k_done[buf] = kb;
                mma_commit(smem_u32(&ctl->tmem_full[buf]));
                mbar_arrive(smem_u32(&ctl->tmem_full[buf]));
            }
            __syncwarp();
            if (end != CEPI_COMPLETE) {
                if (p.alternate) {
                    // the other group of epilogue warps waits for a tile that will not come
                    const int other = buf ^ 1;
                    if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->tmem_empty[other]), ((seg + 1) >> 1) & 1, abort_flag, kCWaitLimitNs))) {
                        if (lane == 0) fail(204);
                        break;
                    }
                    if (issuer) {
                        ctl->epi_kind[other] = CEPI_EXIT;
                        mma_commit(smem_u32(&ctl->tmem_full[other]));
                        mbar_arrive(smem_u32(&ctl->tmem_full[other]));
                    }
                    __syncwarp();
                }
                break;
            }
        }
#ifdef GPX_CGEMM_TIMING
        if (lane == 0) {
            TADD(2, mma_wait_full);
            TADD(3, mma_wait_tmem);
            TADD(4, clock64() - t_mma0);
            TADD(12, mma_kb);
        }
#endif
    } else if (warp == Cfg::kPollWarp) {
        // ------------------------------------------------------------------ preempt-word poller
        // A read of the word takes longer than a K block of a single-plane model: on the producer's
        // path, even one K block ahead, it set the pace of the ring.  Here one lane reads it back to
        // back and the producer looks at a flag in shared memory.  Ends with the producer.
        if (resumable && lane == 0) {
            while (!*(volatile int *)&ctl->poll_done) {
                if (load_word(blp.preempted) != 0) {
                    *(volatile int *)&ctl->word_up = 1;
                    break;
                }
                __nanosleep(100);
            }
        }
        __syncwarp();
    } else if (AFF && warp > Cfg::kPollWarp) {
        // ------------------------------------------------------------------ affine map of A
        // Every thread keeps one of the eight 16-byte pieces of a row (piece c of row r lies at position
        // c XOR (r mod 8), the 128-byte swizzle) and takes eight rows 16 apart: its sixteen scales and
        // shifts are read once per K block, and eight neighbouring threads touch one whole row, so no
        // two of a quarter warp meet in a bank.  ~130 instructions a thread and K block; the normalised
        // copy of the input that a kernel of its own wrote and this one read back (DenseNet-201 b64
        // bf16: 40 % of the forward) is gone.  (One thread per row, re-reading the scales for every
        // piece, took ~1500 cycles a K block on four warps.)
        // One-plane operands go to tensor memory instead of back to shared memory, from where the products then
        // need not read them (32 KB less through its port a K block, of 96) and no fence between proxies is needed.
        // DenseNet-201 b64 bf16, conv1 layers of block 1 206 -> 195 us, block 2 182 -> 173, block 3 604 -> 592,
        // transitions 148 -> 141 (with three groups 192, 169, 567 and 138); a K block of block 3 still takes ~830 cycles.
        // Groups of four warps take the K blocks in turn: a block is a chain of latencies (shared-memory
        // reads, conversions, the fence to the tensor core's proxy or the stores to tensor memory) that the other groups'
        // overlap.  Three groups where one plane leaves the registers for them: DenseNet-201 b64 bf16 2 767 -> 2 750 us,
        // with the maxima taken packed; latency-critical launches have too few blocks, two planes too few stages.
        constexpr int kGroupThreads = kCAffGroup;
        const int group = (warp - Cfg::kPollWarp - 1) / (kGroupThreads / 32);
        const int at = ((int)threadIdx.x - (Cfg::kPollWarp + 1) * 32) % kGroupThreads;
        const int piece = at & 7, row = at >> 3;
        constexpr int kAffRows = kCBM * 8 / kGroupThreads;  // rows per thread
        const uint32_t off = (uint32_t)(row * 128 + ((piece ^ (row & 7)) << 4));  // (rows 16 apart: same swizzle)
        const bool half_fmt = !TWO && p.fmt == PF_F16;
        auto map_block = [&](unsigned char *a, int ch, auto half) {
            const float4 *sc = reinterpret_cast<const float4 *>(aff_s + ch);
            const float4 *sh = reinterpret_cast<const float4 *>(aff_s + kCAffMaxC + ch);
            const float4 s0 = sc[0], s1 = sc[1], b0 = sh[0], b1 = sh[1];
            const float2 ss[4] = {{s0.x, s0.y}, {s0.z, s0.w}, {s1.x, s1.y}, {s1.z, s1.w}};
            const float2 bb[4] = {{b0.x, b0.y}, {b0.z, b0.w}, {b1.x, b1.y}, {b1.z, b1.w}};
            uint4 hv[kAffRows], lv[TWO ? kAffRows : 1];
#pragma unroll
            for (int r = 0; r < kAffRows; ++r) {
                hv[r] = *reinterpret_cast<const uint4 *>(a + r * 2048);
                if (TWO) lv[TWO ? r : 0] = *reinterpret_cast<const uint4 *>(a + Cfg::kABytes + r * 2048);
            }
#pragma unroll
            for (int r = 0; r < kAffRows; ++r) {
                uint32_t h[4] = {hv[r].x, hv[r].y, hv[r].z, hv[r].w}, l[4];
                if (TWO) {
                    const uint4 q = lv[TWO ? r : 0];
                    l[0] = q.x, l[1] = q.y, l[2] = q.z, l[3] = q.w;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float2 x = half ? pf_unpack2(h[q], PF_F16) : make_float2(bf16_lo_to_f32(h[q]), bf16_hi_to_f32(h[q]));
                    if (TWO) x = make_float2(x.x + bf16_lo_to_f32(l[q]), x.y + bf16_hi_to_f32(l[q]));
                    x = fma2(x, ss[q], bb[q]);
                    x = make_float2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f));
                    h[q] = half ? pf_pack2(x.x, x.y, PF_F16) : pack_bf16(x.x, x.y);
                    if (TWO) l[q] = pack_bf16(x.x - bf16_lo_to_f32(h[q]), x.y - bf16_hi_to_f32(h[q]));
                }
                *reinterpret_cast<uint4 *>(a + r * 2048) = make_uint4(h[0], h[1], h[2], h[3]);
                if (TWO) *reinterpret_cast<uint4 *>(a + Cfg::kABytes + r * 2048) = make_uint4(l[0], l[1], l[2], l[3]);
            }
        };
        // Into tensor memory: a thread takes, of rows r8 + 8 i of its warp's 32, four channels of each sixteen.  Odd rows take
        // the four sixteens in another order, so that sixteen lanes meet in no bank.
        const int r8 = lane >> 2, quad = lane & 3, turned = (r8 & 1) << 1;
        auto map_to_tmem = [&](const unsigned char *a, uint32_t cols, int ch, auto half) {
            constexpr int FMT = decltype(half)::value ? PF_F16 : PF_BF16;
            float2 ss[4][2], bb[4][2];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int c = ch + 16 * (b ^ turned) + 4 * quad;
                const float4 s4 = *reinterpret_cast<const float4 *>(aff_s + c), o4 = *reinterpret_cast<const float4 *>(aff_s + kCAffMaxC + c);
                ss[b][0] = make_float2(s4.x, s4.y), ss[b][1] = make_float2(s4.z, s4.w);
                bb[b][0] = make_float2(o4.x, o4.y), bb[b][1] = make_float2(o4.z, o4.w);
            }
            const unsigned char *mine = a + ((warp & 3) * 32 + r8) * 128 + (quad & 1) * 8;
            uint2 v[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    v[i][b] = *reinterpret_cast<const uint2 *>(mine + i * 1024 + (((2 * (b ^ turned) + (quad >> 1)) ^ r8) << 4));
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                uint32_t m[4][2][2], o[16];
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const uint32_t two = k ? v[2 * hh + i][b].y : v[2 * hh + i][b].x;
                            float2 x = half ? pf_unpack2(two, PF_F16) : make_float2(bf16_lo_to_f32(two), bf16_hi_to_f32(two));
                            x = fma2(x, ss[b][k], bb[b][k]);
                            m[b][i][k] = max_packed(pf_pack2(x.x, x.y, FMT), 0u, FMT);
                        }
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int k = 0; k < 2; ++k) o[4 * b + 2 * i + k] = turned ? m[b ^ 2][i][k] : m[b][i][k];
                tmem_st_16x256x4(cols + ((uint32_t)(16 * hh) << 16), o);
            }
        };
        static_assert(Cfg::kKps == 1 || !AFF, "one K block per stage");
        int stage = 0, kb = first_k, turn = 0;
        uint32_t phase = 0;
        bool go = true;
        for (int tile = blockIdx.x + first_iter * gridDim.x; go && tile < total_tiles; tile += gridDim.x, kb = 0) {
            const TileAt t = tile_at(tile);
            for (; kb < t.main_kb; ++kb) {
                if (turn == group) {
                    // (a ring of three stages and two groups, or of eight and three: the round before may be another group's)
                    if (ring_rounds_skipped(nst, Cfg::kAffGroups) &&
                        !__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->ready[stage]), phase ^ 1, abort_flag, kCWaitLimitNs))) {
                        if (lane == 0) fail(502);
                        go = false;
                        break;
                    }
                    if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->full[stage]), phase, abort_flag, kCWaitLimitNs))) {
                        if (lane == 0) fail(501);
                        go = false;
                        break;
                    }
                    if (__any_sync(0xffffffffu, ctl->stage_msg[stage] == CMSG_STOP)) {
                        go = false;
                        break;
                    }
                    unsigned char *a = smem + stage * Cfg::kStageBytes;
                    const int ch = (t.kb_base + kb) * kCBK;
                    if constexpr (Cfg::kTmemA) {
                        tc_fence_after_sync();  // the products that read this stage's columns are behind its barriers
                        const uint32_t cols = tmem_base + Cfg::kACols + 32 * stage + ((uint32_t)((warp & 3) * 32) << 16);
                        if (half_fmt)
                            map_to_tmem(a, cols, ch, std::true_type());
                        else
                            map_to_tmem(a, cols, ch, std::false_type());
                        tmem_st_wait();
                        tc_fence_before_sync();
                    } else {
                        if (half_fmt)
                            map_block(a + off, ch + piece * 8, std::true_type());
                        else
                            map_block(a + off, ch + piece * 8, std::false_type());
                        fence_proxy_async();  // ordinary stores, read by the tensor core
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&ctl->ready[stage]));
                }
                turn = turn + 1 == Cfg::kAffGroups ? 0 : turn + 1;
                if (++stage == nst) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        __syncwarp();
    } else if constexpr (CL) {
        // ------------------------------------------------------------------ epilogue of a cluster reduction
        // Each of the k_splits CTAs finishes 128 / k_splits rows of the tile: every CTA stores the rows of its
        // partial sums, straight from its accumulators, into their owners' shared memory
        // ([split][column / 4][row of the share] of 16 bytes), counted on the owner's barrier, and the
        // owner adds the splits in order from zero, exactly as splitk_finish_kernel adds the workspace rows,
        // then bias, residual, activation, store.  What that needs besides the sums is at hand before.
        // (Staged and copied in bulk, the rows took 2 100 cycles to arrive and another 2 000 to 3 600 to
        // be finished by eight warps; through the workspace the release in front of the barrier alone took 2 800.
        // What travels between SMs moves at about 16 bytes a cycle, so the owner's own rows do not.)
        // Nobody leaves before its own rows are complete, and nothing else is ever stored to it.
        // With one split there is nothing to exchange: a thread takes its row's columns through bias, residual
        // and activation to memory, with everything but the sums at hand before the products end (the loop
        // of the general epilogue takes 2 400 cycles for a tile of two planes).
        const int row = (warp & 3) * 32 + lane;
        constexpr int kCols = BN / Cfg::kEpiParts;
        const int c_lo = ((warp - 2) >> 2) * kCols;
        const uint32_t t_acc = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        auto sums = [&](int c, float *f) {  // sixteen columns of this thread's row
            uint32_t u[16], w[16];
            __syncwarp();  // (lanes with rows and lanes without part behind the columns before)
            tmem_ld_32x16(t_acc + c, u);
            if (TWO) tmem_ld_32x16(t_acc + BN + c, w);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) f[j] = TWO ? __uint_as_float(u[j]) + __uint_as_float(w[j]) : __uint_as_float(u[j]);
        };
        if (threadIdx.x == 64)
            for (int b = 0; b < 2; ++b) mbar_arrive(smem_u32(&ctl->tmem_empty[b]));
        if (p.k_splits == 1) {
            const int vrow = first_tile.m_blk * kCBM + row, col0 = first_tile.n_blk * BN;
            bool live = vrow < p.m_rows;
            size_t out_at = (size_t)vrow * p.out.C + col0, res_at = (size_t)vrow * p.res.C + col0;
            if (!p.identity_rows) {
                const int img = p.in_hs * p.in_ws;
                const int n_img = fast_div(live ? vrow : 0, img, p.inv_img);
                const int r = (live ? vrow : 0) - n_img * img;
                const int hs = fast_div(r, p.in_ws, p.inv_in_ws);
                const int h = hs - p.in_off, w = r - hs * p.in_ws - p.in_off;
                live = live && h >= 0 && h < p.out.H && w >= 0 && w < p.out.W;
                out_at = p.out_f32 ? ((size_t)(n_img * p.out.H + h) * p.out.W + w) * p.cout_valid + col0
                                   : (size_t)layout_row(p.out, n_img, h, w) * p.out.C + col0;
                res_at = (size_t)layout_row(p.res, n_img, h, w) * p.res.C + col0;
            }
            constexpr int kPieces = kCols / 16;
            const int fmt = TWO ? (int)PF_SPLIT : p.fmt, col_lim = p.cout_valid - col0;
            float4 bias4[kPieces][4];
            uint32_t rh[kPieces][8], rl[kPieces][TWO ? 8 : 1];
            if (p.bias)  // (padded to whole column tiles)
#pragma unroll
                for (int q = 0; q < kPieces; ++q)
#pragma unroll
                    for (int j = 0; j < 4; ++j) bias4[q][j] = __ldg(reinterpret_cast<const float4 *>(p.bias + col0 + c_lo + 16 * q) + j);
            pdl_wait();  // the residual is the predecessor's business, everything above is not
            const bool use_res = live && p.res_hi && !p.out_f32;
            if (use_res)
#pragma unroll
                for (int q = 0; q < kPieces; ++q) {
                    if (c_lo + 16 * q >= col_lim) break;
                    ld_global_v8(p.res_hi + res_at + c_lo + 16 * q, rh[q]);
                    if (TWO) ld_global_v8(p.res_lo + res_at + c_lo + 16 * q, rl[q]);
                }
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->tmem_full[0]), 0, abort_flag, kCWaitLimitNs))) {
                if (lane == 0) fail(301);
            } else {
                tc_fence_after_sync();
#pragma unroll
                for (int q = 0; q < kPieces; ++q) {
                    const int c = c_lo + 16 * q;
                    float f[16];
                    sums(c, f);
                    if (p.bias)
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            f[4 * j] += bias4[q][j].x, f[4 * j + 1] += bias4[q][j].y, f[4 * j + 2] += bias4[q][j].z, f[4 * j + 3] += bias4[q][j].w;
                    if (use_res) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float2 r = pf_unpack2(rh[q][j], fmt);
                            f[2 * j] += r.x, f[2 * j + 1] += r.y;
                        }
                        if (TWO)
#pragma unroll
                            for (int j = 0; j < 8; ++j) f[2 * j] += bf16_lo_to_f32(rl[q][j]), f[2 * j + 1] += bf16_hi_to_f32(rl[q][j]);
                    }
                    apply_act_n(f, p.relu);
                    if (!live || c >= col_lim) continue;
                    if (p.out_f32) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c + j < col_lim) p.out_f32[out_at + c + j] = f[j];
                        continue;
                    }
                    uint32_t hi[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) hi[j] = pf_pack2(f[2 * j], f[2 * j + 1], fmt);
                    st_sector(p.out_hi + out_at + c, hi);
                    if (TWO) {
                        uint32_t lo[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) lo[j] = pack_bf16(f[2 * j] - bf16_lo_to_f32(hi[j]), f[2 * j + 1] - bf16_hi_to_f32(hi[j]));
                        st_sector(p.out_lo + out_at + c, lo);
                    }
                }
            }
        } else {
            const SplitKParams &fin = p.fin;
            const int splits = p.k_splits, share = kCBM / splits, lg_share = 31 - __clz(share);
            const int rank = (int)cluster_ctarank();
            const int row0 = first_tile.m_blk * kCBM;
            constexpr int kItems = kCBM / 2 * (BN / 4) / Cfg::kEpiThreads;  // four-channel items a thread finishes (two splits)
            bool live[kItems];
            int col[kItems];
            uint32_t land_at[kItems];
            size_t out_at[kItems], res_at[kItems];
            float4 bias4[kItems];
            uint2 r_hi[kItems], r_lo[kItems];
            const uint32_t land = smem_base + (uint32_t)(Cfg::kRing * Cfg::kStageBytes);
            const int img = fin.in_hs * fin.in_ws;
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                // eight rows by four pieces a warp: sixteen-byte reads without bank conflicts, whole sectors stored
                const int e = (int)threadIdx.x - 64 + i * Cfg::kEpiThreads;
                const int lr = (e & 7) | (((e >> 5) & ((share >> 3) - 1)) << 3), piece = ((e >> 3) & 3) | ((e >> (2 + lg_share)) << 2);
                const int vrow = row0 + rank * share + lr;
                col[i] = first_tile.n_blk * BN + piece * 4;
                land_at[i] = land + (uint32_t)(piece * share + lr) * 16;
                live[i] = piece < BN / 4 && vrow < fin.m_rows && col[i] < fin.cout_padded;
                if (live[i]) {
                    const int n_img = fast_div(vrow, img, p.inv_img);
                    const int r = vrow - n_img * img;
                    const int hs = fast_div(r, fin.in_ws, p.inv_in_ws);
                    const int h = hs - fin.in_off, w = r - hs * fin.in_ws - fin.in_off;
                    live[i] = h >= 0 && h < fin.out.H && w >= 0 && w < fin.out.W;
                    if (live[i]) {
                        if (fin.bias) bias4[i] = __ldg(reinterpret_cast<const float4 *>(fin.bias + col[i]));
                        if (fin.res_hi) res_at[i] = (size_t)layout_row(fin.res, n_img, h, w) * fin.res.C + col[i];
                        out_at[i] = fin.out_f32 ? ((size_t)(n_img * fin.out.H + h) * fin.out.W + w) * fin.cout_valid + col[i]
                                                : (size_t)layout_row(fin.out, n_img, h, w) * fin.out.C + col[i];
                    }
                }
            }
            __syncwarp();
            cluster_wait();  // every CTA of the cluster runs
            pdl_wait();      // the residual is the predecessor's business, everything above is not
            if (fin.res_hi)
#pragma unroll
                for (int i = 0; i < kItems; ++i)
                    if (live[i]) {
                        r_hi[i] = *reinterpret_cast<const uint2 *>(fin.res_hi + res_at[i]);
                        if (TWO) r_lo[i] = *reinterpret_cast<const uint2 *>(fin.res_lo + res_at[i]);
                    }
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->tmem_full[0]), 0, abort_flag, kCWaitLimitNs))) {
                if (lane == 0) fail(301);
            } else {
                tc_fence_after_sync();
                const int owner = row >> lg_share;
                const uint32_t bar = cluster_map_shared(smem_u32(&ctl->landed), (uint32_t)owner);
                const uint32_t mine = land + ((uint32_t)(rank * (BN / 4)) * share + (row & (share - 1))) * 16;
                const uint32_t to = cluster_map_shared(mine, (uint32_t)owner);
#pragma unroll
                for (int c = c_lo; c < c_lo + kCols; c += 16) {
                    float f[16];
                    sums(c, f);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t at = (uint32_t)((c / 4 + j) * share) * 16;
                        if (owner == rank)
                            sts_f4(mine + at, f + 4 * j);
                        else if (row0 + row < p.m_rows)
                            st_async_v4(to + at, f + 4 * j, bar);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl->landed));
            volatile int never = 0;  // (a CTA that failed waits here as well, so that no store finds its memory gone)
            // (at cluster scope: the stores that complete it are other CTAs')
            if (!mbar_wait_cluster(smem_u32(&ctl->landed), 0, &never, kCWaitLimitNs + kCWaitLimitNs / 2)) fail(601);
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                if (!live[i]) continue;
                float f[4] = {0.f, 0.f, 0.f, 0.f};
                const uint32_t stride = (uint32_t)(share * (BN / 4)) * 16;
                for (int sp = 0; sp < splits; sp += 2) {
                    const float4 a = lds_f4(land_at[i] + sp * stride), b = lds_f4(land_at[i] + (sp + 1) * stride);
                    f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
                    f[0] += b.x; f[1] += b.y; f[2] += b.z; f[3] += b.w;
                }
                if (fin.bias) f[0] += bias4[i].x, f[1] += bias4[i].y, f[2] += bias4[i].z, f[3] += bias4[i].w;
                if (fin.res_hi) {
                    float2 r0 = pf_unpack2(r_hi[i].x, TWO ? (int)PF_SPLIT : fin.res.fmt), r1 = pf_unpack2(r_hi[i].y, TWO ? (int)PF_SPLIT : fin.res.fmt);
                    if (TWO) {
                        r0.x += bf16_lo_to_f32(r_lo[i].x), r0.y += bf16_hi_to_f32(r_lo[i].x);
                        r1.x += bf16_lo_to_f32(r_lo[i].y), r1.y += bf16_hi_to_f32(r_lo[i].y);
                    }
                    f[0] += r0.x, f[1] += r0.y, f[2] += r1.x, f[3] += r1.y;
                }
                apply_act_n(f, fin.relu);
                if (fin.out_f32) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (col[i] + j < fin.cout_valid) fin.out_f32[out_at[i] + j] = f[j];
                } else {
                    const int fmt = TWO ? (int)PF_SPLIT : fin.out.fmt;
                    const uint32_t h0 = pf_pack2(f[0], f[1], fmt), h1 = pf_pack2(f[2], f[3], fmt);
                    *reinterpret_cast<uint2 *>(fin.out_hi + out_at[i]) = make_uint2(h0, h1);
                    if (TWO)
                        *reinterpret_cast<uint2 *>(fin.out_lo + out_at[i]) =
                            make_uint2(pack_bf16(f[0] - bf16_lo_to_f32(h0), f[1] - bf16_hi_to_f32(h0)),
                                       pack_bf16(f[2] - bf16_lo_to_f32(h1), f[3] - bf16_hi_to_f32(h1)));
                }
            }
        }
        if (threadIdx.x == 64 && blp.trace && !*abort_flag) atomicAdd(blp.trace + 3, 1ull);
    } else {
        // ------------------------------------------------------------------ epilogue
        const int quarter = warp & 3;
        // Either all warps drain every tile, each its share of the columns, or (p.alternate) two groups take
        // the tiles, and with them the accumulator buffers, in turn: draining a tile is a chain of
        // ~2 800 cycles (wait, tensor memory, conversion, store, hand-over) however few columns a warp has,
        // and a layer of one or two K blocks waits for it (VGG-16's first, 16 images fp16: 70 -> 54 us).
        const int groups = p.alternate ? 2 : 1;
        const int parts = Cfg::kEpiParts / groups;        // warps of a group per lane quarter
        const int share = (warp - 2) >> 2, group = share / parts, part = share - group * parts;
        const int group_threads = 128 * parts;
        const int c_lo = part * (BN / parts), c_hi = c_lo + BN / parts;
        auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(group_threads) : "memory"); };
        // this warp's columns of one accumulator buffer when it restores (all warps) or spills (its group)
        constexpr int kRestoreCols = kBufCols / Cfg::kEpiParts;
        const int spill_cols = kBufCols / parts;
        const int row = quarter * 32 + lane;
        const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const bool leader = (int)threadIdx.x == 64 + group * group_threads;
        uint32_t v[32];
        if (first_k > 0) {
            for (int c = share * kRestoreCols; c < (share + 1) * kRestoreCols; c += 32) {
                // Spill layout: private to this kernel, so it is chosen for the stores: the j-th
                // 16-byte piece of a 32-column chunk of all 128 rows is contiguous, one warp store
                // writes 512 consecutive bytes (row-major rows 2 KB apart cost a line per thread).
                const uint4 *src = reinterpret_cast<const uint4 *>(spill) + (size_t)(c / 32) * 8 * kCBM + row;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    uint4 q = src[j * kCBM];
                    v[4 * j + 0] = q.x;
                    v[4 * j + 1] = q.y;
                    v[4 * j + 2] = q.z;
                    v[4 * j + 3] = q.w;
                }
                tmem_st_32x32(t_lane + c, v);
            }
            tmem_st_wait();
        }
        tc_fence_before_sync();
        asm volatile("bar.sync 3, %0;" ::"n"(Cfg::kEpiThreads) : "memory");
        if (threadIdx.x == 64)
            for (int b = 0; b < 2; ++b) mbar_arrive(smem_u32(&ctl->tmem_empty[b]));
        int it = first_iter + group;
        int seg_k0 = group == 0 ? first_k : 0;
        int tiles_done = 0;
        const int img = p.in_hs * p.in_ws;
        // Fields the drain loop needs, in registers: the loop is full of asm statements that clobber
        // memory, after each of which they would be read from the parameter block again.
        const float *const bias = p.partial ? nullptr : p.bias;
        const int relu = p.relu, fmt = p.fmt;
        float *const partial = p.partial;
        float *const out_f32 = p.out_f32;
        bf16_bits *const out_hi = p.out_hi, *const out_lo = p.out_lo;
        const bf16_bits *const res_hi = p.res_hi, *const res_lo = p.res_lo;
        float bias_next = 0.f;  // this thread's bias element of the next tile to drain
        if (bias) {
            const int t = (int)threadIdx.x - 64 - group * group_threads;
            const int first = blockIdx.x + it * gridDim.x;
            if (t < BN && first < total_tiles) bias_next = __ldg(bias + tile_at(first).n_blk * BN + t);
        }
        TCK(t_epi0);
#ifdef GPX_CGEMM_TIMING
        long long e_wait = 0, e_tmem = 0, e_math = 0, e_store = 0, e_bar = 0;
#endif
        for (uint32_t seg = group;; seg += groups) {
            const int tile = blockIdx.x + it * gridDim.x;
            if (tile >= total_tiles) {
                // (of two groups, the one that had the last tile: the other's end says nothing about that tile)
                if (leader && resumable && (groups == 1 || tile - (int)gridDim.x >= total_tiles)) {
                    slot->next_iter = it;
                    slot->k_done = 0;
                    slot->grid = gridDim.x;
                }
                break;
            }
            const int buf = (int)(seg & 1);
            const uint32_t t_acc = t_lane + buf * kBufCols;
            TCK(t_wait0);
            const TileAt at = tile_at(tile);
            const int n_blk = at.n_blk;
            // The bias of the tile this buffer holds goes to shared memory before the drain loop
            // (read from global memory inside it, its latency - an L2 round trip under load - was
            // paid once per 16-column piece).  The value stored now was requested one tile ago
            // and the request for the tile after this one is issued here, so the round trip
            // overlaps the drain of this tile instead of delaying its start.
            if (bias) {
                const int t = (int)threadIdx.x - 64 - group * group_threads;
                if (t < BN) {
                    ctl->bias_s[buf][t] = bias_next;
                    const int after = tile + groups * gridDim.x;
                    if (after < total_tiles) bias_next = __ldg(bias + tile_at(after).n_blk * BN + t);
                }
            }
            // Which output pixel, if any, does this GEMM row stand for?  (Before the wait: the answer
            // does not depend on the products.)
            const int vrow = at.m_blk * kCBM + row;
            bool valid = vrow < p.m_rows;
            size_t out_off = 0, res_off = 0;
            if (p.identity_rows) {
                // plain rows in, plain rows out (and a plain residual): row m of the GEMM is
                // row m of the output, no pixel arithmetic is needed
                if (valid) {
                    out_off = (size_t)vrow * p.out.C + (size_t)n_blk * BN;
                    if (res_hi) res_off = (size_t)vrow * p.res.C + (size_t)n_blk * BN;
                }
            } else {
                int n_img = 0, h = 0, w = 0;
                if (valid) {
                    n_img = fast_div(vrow, img, p.inv_img);
                    int r = vrow - n_img * img;
                    int hs = fast_div(r, p.in_ws, p.inv_in_ws);
                    int ws = r - hs * p.in_ws;
                    h = hs - p.in_off;
                    w = ws - p.in_off;
                    valid = h >= 0 && h < p.out.H && w >= 0 && w < p.out.W;
                }
                if (valid) {
                    out_off = out_f32 ? ((size_t)(n_img * p.out.H + h) * p.out.W + w) * p.cout_valid
                                      : (size_t)layout_row(p.out, n_img, h, w) * p.out.C + (size_t)n_blk * BN;
                    if (res_hi) res_off = (size_t)layout_row(p.res, n_img, h, w) * p.res.C + (size_t)n_blk * BN;
                }
            }
            float *const part_row = partial ? partial + ((size_t)at.split * p.partial_rows + vrow) * p.partial_ld + n_blk * BN : nullptr;
            const bool part_valid = vrow < p.m_rows;
            const int col_lim = p.cout_valid - n_blk * BN;
            if (leader) {
                bool ok = mbar_wait(smem_u32(&ctl->tmem_full[buf]), (seg >> 1) & 1, abort_flag, kCWaitLimitNs);
                if (!ok) fail(301);
                ctl->epi_go[group] = ok ? 1 : 0;
            }
            group_sync();
#ifdef GPX_CGEMM_TIMING
            e_wait += clock64() - t_wait0;
#endif
#ifdef GPX_CGEMM_TIMING
            if (leader && seg == 0) TADD(17, clock64() - t_begin);
#endif
            if (!ctl->epi_go[group]) break;
            tc_fence_after_sync();
            const int kind = ctl->epi_kind[buf];
            const int k_done = ctl->epi_k_done[buf];
            if (kind == CEPI_EXIT) break;
            if (kind == CEPI_COMPLETE) {
                // Every lane owns one row of the tile (its TMEM lane): 16 columns of a plane are 32
                // contiguous bytes of that row, one 256-bit access, a whole sector.
                const bool use_res = !partial && !out_f32 && res_hi && valid;
                constexpr int CH = (TWO || AFF || BN == 256) ? 16 : 32;  // columns per piece
                // (columns past the real output, a quarter to a half of a tile for a DenseNet layer, are left out;
                // partial sums go out whole)
                const int c_end = partial || c_hi < col_lim ? c_hi : col_lim;
#pragma unroll 1
                for (int c = c_lo; c < c_end; c += CH) {
                    float f[CH];
                    // The residual is requested first so its latency overlaps the TMEM reads.
                    TCK(t_p0);
                    uint32_t rh[CH / 2], rl[TWO ? CH / 2 : 1];
                    if (use_res) {
#pragma unroll
                        for (int q = 0; q < CH / 16; ++q) ld_global_v8(res_hi + res_off + c + 16 * q, rh + 8 * q);
                        if (TWO) ld_global_v8(res_lo + res_off + c, rl);
                    }
                    __syncwarp();  // (lanes with rows and lanes without part behind the piece before)
                    if constexpr (TWO) {
                        uint32_t t16[16], u16[16];
                        tmem_ld_32x16(t_acc + c, t16);
                        tmem_ld_32x16(t_acc + BN + c, u16);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(t16[j]) + __uint_as_float(u16[j]);
                    } else {
                        uint32_t t32[CH];
                        if constexpr (CH == 32)
                            tmem_ld_32x32(t_acc + c, t32);
                        else
                            tmem_ld_32x16(t_acc + c, t32);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < CH; ++j) f[j] = __uint_as_float(t32[j]);
                    }
#ifdef GPX_CGEMM_TIMING
                    long long t_p1 = clock64();
                    e_tmem += t_p1 - t_p0;
#endif
                    if (partial) {
                        // Split K: the raw fp32 sum of this K range goes to the workspace; the
                        // finishing kernel adds the ranges in split order and applies the rest.
                        if (part_valid) {
                            float4 *dst = reinterpret_cast<float4 *>(part_row + c);
#pragma unroll
                            for (int j = 0; j < CH / 4; ++j)
                                dst[j] = make_float4(f[4 * j], f[4 * j + 1], f[4 * j + 2], f[4 * j + 3]);
                        }
                        continue;
                    }
                    if (bias) {
                        const float4 *b4 = reinterpret_cast<const float4 *>(&ctl->bias_s[buf][c]);
#pragma unroll
                        for (int j = 0; j < CH / 4; ++j) {
                            float4 b = b4[j];
                            f[4 * j + 0] += b.x;
                            f[4 * j + 1] += b.y;
                            f[4 * j + 2] += b.z;
                            f[4 * j + 3] += b.w;
                        }
                    }
                    if (use_res) {
#pragma unroll
                        for (int q = 0; q < CH / 2; ++q) {
                            float2 r = pf_unpack2(rh[q], TWO ? (int)PF_SPLIT : fmt);
                            f[2 * q] += r.x;
                            f[2 * q + 1] += r.y;
                        }
                        if constexpr (TWO) {
#pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                f[2 * q] += bf16_lo_to_f32(rl[q]);
                                f[2 * q + 1] += bf16_hi_to_f32(rl[q]);
                            }
                        }
                    }
                    apply_act_n(f, relu);
                    if (out_f32) {
                        const int col0 = n_blk * BN + c;
                        if (valid) {
#pragma unroll
                            for (int j = 0; j < CH; ++j)
                                if (c + j < col_lim) out_f32[out_off + col0 + j] = f[j];
                        }
                        continue;
                    }
                    uint32_t hi[CH / 2];
                    if (TWO || fmt != PF_F16) {
#pragma unroll
                        for (int q = 0; q < CH / 2; ++q) hi[q] = pack_bf16(f[2 * q], f[2 * q + 1]);
                    } else {
#pragma unroll
                        for (int q = 0; q < CH / 2; ++q) hi[q] = pf_pack2(f[2 * q], f[2 * q + 1], PF_F16);
                    }
#ifdef GPX_CGEMM_TIMING
                    long long t_p2 = clock64();
                    e_math += t_p2 - t_p1;
#endif
                    // The output may be a channel slice: nothing is stored past cout_valid.
#pragma unroll
                    for (int q = 0; q < CH / 16; ++q)
                        if (valid && c + 16 * q < col_lim) st_sector(out_hi + out_off + c + 16 * q, hi + 8 * q);
                    if constexpr (TWO) {
                        uint32_t lo[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            lo[q] = pack_bf16(f[2 * q] - bf16_lo_to_f32(hi[q]), f[2 * q + 1] - bf16_hi_to_f32(hi[q]));
                        if (valid && c < col_lim) st_sector(out_lo + out_off + c, lo);
                    }
#ifdef GPX_CGEMM_TIMING
                    e_store += clock64() - t_p2;
#endif
                }
                it += groups;
                ++tiles_done;
                seg_k0 = 0;
                tc_fence_before_sync();
                TCK(t_b0);
                group_sync();
#ifdef GPX_CGEMM_TIMING
                e_bar += clock64() - t_b0;
#endif
                if (leader) {
                    mbar_arrive(smem_u32(&ctl->tmem_empty[buf]));
                    if (blp.executed) atomicAdd(blp.executed, 1);
                }
                continue;
            }
            // CEPI_PARTIAL
            const int keep_k = p.drop_on_stop ? 0 : k_done;
            if (keep_k > seg_k0) {
                for (int c = part * spill_cols; c < (part + 1) * spill_cols; c += 32) {
                    tmem_ld_32x32(t_acc + c, v);
                    tmem_ld_wait();
                    uint4 *dst = reinterpret_cast<uint4 *>(spill) + (size_t)(c / 32) * 8 * kCBM + row;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        dst[j * kCBM] = make_uint4(v[4 * j + 0], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
            }
            if (leader) {
                slot->next_iter = it;
                slot->k_done = keep_k;
                slot->grid = gridDim.x;
                if (blp.stop_index) atomicCAS(blp.stop_index, -1, blp.kernel_id);
            }
            break;
        }
        if (leader && blp.trace && tiles_done) atomicAdd(blp.trace + 3, (unsigned long long)tiles_done);
#ifdef GPX_CGEMM_TIMING
        if (lane == 0) {
            TADD(5, e_wait);
            TADD(6, e_tmem);
            TADD(7, e_math);
            TADD(8, e_store);
            TADD(9, e_bar);
            TADD(10, clock64() - t_epi0);
        }
        if (leader) TADD(11, tiles_done);
#endif
    }

    tc_fence_before_sync();
    __syncwarp();
    if (CL && (warp < 2 || warp >= Cfg::kPollWarp)) cluster_wait();
    __syncthreads();
    if (warp == 0 && lane == 0 && *abort_flag) {
        for (int spin = 0; spin < 64; ++spin) __nanosleep(1000);
    }
    if (warp == 1) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
    if (threadIdx.x == 0 && blp.trace) atomicMax(blp.trace + 1, globaltimer_ns());
#ifdef GPX_CGEMM_TIMING
    if (threadIdx.x == 0) {
        TADD(13, clock64() - t_start);
        TADD(15, 1);
    }
#endif
}

#ifdef GPX_CGEMM_TIMING
// Development build only: copies the phase timers to the host and optionally clears them.
extern "C" int gpx_debug_cgemm_timing(unsigned long long *out, int reset) {
    if (cudaMemcpyFromSymbol(out, g_cgemm_timing, sizeof(unsigned long long) * 32) != cudaSuccess) return 1;
    if (reset) {
        static unsigned long long zeros[32] = {0};
        if (cudaMemcpyToSymbol(g_cgemm_timing, zeros, sizeof(zeros)) != cudaSuccess) return 1;
    }
    return 0;
}
#endif

// Calls f with the kernel instance of a tile width, operand format, A treatment and reduction (as a struct of
// constants).  256-column tiles exist for single-plane operands used as they are: two planes' two
// accumulators in two buffers would not fit tensor memory, and no layer behind an affine map is wide.
template <int BN, bool TWO, bool AFF, bool CL>
struct CgemmInstance {
    using Cfg = CgemmCfg<BN, TWO, AFF, CL>;
    static constexpr auto kernel() { return cgemm_tcgen05_kernel<BN, TWO, AFF, CL>; }
};
template <typename F>
static auto cgemm_instance(int bn, bool two, bool aff, bool cluster, F &&f) {
    if (cluster) {
        if (two) return aff ? f(CgemmInstance<64, true, true, true>()) : f(CgemmInstance<64, true, false, true>());
        return aff ? f(CgemmInstance<64, false, true, true>()) : f(CgemmInstance<64, false, false, true>());
    }
    if (two && aff) return bn == 128 ? f(CgemmInstance<128, true, true, false>()) : f(CgemmInstance<64, true, true, false>());
    if (two) return bn == 128 ? f(CgemmInstance<128, true, false, false>()) : f(CgemmInstance<64, true, false, false>());
    if (aff) return bn == 128 ? f(CgemmInstance<128, false, true, false>()) : f(CgemmInstance<64, false, true, false>());
    if (bn == 256) return f(CgemmInstance<256, false, false, false>());
    return bn == 128 ? f(CgemmInstance<128, false, false, false>()) : f(CgemmInstance<64, false, false, false>());
}

cudaError_t cgemm_prepare(int device) {
    static bool done[64] = {false};
    if (device < 0 || device >= 64 || done[device]) return cudaSuccess;
    auto allow = [](auto k) {
        return cudaFuncSetAttribute(k.kernel(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)decltype(k)::Cfg::kSmem);
    };
    for (int two = 0; two < 2; ++two)
        for (int aff = 0; aff < 2; ++aff) {
            for (int bn : {64, 128, 256}) {
                if (bn == 256 && (two || aff)) continue;
                cudaError_t e = cgemm_instance(bn, two != 0, aff != 0, false, allow);
                if (e != cudaSuccess) return e;
            }
            cudaError_t e = cgemm_instance(64, two != 0, aff != 0, true, allow);
            if (e != cudaSuccess) return e;
        }
    done[device] = true;
    return cudaSuccess;
}

// CTAs of clusters of `cluster` CTAs of the reducing kernel that the device keeps resident at once.
int cgemm_max_cluster(int fmt, bool aff, int cluster) {
    int clusters = 0;
    cudaError_t err = cgemm_instance(64, fmt == PF_SPLIT, aff, true, [&](auto k) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)cluster);
        cfg.blockDim = dim3((unsigned)decltype(k)::Cfg::kThreads);
        cfg.dynamicSmemBytes = decltype(k)::Cfg::kSmem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)cluster;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return cudaOccupancyMaxActiveClusters(&clusters, k.kernel(), &cfg);
    });
    if (err != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return clusters * cluster;
}

cudaError_t cgemm_launch(const CgemmParams &p, int bn, int grid, const BlpArgs &blp, cudaStream_t s) {
    if (p.narrow) return conv3x3_narrow_launch(p, grid, blp, s);
    return cgemm_instance(bn, p.fmt == PF_SPLIT, p.aff_scale != nullptr, p.cluster_reduce != 0, [&](auto k) {
        void *args[] = {const_cast<CgemmParams *>(&p), const_cast<BlpArgs *>(&blp)};
        return launch_direct(reinterpret_cast<const void *>(k.kernel()), (unsigned)grid, (unsigned)decltype(k)::Cfg::kThreads,
                             decltype(k)::Cfg::kSmem, s, p.cluster_reduce ? (unsigned)p.k_splits : 1u, args);
    });
}

int cgemm_threads(int bn, int fmt, bool aff) {
    return cgemm_instance(bn, fmt == PF_SPLIT, aff, false, [](auto k) { return decltype(k)::Cfg::kThreads; });
}

}  // namespace gpx
