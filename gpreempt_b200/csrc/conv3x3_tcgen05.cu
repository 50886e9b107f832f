// 3x3 stride-1 convolution with few output channels (32 or 64) on the tcgen05 tensor cores, for the
// single-plane (bf16 / fp16) models: DenseNet's growth layers, the 64-channel layers of VGG and ResNet.
//
// The general kernel (cgemm_tcgen05.cu) fetches the 128 rows of a tile once for each of the nine taps and
// multiplies them by a 64-column tile that is padding from column 32 on for a growth layer; what bounds it is
// the fill of shared memory (24 KB a K block, ~72 bytes a cycle and SM) and the ~110 cycles an instruction of 64 columns
// takes there.  Here all weights (72 KB) stay in shared memory and the rows are fetched three times, once for a filter row.
//
// 32 channels: the three taps of a filter row are columns of one operand.  For filter row dy
//     acc[r][dx][co] += A[r + (dy - 1) * Ws][:] . W[dy][dx][co][:]
// is one product of 96 columns, and the output is
//     out[m][co] = acc[m - 1][0][co] + acc[m][1][co] + acc[m + 1][2][co],
// sums over neighbouring rows, which are neighbouring lanes of tensor memory: shuffles, and shared memory where
// a warp's 32 lanes end.  A tile of 128 rows yields 126 outputs.  Bound by its products (67 cycles each).  64 images bf16,
// 56x56, 128 channels in: 44 us in the general kernel, 21 like this.
//
// 64 channels: shuffling 128 values a row takes the epilogue 3 700 cycles a tile (VGG-16's 64 -> 64 at 224x224, 16 images:
// 97 us in the general kernel, 94 so).  Instead a strip of 136 rows is fetched for a filter row and its three taps
// read it from row 0, 1 and 2 on: a K-major operand may begin at any 128-byte row, as the swizzle goes by the
// address: 72 us, the same bits as the general kernel.
//
// Roles, messages and the preempt / spill / resume protocol are those of the general kernel, with a ring
// stage of twelve products (the three filter rows of 64 input channels, or one of them) as the unit at which a CTA
// stops, and two groups of four epilogue warps that take the tiles in turn.
#include "layers.cuh"
#include "sm100.cuh"

#include <cuda_bf16.h>

namespace gpx {

using namespace sm100;

namespace {

constexpr int kNM = 128, kNK = 64;
constexpr int kNEpiThreads = 256;         // two groups of four warps
constexpr int kNPollWarp = 2 + kNEpiThreads / 32;
constexpr int kNThreads = 64 + kNEpiThreads + 32;
constexpr int kNStagesMax = 8;
constexpr uint32_t kNWBytes = 72 * 1024;           // 3 cin_blocks tiles of 3 CO rows: 9 x 64 x 128 x 32 or 9 x 64 x 64
constexpr unsigned long long kNWaitLimitNs = 2000000000ull;

enum : int { NMSG_DATA = 0, NMSG_STOP = 1 };
enum : int { NEPI_COMPLETE = 0, NEPI_PARTIAL = 1, NEPI_EXIT = 2 };

struct NarrowControl {
    unsigned long long full[kNStagesMax], empty[kNStagesMax];
    unsigned long long weights;
    unsigned long long tmem_full[2], tmem_empty[2];
    uint32_t tmem_base;
    int stage_msg[kNStagesMax];
    int epi_kind[2], epi_k_done[2], epi_go[2];
    int raised, word_up, poll_done, abort_flag;
    alignas(16) float bias[64];
    alignas(16) float edge[2][4][2][32];  // [group][warp][its last row, left tap / first row, right tap]
};

template <int CO>
struct NarrowCfg {
    static constexpr bool kFold = CO == 32;           // taps of a filter row as columns, or a strip they share
    static constexpr int kN = kFold ? 3 * CO : CO;    // columns of a product
    static constexpr int kOut = kFold ? kNM - 2 : kNM;  // output rows of a tile
    static constexpr int kARows = kFold ? kNM : kNM + 8;
    static constexpr uint32_t kABytes = kARows * kNK * 2;
    static constexpr int kATiles = kFold ? 3 : 1;     // filter rows in a ring stage
    static constexpr uint32_t kStageBytes = kATiles * kABytes;
    static constexpr int kStages = kFold ? 3 : 8;
    static constexpr uint32_t kWTap = CO * kNK * 2, kWTile = 3 * kWTap;  // weights of one tap and 64 input channels, of a filter row
    static constexpr int kBufCols = kFold ? 128 : 64, kTmemCols = 2 * kBufCols;
    static constexpr size_t kSmem = 1024 + kNWBytes + kStages * kStageBytes + sizeof(NarrowControl);
    static_assert(kSmem <= 227 * 1024 && kStages <= kNStagesMax && kABytes % 1024 == 0, "tile does not fit");
};

template <int CO>
__global__ void __launch_bounds__(kNThreads, 1)
conv3x3_narrow_kernel(const __grid_constant__ CgemmParams p, BlpArgs blp) {
    using Cfg = NarrowCfg<CO>;
    constexpr bool kFold = Cfg::kFold;
    constexpr int N = Cfg::kN, kBufCols = Cfg::kBufCols, kTmemCols = Cfg::kTmemCols, kNStages = Cfg::kStages, kNOut = Cfg::kOut;
    constexpr uint32_t kNABytes = Cfg::kABytes, kNStageBytes = Cfg::kStageBytes, kWTile = Cfg::kWTile;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    unsigned char *smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    const uint32_t w_base = smem_u32(smem), ring = w_base + kNWBytes;
    NarrowControl *ctl = reinterpret_cast<NarrowControl *>(smem + kNWBytes + kNStages * kNStageBytes);
    volatile int *abort_flag = &ctl->abort_flag;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int total_tiles = p.tiles_m;
    const int stages = p.cin_blocks * 3 / Cfg::kATiles;  // of a tile
    const bool resumable = blp.preempted != nullptr;
    const bool issuer = elect_one();
    CgemmSlot *slot = p.slots + blockIdx.x;
    float *spill = p.spill + (size_t)blockIdx.x * kCgemmSpillFloats;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kNStages; ++s) {
            mbar_init(smem_u32(&ctl->full[s]), 1);
            mbar_init(smem_u32(&ctl->empty[s]), 1);
        }
        mbar_init(smem_u32(&ctl->weights), 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&ctl->tmem_full[b]), 2);
            mbar_init(smem_u32(&ctl->tmem_empty[b]), 1);
            ctl->epi_kind[b] = NEPI_COMPLETE;
            ctl->epi_k_done[b] = 0;
            ctl->epi_go[b] = 0;
        }
        ctl->raised = ctl->word_up = ctl->poll_done = ctl->abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
        prefetch_tensormap(&p.a_hi);
        prefetch_tensormap(&p.w_hi);
    }
    if (threadIdx.x >= 64 && threadIdx.x < 64 + CO) ctl->bias[threadIdx.x - 64] = p.bias ? __ldg(p.bias + threadIdx.x - 64) : 0.f;
    if (warp == 1) tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = ctl->tmem_base;
    // Weights are never written by a kernel: a non-preemptible launch fetches them under its predecessor's tail.
    auto fetch_weights = [&]() {
        if (issuer) {
            const uint32_t bar = smem_u32(&ctl->weights);
            const int blocks = 3 * p.cin_blocks;  // (64 input channels, filter row)
            mbar_arrive_expect_tx(bar, blocks * kWTile);
            for (int kb = 0; kb < blocks; ++kb)
                for (int dx = 0; dx < 3; ++dx)
                    tma_load_2d(w_base + kb * kWTile + dx * Cfg::kWTap, &p.w_hi, bar, ((kb % 3) * 3 + dx) * p.cin + kb / 3 * kNK, 0);
        }
        __syncwarp();
    };
    if (!resumable && warp == 0) fetch_weights();
    pdl_wait();
    pdl_launch_dependents();
    const int first_iter = resumable ? slot->next_iter : 0;
    const int first_k = resumable ? slot->k_done : 0;  // ring stages of the first tile that are accumulated already
    const int slot_grid = resumable ? slot->grid : 0;
    if (resumable) {
        // launched while the word is raised: leave at once, a stop point if there is work left
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
                tmem_dealloc(tmem_base, kTmemCols);
            }
            return;
        }
    }
    if (threadIdx.x == 0) trace_begin(blp);
    auto fail = [&](int code) {
        ctl->abort_flag = 1;
        if (atomicCAS(p.error, 0, code) == 0) p.error[1] = blp.kernel_id * 1000 + (int)blockIdx.x;
    };
    auto wait_all = [&](unsigned long long *bar, uint32_t phase, int code) {  // a whole warp
        if (__all_sync(0xffffffffu, mbar_wait(smem_u32(bar), phase, abort_flag, kNWaitLimitNs))) return true;
        if (lane == 0) fail(code);
        return false;
    };
    bool weights_asked = !resumable;

    if (slot_grid != 0 && slot_grid != (int)gridDim.x) {
        if (threadIdx.x == 0) fail(900);
    } else if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (!weights_asked) fetch_weights();
        weights_asked = true;
        int s = 0, k = first_k;
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x + first_iter * gridDim.x; ok && tile < total_tiles; tile += gridDim.x, k = 0) {
            const int row0 = tile * kNOut - 1 - p.in_ws;  // of filter row 0
            for (; k < stages; ++k) {
                const bool stop = resumable && __any_sync(0xffffffffu, *(volatile int *)&ctl->word_up);
                if (!wait_all(&ctl->empty[s], phase ^ 1, 1101)) {
                    ok = false;
                    break;
                }
                if (issuer) {
                    const uint32_t bar = smem_u32(&ctl->full[s]), dst = ring + s * kNStageBytes;
                    ctl->stage_msg[s] = stop ? NMSG_STOP : NMSG_DATA;
                    if (stop) {
                        mbar_arrive(bar);
                        if (blp.trace) atomicMin(blp.trace + 2, globaltimer_ns());
                    } else {
                        mbar_arrive_expect_tx(bar, kNStageBytes);
                        if (kFold) {
#pragma unroll
                            for (int dy = 0; dy < 3; ++dy) tma_load_2d(dst + dy * kNABytes, &p.a_hi, bar, k * kNK, row0 + dy * p.in_ws);
                        } else {
                            const int cb = k / 3;
                            tma_load_2d(dst, &p.a_hi, bar, cb * kNK, row0 + (k - 3 * cb) * p.in_ws);
                        }
                    }
                }
                __syncwarp();
                if (stop) {
                    ok = false;
                    break;
                }
                if (++s == kNStages) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
        if (lane == 0) *(volatile int *)&ctl->poll_done = 1;
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const uint32_t idesc = p.fmt == PF_F16 ? make_idesc_f16_f32(kNM, N) : make_idesc_bf16_f32(kNM, N);
        const uint64_t a_desc = make_smem_desc_sw128(ring), w_desc = make_smem_desc_sw128(w_base);
        int s = 0, k = first_k;
        uint32_t phase = 0, seg = 0;
        bool ok = wait_all(&ctl->weights, 0, 1205);
        for (int tile = blockIdx.x + first_iter * gridDim.x; ok && tile < total_tiles; tile += gridDim.x, ++seg, k = 0) {
            const int buf = (int)(seg & 1);
            const uint32_t acc = tmem_base + buf * kBufCols;
            if (!wait_all(&ctl->tmem_empty[buf], (seg >> 1) & 1, 1202)) break;
            tc_fence_after_sync();
            int end = NEPI_COMPLETE;
            for (; k < stages; ++k) {
                if (!wait_all(&ctl->full[s], phase, 1201)) {
                    end = -1;
                    break;
                }
                tc_fence_after_sync();
                if (__any_sync(0xffffffffu, ctl->stage_msg[s] == NMSG_STOP)) {
                    end = NEPI_PARTIAL;
                    break;
                }
                if (issuer) {
                    const uint64_t a = a_desc + (uint64_t)(s * (kNStageBytes >> 4)), w = w_desc + (uint64_t)(k * (Cfg::kATiles * kWTile >> 4));
                    // three filter rows, or three taps of one: the strip from row t on
                    constexpr uint64_t a_step = kFold ? kNABytes >> 4 : kNK * 2 >> 4, w_step = (kFold ? kWTile : Cfg::kWTap) >> 4;
#pragma unroll
                    for (int t = 0; t < 3; ++t)
#pragma unroll
                        for (int q = 0; q < kNK / 16; ++q)
                            mma_f16_ss(acc, a + t * a_step + 2 * q, w + t * w_step + 2 * q, idesc, (t > 0 || q > 0 || k > 0) ? 1u : 0u);
                    mma_commit(smem_u32(&ctl->empty[s]));
                }
                __syncwarp();
                if (++s == kNStages) {
                    s = 0;
                    phase ^= 1;
                }
            }
            if (end < 0) break;
            if (issuer) {
                ctl->epi_kind[buf] = end;
                ctl->epi_k_done[buf] = k;
                mma_commit(smem_u32(&ctl->tmem_full[buf]));
                mbar_arrive(smem_u32(&ctl->tmem_full[buf]));
            }
            __syncwarp();
            if (end != NEPI_COMPLETE) {
                // the other group of epilogue warps waits for a tile that will not come
                const int other = buf ^ 1;
                if (!wait_all(&ctl->tmem_empty[other], ((seg + 1) >> 1) & 1, 1204)) break;
                if (issuer) {
                    ctl->epi_kind[other] = NEPI_EXIT;
                    mma_commit(smem_u32(&ctl->tmem_full[other]));
                    mbar_arrive(smem_u32(&ctl->tmem_full[other]));
                }
                __syncwarp();
                break;
            }
        }
    } else if (warp == kNPollWarp) {
        // ------------------------------------------------------------------ preempt-word poller
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
    } else {
        // ------------------------------------------------------------------ epilogue
        const int group = (warp - 2) >> 2, quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const bool leader = (int)threadIdx.x == 64 + group * 128;
        auto group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
        if (first_k > 0 && group == 0) {
            // (spilled as the general kernel spills: the j-th 16-byte piece of a 32-column chunk of all rows is contiguous)
            uint32_t v[32];
            for (int c = 0; c < N; c += 32) {
                const uint4 *src = reinterpret_cast<const uint4 *>(spill) + (size_t)(c / 32) * 8 * kNM + row;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint4 q = src[j * kNM];
                    v[4 * j] = q.x, v[4 * j + 1] = q.y, v[4 * j + 2] = q.z, v[4 * j + 3] = q.w;
                }
                tmem_st_32x32(t_lane + c, v);
            }
            tmem_st_wait();
        }
        tc_fence_before_sync();
        group_sync();
        if (leader) mbar_arrive(smem_u32(&ctl->tmem_empty[group]));
        const int img = p.in_hs * p.in_ws;
        int it = first_iter + group, tiles_done = 0;
        for (uint32_t seg = group;; seg += 2, it += 2) {
            const int tile = blockIdx.x + it * gridDim.x;
            if (tile >= total_tiles) {
                // (the group that had the last tile says so)
                if (leader && resumable && tile - (int)gridDim.x >= total_tiles) {
                    slot->next_iter = it;
                    slot->k_done = 0;
                    slot->grid = gridDim.x;
                }
                break;
            }
            const int buf = (int)(seg & 1);
            const uint32_t t_acc = t_lane + buf * kBufCols;
            const int vrow = tile * kNOut + row - (kFold ? 1 : 0);
            bool valid = (!kFold || (row > 0 && row < kNM - 1)) && vrow < p.m_rows;
            size_t out_off = 0;
            if (valid) {
                const int n_img = fast_div(vrow, img, p.inv_img);
                const int r = vrow - n_img * img;
                const int hs = fast_div(r, p.in_ws, p.inv_in_ws);
                const int h = hs - p.in_off, w = r - hs * p.in_ws - p.in_off;
                valid = h >= 0 && h < p.out.H && w >= 0 && w < p.out.W;
                if (valid) out_off = (size_t)layout_row(p.out, n_img, h, w) * p.out.C;
            }
            if (leader) {
                const bool ok = mbar_wait(smem_u32(&ctl->tmem_full[buf]), (seg >> 1) & 1, abort_flag, kNWaitLimitNs);
                if (!ok) fail(1301);
                ctl->epi_go[group] = ok ? 1 : 0;
            }
            group_sync();
            if (!ctl->epi_go[group]) break;
            tc_fence_after_sync();
            const int kind = ctl->epi_kind[buf], k_done = ctl->epi_k_done[buf];
            if (kind == NEPI_EXIT) break;
            if (kind == NEPI_PARTIAL) {
                const int keep = p.drop_on_stop ? 0 : k_done;
                if (keep > (it == first_iter ? first_k : 0)) {
                    uint32_t v[32];
                    for (int c = 0; c < N; c += 32) {
                        tmem_ld_32x32(t_acc + c, v);
                        tmem_ld_wait();
                        uint4 *dst = reinterpret_cast<uint4 *>(spill) + (size_t)(c / 32) * 8 * kNM + row;
#pragma unroll
                        for (int j = 0; j < 8; ++j) dst[j * kNM] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    }
                }
                if (leader) {
                    slot->next_iter = it;
                    slot->k_done = keep;
                    slot->grid = gridDim.x;
                    if (blp.stop_index) atomicCAS(blp.stop_index, -1, blp.kernel_id);
                }
                break;
            }
#pragma unroll
            for (int half = 0; half < CO / 32; ++half) {
                float f[32];
                if constexpr (kFold) {
                    uint32_t l[32], m[32], r[32];
                    __syncwarp();
                    tmem_ld_32x32(t_acc, l);
                    tmem_ld_32x32(t_acc + CO, m);
                    tmem_ld_32x32(t_acc + 2 * CO, r);
                    tmem_ld_wait();
                    // the rows where this warp's lanes end, for the neighbouring warps
                    if (lane == 31 || lane == 0) {
                        float4 *e = reinterpret_cast<float4 *>(ctl->edge[group][quarter][lane == 31 ? 0 : 1]);
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            e[j] = lane == 31 ? make_float4(__uint_as_float(l[4 * j]), __uint_as_float(l[4 * j + 1]), __uint_as_float(l[4 * j + 2]), __uint_as_float(l[4 * j + 3]))
                                              : make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
                    }
                    tc_fence_before_sync();
                    group_sync();
                    if (leader) mbar_arrive(smem_u32(&ctl->tmem_empty[buf]));  // everything is in registers
                    const float *el = ctl->edge[group][quarter > 0 ? quarter - 1 : 0][0], *er = ctl->edge[group][quarter < 3 ? quarter + 1 : 3][1];
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
                        if (lane == 0) a = *reinterpret_cast<const float4 *>(el + j);
                        if (lane == 31) b = *reinterpret_cast<const float4 *>(er + j);
                        const float ea[4] = {a.x, a.y, a.z, a.w}, eb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float left = __shfl_up_sync(0xffffffffu, __uint_as_float(l[j + i]), 1), right = __shfl_down_sync(0xffffffffu, __uint_as_float(r[j + i]), 1);
                            left = lane == 0 ? ea[i] : left;
                            right = lane == 31 ? eb[i] : right;
                            f[j + i] = (left + __uint_as_float(m[j + i])) + right;
                        }
                    }
                } else {
                    uint32_t m[32];
                    __syncwarp();  // (lanes with rows and lanes without part behind the half before)
                    tmem_ld_32x32(t_acc + 32 * half, m);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(m[j]);
                    if (half == CO / 32 - 1) {
                        tc_fence_before_sync();
                        group_sync();
                        if (leader) mbar_arrive(smem_u32(&ctl->tmem_empty[buf]));
                    }
                }
                const float4 *b4 = reinterpret_cast<const float4 *>(ctl->bias + 32 * half);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 b = b4[j];
                    f[4 * j] += b.x, f[4 * j + 1] += b.y, f[4 * j + 2] += b.z, f[4 * j + 3] += b.w;
                }
                apply_act_n(f, p.relu);
                if (valid) {
                    uint32_t hi[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) hi[q] = pf_pack2(f[2 * q], f[2 * q + 1], p.fmt);
                    st_sector(p.out_hi + out_off + 32 * half, hi);
                    st_sector(p.out_hi + out_off + 32 * half + 16, hi + 8);
                }
            }
            ++tiles_done;
            if (leader && blp.executed) atomicAdd(blp.executed, 1);
        }
        if (leader && blp.trace && tiles_done) atomicAdd(blp.trace + 3, (unsigned long long)tiles_done);
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0 && lane == 0) {
        // nothing may still be on its way to this CTA's shared memory
        if (weights_asked) mbar_wait(smem_u32(&ctl->weights), 0, &ctl->raised, kNWaitLimitNs);
        if (*abort_flag)
            for (int spin = 0; spin < 64; ++spin) __nanosleep(1000);
    }
    if (warp == 1) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (threadIdx.x == 0 && blp.trace) atomicMax(blp.trace + 1, globaltimer_ns());
}

}  // namespace

cudaError_t conv3x3_narrow_prepare() {
    cudaError_t e = cudaFuncSetAttribute(conv3x3_narrow_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NarrowCfg<32>::kSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(conv3x3_narrow_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NarrowCfg<64>::kSmem);
}
int conv3x3_narrow_threads() { return kNThreads; }
int conv3x3_narrow_tiles(int m_rows, int cout) {
    const int out = cout == 32 ? NarrowCfg<32>::kOut : NarrowCfg<64>::kOut;
    return (m_rows + out - 1) / out;
}
int conv3x3_narrow_box(int cout) { return cout == 32 ? NarrowCfg<32>::kARows : NarrowCfg<64>::kARows; }

// 32 or 64 output channels whose weights fill the resident 72 KB at most.
bool conv3x3_narrow_fits(int cout, int cin) {
    return (cout == 32 || cout == 64) && cin % kNK == 0 && (uint32_t)(9 * cin * cout * 2) <= kNWBytes;
}

cudaError_t conv3x3_narrow_launch(const CgemmParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    void *args[] = {const_cast<CgemmParams *>(&p), const_cast<BlpArgs *>(&blp)};
    const bool few = p.cout_valid == 32;
    return launch_direct(few ? reinterpret_cast<const void *>(conv3x3_narrow_kernel<32>) : reinterpret_cast<const void *>(conv3x3_narrow_kernel<64>),
                         (unsigned)grid, (unsigned)kNThreads, few ? NarrowCfg<32>::kSmem : NarrowCfg<64>::kSmem, s, 1, args);
}

}  // namespace gpx
