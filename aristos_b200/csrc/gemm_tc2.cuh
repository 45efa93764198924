// Expert-FFN GEMM with paired blocks (tcgen05 cta_group::2): a cluster of two blocks on
// neighbouring SMs computes a 256 x 256 output tile -- two 128-row panels of the same local
// expert against the same 256 weight rows.  Each block TMA-loads its own panel (A) and only
// HALF of the weight tile (B), so the bytes pulled into an SM per FLOP drop by a third compared
// with one block per 128 x 256 tile.  Shared memory holds six 64-wide K slices per block, used
// as six shallow or three deep pipeline stages (template parameter kSub).  The epilogue stages
// its rows through a swizzled shared-memory tile so that every store instruction writes whole
// 128-byte lines, also when the destination is a peer's cell.  No load is multicast: every block
// fetches exactly the bytes it keeps.
//
// Per block, 384 threads:
//   warp 0      TMA producer (one lane): waits on its own `empty`, loads into its own shared
//               memory, credits the bytes to the LEADER's `full` barrier
//   warp 1      leader only: issues tcgen05.mma.cta_group::2, commits to `empty` and
//               `acc_full` of BOTH blocks
//   warp 2      tensor-memory allocation / release (both blocks, cta_group::2 forms)
//   warps 4..11 epilogue of the block's own 128 accumulator rows, half of the columns each; arrives
//               on the LEADER's `acc_empty`
// Work and epilogue semantics follow the reference's tile worker (os/processor/processor.cuh:
// 350-489,706-741).  Every wait is bounded.  This kernel runs one GEMM over a finished panel
// list (the dense single-expert layer, and the routed layer when its phases are launched one
// by one); the persistent kernel in moe_flow.cuh reuses its tile shapes and pipeline.
//
// Element types: bf16, fp16, and TF32 words (kind::tf32, torch_dtype 1; the reference's mma.sync
// m16n8k8 block GEMM, os/processor/mmaConfig.cuh:73-81).  A K slice is 128 bytes of a row and four
// instructions in either case: 64 16-bit or 32 4-byte elements.
// TF32, 4096 tokens, 16 experts, H = I = 2048: 120 and 127 us per launch of 68.7 GFLOP (573 and 541
// TFLOP/s); the 128 x 256 tiles of single blocks that it replaced took 148.
#pragma once

#include <cuda.h>

#include "gemm_common.cuh"
#include "tc_common.cuh"

namespace kleos {
namespace gemm_tc2 {

constexpr int BM = 128, BN = 256, BK = 64, UMMA_K = 16;  // BK: of 16-bit elements
constexpr int kSteps = BK / UMMA_K;                 // instructions per K slice, 32 bytes of a row each
constexpr int kSlices = 6;                        // 64-wide K slices of shared memory in total
constexpr int A_STAGE_BYTES = BM * BK * 2;        // 16 KiB: one K slice of this block's panel
constexpr int B_STAGE_BYTES = (BN / 2) * BK * 2;  // 16 KiB: one K slice of this block's half weight tile
constexpr int SLICE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
constexpr int kBackWarps = 8, kThreads = (4 + kBackWarps) * 32;
constexpr int TMEM_COLS = 512;  // two accumulators of 256 fp32 columns
constexpr int SMEM_BYTES = kSlices * SLICE_BYTES + 1024 + 28672;

struct Control {
    unsigned long long full[kSlices];   // used on the leader (one per pipeline stage)
    unsigned long long empty[kSlices];  // one per block
    unsigned long long acc_full[2];    // one per block
    unsigned long long acc_empty[2];   // used on the leader, 16 arrivals (8 warps x 2 blocks)
    uint32_t tmem_base;
    int abort;
    int le_start[257];
    __align__(16) float bias_s[kBackWarps][BN / 2];   // bias of the columns being read back, per epilogue warp
    __align__(16) uint4 stage_s[kBackWarps][16 * 8];  // per epilogue warp: 16 rows x 128 bytes, swizzled
};

static_assert(sizeof(Control) <= 28672, "control block must fit the shared memory set aside for it");

struct PairTile {
    int panel0, n_panels_left, nt, le;
};

// Tiles ordered by local expert, then N tile, then panel pair.
__device__ __forceinline__ bool decode_pair_tile(int t, const int* le_start, int le_begin,
                                                 int le_end, int NT, PairTile* c) {
    for (int le = le_begin; le < le_end; ++le) {
        const int p0 = le_start[le], np = le_start[le + 1] - p0;
        const int npair = (np + 1) >> 1;
        const int tiles = npair * NT;
        if (t < tiles) {
            const int nt = t / npair, pi = t - nt * npair;
            c->le = le;
            c->nt = nt;
            c->panel0 = p0 + 2 * pi;
            c->n_panels_left = np - 2 * pi;  // 1 when the pair's second panel does not exist
            return true;
        }
        t -= tiles;
    }
    return false;
}

__device__ __forceinline__ int total_pair_tiles(const int* le_start, int le_begin, int le_end,
                                                int NT) {
    int total = 0;
    for (int le = le_begin; le < le_end; ++le) total += ((le_start[le + 1] - le_start[le] + 1) >> 1) * NT;
    return total;
}

template <typename TE>
__host__ __device__ constexpr uint32_t instr_desc() {
    if constexpr (sizeof(TE) == 4) return tc::make_instr_desc_tf32(2 * BM, BN);
    else return tc::make_instr_desc_16b(2 * BM, BN, Pack2<TE>::kMmaFormat);
}

}  // namespace gemm_tc2

// kEpi selects the fused epilogue at compile time (0: bias + ReLU, 1: bias + GELU, 2: bias only)
// so the read-back loop stays a short straight-line sequence.
// kSub = 64-wide K slices per pipeline stage: 1 gives six shallow stages (best when the weights
// stream from HBM), 2 gives three deep stages and half the barrier round trips (best when the
// operands come from L2 and the tensor pipe is the limit).
template <typename TE, int kEpi, int kSub>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(gemm_tc2::kThreads, 1)
ffn_gemm_tc2(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
             GemmArgs g) {
    using namespace tc;
    using namespace gemm_tc2;
    constexpr int SUB = kSub, STAGES = kSlices / kSub, STAGE_BYTES = kSub * SLICE_BYTES;
    constexpr int NST = STAGES;
    constexpr bool kWide = sizeof(TE) == 4;           // TF32
    constexpr int BKE = 128 / (int)sizeof(TE);        // elements of a K slice
    constexpr uint32_t kInstrDesc = instr_desc<TE>();
    const long long t_kernel = clock64();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    Control* ctl = reinterpret_cast<Control*>(tiles + kSlices * SLICE_BYTES);
    __shared__ bool last_block;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t cta_rank = cluster_ctarank();
    const bool leader = cta_rank == 0;
    volatile int* abort_flag = &ctl->abort;

    if (tid == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(&ctl->full[s], 1);
            mbar_init(&ctl->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctl->acc_full[b], 1);
            mbar_init(&ctl->acc_empty[b], 2 * kBackWarps);
        }
        ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&ctl->tmem_base)), "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    pdl_trigger();
    for (int i = tid; i <= g.nLx; i += blockDim.x) ctl->le_start[i] = g.le_start[i];
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // both blocks' barriers exist before anything remote touches them
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    if (g.stats && tid == 0) g.stats[blockIdx.x * kStatSlots + 8] = clock64() - t_kernel;
    auto panel_at = [&](int i) -> PanelEntry { return g.panels[i]; };

    const int NT = (g.N + BN - 1) / BN;
    const int total = total_pair_tiles(ctl->le_start, g.le_begin, g.le_end, NT);
    const int KS = g.Kd / BKE;                // K slices
    const int KB = (KS + SUB - 1) / SUB;      // pipeline stages per tile
    const int n_clusters = (int)gridDim.x >> 1, cluster_id = blockIdx.x >> 1;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (both blocks)
        if (lane == 0) {
            asm volatile("fence.proxy.async;" ::: "memory");
            uint32_t it = 0;
            long long w_empty = 0;
            const long long t_begin = clock64();
            for (int t = cluster_id; t < total && !*abort_flag; t += n_clusters) {
                PairTile pt;
                if (!decode_pair_tile(t, ctl->le_start, g.le_begin, g.le_end, NT, &pt)) break;
                // the block without a panel of its own re-reads the first one and discards
                const int my_panel = pt.panel0 + ((int)cta_rank < pt.n_panels_left ? (int)cta_rank : 0);
                const PanelEntry p = panel_at(my_panel);
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const int s = it % NST;
                    const uint32_t ph = (it / NST) & 1;
                    if (!mbar_wait_timed(&ctl->empty[s], ph ^ 1, g.wait_cycles, abort_flag, &w_empty)) {
                        report_error(g.status, KLEOS_AT_GEMM_PRODUCER, t, (int)g.epoch);
                        *abort_flag = 1;
                        break;
                    }
                    // the leader announces the bytes of both blocks on its own barrier
                    const int nsub = min(SUB, KS - kb * SUB);
                    if (leader) mbar_expect_tx(&ctl->full[s], 2 * nsub * SLICE_BYTES);
                    const uint32_t full_leader = map_to_cta(smem_u32(&ctl->full[s]), 0);
                    uint8_t* sa = tiles + s * STAGE_BYTES;
                    for (int sub = 0; sub < nsub; ++sub) {
                        const int kx = (kb * SUB + sub) * BKE;
                        tma_load_2d_pair(sa + sub * SLICE_BYTES, &map_a, kx, p.row_base, full_leader);
                    }
                }
            }
            if (g.stats) {
                g.stats[blockIdx.x * kStatSlots + 0] = w_empty;
                g.stats[blockIdx.x * kStatSlots + 1] = clock64() - t_begin;
            }
        }
        __syncwarp();
    } else if (warp == 3) {
        // ------------------------------------------------------------ second TMA producer (both blocks)
        // The weight slices are issued by a thread of their own, next to the panel slices of
        // warp 0 (measured: 1.6 % off the launch).  It waits for the same free-stage barrier and
        // its bytes complete on the same full barrier; the byte count announced by warp 0 covers
        // both, and a slice landing before that announcement only makes the barrier's byte
        // count negative for a moment (the phase cannot complete before warp 0 has arrived).
        if (lane == 0) {
            asm volatile("fence.proxy.async;" ::: "memory");
            uint32_t it = 0;
            long long w_unused = 0;
            for (int t = cluster_id; t < total && !*abort_flag; t += n_clusters) {
                PairTile pt;
                if (!decode_pair_tile(t, ctl->le_start, g.le_begin, g.le_end, NT, &pt)) break;
                const int brow = pt.le * g.N + pt.nt * BN + (int)cta_rank * (BN / 2);
                bool ok = true;
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const int s = it % NST;
                    const uint32_t ph = (it / NST) & 1;
                    if (!mbar_wait_timed(&ctl->empty[s], ph ^ 1, g.wait_cycles, abort_flag, &w_unused)) {
                        ok = false;  // the first producer reports the failure
                        break;
                    }
                    const int nsub = min(SUB, KS - kb * SUB);
                    const uint32_t full_leader = map_to_cta(smem_u32(&ctl->full[s]), 0);
                    uint8_t* sa = tiles + s * STAGE_BYTES;
                    for (int sub = 0; sub < nsub; ++sub)
                        tma_load_2d_pair(sa + sub * SLICE_BYTES + A_STAGE_BYTES, &map_b, (kb * SUB + sub) * BKE, brow,
                                         full_leader);
                }
                if (!ok) break;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader only)
        // (the whole warp runs the loop and the elected lane issues, see tc::elect_one)
        if (leader) {
            const uint32_t elected = elect_one();
            const uint32_t slices = smem_u32(tiles), bars = smem_u32(ctl), tmem = (uint32_t)uniform((int)tmem_base);
            const int n_tiles = uniform(total);
            uint32_t s = 0, ph = 0, tile_n = 0;
            long long w_acc = 0, w_full = 0;
            const long long t_begin = clock64();
            for (int t = cluster_id; t < n_tiles; t += n_clusters, ++tile_n) {
                const uint32_t buf = tile_n & 1, use = tile_n >> 1;
                if (!mbar_wait_timed(&ctl->acc_empty[buf], (use & 1) ^ 1, g.wait_cycles, abort_flag, &w_acc)) {
                    if (lane == 0) report_error(g.status, KLEOS_AT_GEMM_MMA, t, (int)g.epoch);
                    *abort_flag = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem + buf * BN;
                bool ok = true;
                for (int kb = 0; kb < KB; ++kb) {
                    if (!mbar_wait_timed(&ctl->full[s], ph, g.wait_cycles, abort_flag, &w_full)) {
                        if (lane == 0) report_error(g.status, KLEOS_AT_GEMM_MMA, t, (int)g.epoch);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = slices + s * STAGE_BYTES;
#pragma unroll
                    for (int sub = 0; sub < SUB; ++sub) {
                        if (sub > 0 && kb * SUB + sub >= KS) break;  // the last deep stage may be half full
                        const uint64_t da = make_smem_desc(sa + sub * SLICE_BYTES);
                        const uint64_t db = make_smem_desc(sa + sub * SLICE_BYTES + A_STAGE_BYTES);
#pragma unroll
                        for (int k = 0; k < kSteps; ++k) {
                            const uint32_t more = (sub | k) != 0 ? 1u : (uint32_t)(kb != 0);
                            if constexpr (kWide) umma_tf32_pair_if(elected, d_tmem, da + 2 * k, db + 2 * k, kInstrDesc, more);
                            else umma_bf16_pair_if(elected, d_tmem, da + 2 * k, db + 2 * k, kInstrDesc, more);
                        }
                    }
                    // the stage is free in both blocks once these MMAs have read it
                    umma_commit_both_if(elected, bars + (uint32_t)offsetof(Control, empty) + 8 * s);
                    if (++s == NST) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (!ok) break;
                umma_commit_both_if(elected, bars + (uint32_t)offsetof(Control, acc_full) + 8 * buf);
            }
            if (g.stats && lane == 0) {
                g.stats[blockIdx.x * kStatSlots + 2] = w_acc;
                g.stats[blockIdx.x * kStatSlots + 3] = w_full;
                g.stats[blockIdx.x * kStatSlots + 4] = clock64() - t_begin;
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        // ------------------------------------------------------------ epilogue (both blocks)
        // Eight warps, two per quadrant of the accumulator rows, and a rolled loop over 64-column groups.
        // With four warps and the tile's 256 erff per thread unrolled, layers with GELU waited for their
        // read-back and for instructions: 6016 tokens, H = 1472, I = 3008, dense: 166 -> 91 us.
        const int q = warp & 3, half = (warp - 4) >> 2, w8 = warp - 4;
        const TE* bias = static_cast<const TE*>(g.bias);
        uint32_t tile_n = 0;
        long long w_accfull = 0, w_tmem = 0;
        const long long t_begin = clock64();
        for (int t = cluster_id; t < total; t += n_clusters, ++tile_n) {
            PairTile pt;
            if (!decode_pair_tile(t, ctl->le_start, g.le_begin, g.le_end, NT, &pt)) break;
            const bool have_panel = (int)cta_rank < pt.n_panels_left;
            const PanelEntry p = panel_at(pt.panel0 + (have_panel ? (int)cta_rank : 0));
            const int rows = have_panel ? p.rows : 0;
            const uint32_t buf = tile_n & 1, use = tile_n >> 1;
            if (*abort_flag) break;
            {
                // stage the bias of this warp's 128 columns in shared memory (one load per lane)
                // while the main loop of the tile is still running: global loads issued later would
                // queue behind the operand traffic streaming into this SM
                const int nb = pt.nt * BN + half * (BN / 2) + 4 * lane;
                float* bs = &ctl->bias_s[w8][4 * lane];
                if (nb < g.N) {
                    const TE* src = bias + (size_t)pt.le * g.N + nb;
                    if constexpr (kWide) {
                        *reinterpret_cast<float4*>(bs) = __ldg(reinterpret_cast<const float4*>(src));
                    } else {
                        using TE2 = typename Pack2<TE>::type;
                        const uint2 raw = __ldg(reinterpret_cast<const uint2*>(src));
                        const TE2* h2 = reinterpret_cast<const TE2*>(&raw);
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const float2 f = Pack2<TE>::to_f2(h2[j]);
                            bs[2 * j] = f.x;
                            bs[2 * j + 1] = f.y;
                        }
                    }
                }
                __syncwarp();
            }
            if (!mbar_wait_timed(&ctl->acc_full[buf], use & 1, g.wait_cycles, abort_flag, &w_accfull)) {
                if (lane == 0) report_error(g.status, KLEOS_AT_GEMM_EPILOGUE, t, (int)g.epoch);
                *abort_flag = 1;
                break;
            }
            tc_fence_after();
            const int n0 = pt.nt * BN + half * (BN / 2);
            const uint32_t taddr = tmem_base + buf * BN + half * (BN / 2) + (static_cast<uint32_t>(q * 32) << 16);
            // this warp's 32 accumulator rows; rows_w of them carry tokens
            const int rows_w = min(32, rows - q * 32);
            if (rows_w <= 0) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_pair(map_to_cta(smem_u32(&ctl->acc_empty[buf]), 0));
                continue;
            }
            TE* obase = out_ptr<TE>(g, p, q * 32, n0);
            uint4* stg = ctl->stage_s[w8];
            // Every 128 bytes of the rows (64 or 32 columns) the warp transposes through a swizzled
            // shared-memory tile, sixteen rows at a time, so that each store instruction writes four
            // complete 128-byte lines (one row segment per 8 lanes) instead of 32 scattered 16-byte
            // pieces: this is what the NVLink path to a peer's cell needs.
#pragma unroll 1
            for (int cc = 0; cc < BN / 2; cc += BKE) {
                uint32_t r[BKE];
                tmem_ld_32x32(taddr + cc, r);
                if constexpr (!kWide) tmem_ld_32x32(taddr + cc + 32, r + 32);
                const long long tq = clock64();
                tmem_ld_wait();
                w_tmem += clock64() - tq;
                if (cc + BKE == BN / 2) {
                    // this warp's part of the accumulator is in registers: hand it back to the MMA issuer
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_pair(map_to_cta(smem_u32(&ctl->acc_empty[buf]), 0));
                }
                if (n0 + cc >= g.N) continue;
                const float4* bq = reinterpret_cast<const float4*>(&ctl->bias_s[w8][cc]);
#pragma unroll
                for (int j = 0; j < BKE / 2; ++j) {
                    const float4 bf = bq[j >> 1];
                    float v0 = __uint_as_float(r[2 * j]) + ((j & 1) ? bf.z : bf.x);
                    float v1 = __uint_as_float(r[2 * j + 1]) + ((j & 1) ? bf.w : bf.y);
                    if constexpr (kEpi == 0) {
                        v0 = fmaxf(v0, 0.f);
                        v1 = fmaxf(v1, 0.f);
                    } else if constexpr (kEpi == 1) {
                        v0 = apply_act(v0, 1);
                        v1 = apply_act(v1, 1);
                    }
                    if constexpr (kWide) {
                        r[2 * j] = __float_as_uint(round_tf32(v0));
                        r[2 * j + 1] = __float_as_uint(round_tf32(v1));
                    } else {
                        const auto h = Pack2<TE>::from_f2(v0, v1);
                        r[j] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                }
#pragma unroll
                for (int p0 = 0; p0 < 32; p0 += 16) {
                    if (p0 >= rows_w) break;
                    if ((lane & 16) == p0) {
#pragma unroll
                        for (int ch = 0; ch < 8; ++ch)
                            stg[(lane & 15) * 8 + (ch ^ (lane & 7))] =
                                make_uint4(r[4 * ch], r[4 * ch + 1], r[4 * ch + 2], r[4 * ch + 3]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int it = 0; it < 4; ++it) {
                        const int rr = it * 4 + (lane >> 3), ch = lane & 7;
                        const uint4 v = stg[rr * 8 + (ch ^ (rr & 7))];
                        if (p0 + rr < rows_w)
                            *reinterpret_cast<uint4*>(obase + (size_t)(p0 + rr) * g.N + cc + ch * (16 / (int)sizeof(TE))) = v;
                    }
                    __syncwarp();
                }
            }
        }
        if (g.stats && warp == 4 && lane == 0) {
            g.stats[blockIdx.x * kStatSlots + 5] = w_accfull;
            g.stats[blockIdx.x * kStatSlots + 6] = clock64() - t_begin;
            g.stats[blockIdx.x * kStatSlots + 7] = w_tmem;
        }
    }

    // teardown: neither block may leave while its partner can still touch its shared memory,
    // barriers or tensor memory
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) settle_after_abort();
    cluster_sync_all();
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(TMEM_COLS)
                     : "memory");
    }
    if (g.mode == 1) publish_return_flags(g.ret, &last_block);
}

}  // namespace kleos
