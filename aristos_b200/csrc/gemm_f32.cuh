// Expert-FFN GEMM of float layers (torch_dtype 0) on the 5th-generation tensor cores.
//
// Every fp32 operand is the exact sum of three bf16 values, its leading, middle and trailing eight
// significand bits (x = h + m + l, each part a truncation of what the parts before it leave), so
// a product of two operands is nine bf16 products.  All but l*l, which is below 2^-30 of the product,
// are computed.  An operand below 2^-110 loses its bits under 2^-133, the smallest bf16 value.
// (Splitting fp32 operands over several low-precision products: Henry, Tang, Heinecke, "Leveraging the
// bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations", ARITH 2019; summing
// short runs on the matrix unit and the runs in fp32 registers: Ootomo, Yokota, "Recovering single
// precision accuracy from Tensor Cores", IJHPCA 2022.)  The matrix unit does not
// round its running sum to nearest, so h*h is summed apart from the seven small products, which
// together are below 2^-6 of it, and no sum stays there for long: the h*h sums are read back every two
// K slices of 32 (a step) and the small sums every two steps, and both are added up in registers with
// ordinary fp32 additions.  So a sum of one term is as exact as a rounded fp32 product (at most 2^-24
// (1 + 2^-4) of it); six products in one accumulator left up to 5e-7.  With the small sums kept for
// four steps a launch was 2 % faster, and sums of positive terms less exact (2.2e-7, now 1.9e-7).
//
// An infinity or NaN among the operands makes the h*h sums what fp32 multiply-adds give: the leading
// part of such a value is one too.  The small sums beside it are NaN; they are limited to finite values
// on the way to the registers and so leave an infinity or NaN there as it is.
//
// A cluster of two blocks computes a 256 x BN tile (cta_group::2), as in
// moe_flow.cuh.  The parts of the
// panel go to tensor memory (the MMA's A operand may come from there), those of the weight rows to
// shared memory: with both in shared memory the eight products' operand reads would make its bandwidth
// the limit (per K slice and block at BN = 128: 96 KiB of them, 36 KiB of part stores and 24 KiB each way
// for the fp32 rows, 1440 cycles at 128 bytes a cycle, against sixteen instructions of 64 cycles; this
// way 92 KiB in all, 736 cycles).  BN = 64 is for layers with too few tiles to fill the chip.
//
// Per block, 512 threads:
//   warps 0..7    drain: the sums of every step are added to the warp's registers (32 rows x
//                 BN / 2 columns); after a tile's last step bias, activation and stores
//   warps 8..11   split the panel: one row per thread, fp32 slice -> three parts in tensor memory
//   warps 12, 13  split the weight rows: fp32 slice -> three part planes in shared memory, in the
//                 swizzle the MMA reads
//   warp 14       tensor-memory owner; in the leader block also the MMA issuer
//   warp 15       TMA producer: fp32 rows, 32 columns at a time, into a ring
// Measured (4096 tokens, 16 experts, H = I = 2048, one launch = 68.7 GFLOP): 404 us, where the FP32
// FMA kernel (gemm_simt.cuh) took 1630; the layer's output is 2.9e-7 from the 64-bit result (relative
// 2-norm), with that kernel 1.2e-6.  A slice takes 1380 cycles of the 1024 its MMAs need.  Slower forms,
// measured with six products: rows loaded into registers instead of staged by TMA 510 us (the stages
// leave little L1 for loads in flight) where this form took 368, panel parts in shared memory 388, two
// roles fewer (the same warps split and drain) 420.
#pragma once

#include <cfloat>
#include <type_traits>

#include "gemm_common.cuh"
#include "tc_common.cuh"

namespace kleos {
namespace gemm_f32 {
using namespace tc;

constexpr int BM = 128, BK = 32, UMMA_K = 16;
constexpr int ROW = BK * 2;  // bytes of a part row: 64, the swizzle span
constexpr int kDrain = 8, kSplitA = 4, kSplitB = 2, kSplit = kSplitA + kSplitB;  // warps
constexpr int kMmaWarp = kDrain + kSplit, kTmaWarp = kMmaWarp + 1;
constexpr int kThreads = (kTmaWarp + 1) * 32;  // 128 registers a thread
constexpr int kStages = 4, kMaxRing = 6;
constexpr int kStep = 2;   // K slices whose h*h products share a read-back
constexpr int kGroup = 2;  // steps whose small products share one
constexpr int A_COLS = 3 * BK / 2;  // tensor-memory columns of a stage's panel parts, two bf16 a column

struct Control {
    unsigned long long ring_full[kMaxRing];   // TMA bytes of the slot have landed
    unsigned long long ring_empty[kMaxRing];  // the team of split warps has read the slot
    unsigned long long full[kStages];         // used on the leader: the slice's parts are in place, a team of both blocks
    unsigned long long done[kStages];         // one per block: the MMAs of the slice have completed
    unsigned long long sum_full[2];           // one per block: [0] the h*h sums of a step, [1] the small sums of a group are complete
    unsigned long long sum_empty[2];          // used on the leader: ... and have been read, drain warps of both blocks
    uint32_t tmem_base;
    int abort;
    int last_block;
    int le_start[257];
};
static_assert(sizeof(Control) <= 2048, "control block must fit the shared memory set aside for it");

template <int BN>
struct Shape {
    static constexpr int HALF = BN / 2;                  // weight rows this block supplies
    static constexpr int PLANE = HALF * ROW;             // one part of them
    static constexpr int STAGE_BYTES = 3 * PLANE;
    static constexpr int SLOT_BYTES = (BM + HALF) * BK * 4;  // panel rows, then weight rows
    static constexpr int RING = 6;
    static constexpr int A_COL0 = 2 * BN;                // tensor memory: h*h sums, small sums, then the panel parts
    static_assert(A_COL0 + kStages * A_COLS <= 512, "tensor memory has 512 columns");
    static constexpr int STORE_BYTES = kDrain * 1024;    // per drain warp: 8 rows x 32 columns on the way out
    static constexpr int SMEM_BYTES = kStages * STAGE_BYTES + RING * SLOT_BYTES + STORE_BYTES + 1024 + 2048;
    static constexpr int TMEM_COLS = 512;
};
static_assert(Shape<128>::SMEM_BYTES <= 232448 && Shape<64>::SMEM_BYTES <= 232448,
              "227 KiB of shared memory per block");

// Shared-memory matrix descriptor of a part plane: K-major, rows of 64 bytes with the swizzle of that
// span, groups of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t part_desc(uint32_t addr) {
    return (make_smem_desc(addr) & ~((7ull << 61) | (0x3fffull << 32))) | (4ull << 61) |
           (static_cast<uint64_t>(512 >> 4) << 32);
}

// 256 x N accumulator += A (tensor memory of each block of the pair, 128 rows) x B (shared memory)
__device__ __forceinline__ void umma_bf16_pair_ta(uint32_t issue, uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b,
                                                  uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(issue)
        : "memory");
}
// 16 registers per thread -> 32 lanes x 16 columns of tensor memory
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
        : "memory");
}

// Four consecutive fp32 values -> their leading, middle and trailing eight bits as bf16.  The leading part
// of an infinity or NaN is one too (the conversion keeps every NaN a NaN); the other two are then NaN.
__device__ __forceinline__ void split4(const float4& x, uint2* h, uint2* m, uint2* l) {
    const float v[4] = {x.x, x.y, x.z, x.w};
    uint32_t top[2], mid[4], low[4];
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
        asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(top[k / 2]) : "f"(v[k + 1]), "f"(v[k]));
        const float r[2] = {v[k] - __uint_as_float(top[k / 2] << 16), v[k + 1] - __uint_as_float(top[k / 2] & 0xffff0000u)};  // exact
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mid[k + i] = __float_as_uint(r[i]);
            low[k + i] = __float_as_uint(r[i] - __uint_as_float(mid[k + i] & 0xffff0000u));
        }
    }
    *h = make_uint2(top[0], top[1]);
    *m = make_uint2(__byte_perm(mid[0], mid[1], 0x7632), __byte_perm(mid[2], mid[3], 0x7632));
    *l = make_uint2(__byte_perm(low[0], low[1], 0x7632), __byte_perm(low[2], low[3], 0x7632));
}

// Bounded wait without a pause between the polls (each of which already waits in hardware for a while):
// here the waits hand a slice of under a thousand cycles from one role to the next.
__device__ __forceinline__ bool mbar_spin(unsigned long long* bar, uint32_t parity, long long budget, volatile int* abort) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity))
        if (*abort || clock64() - t0 > budget) return false;
    return true;
}

// Position in a ring of n buffers and the parity of the current round.
struct Turn {
    int n, at = 0;
    uint32_t parity = 0;
    __device__ __forceinline__ explicit Turn(int n_) : n(n_) {}
    __device__ __forceinline__ void next() {
        if (++at == n) {
            at = 0;
            parity ^= 1;
        }
    }
};

}  // namespace gemm_f32

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(gemm_f32::kThreads, 1)
ffn_gemm_f32(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, GemmArgs g) {
    using namespace tc;
    using namespace gemm_f32;
    using Sh = Shape<BN>;
    constexpr uint32_t kInstrDesc = make_instr_desc_bf16(2 * BM, BN);
    constexpr int CW = BN / 2;  // accumulator columns a drain warp keeps
    extern __shared__ uint8_t smem_raw[];
    uint8_t* stages = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* ring = stages + kStages * Sh::STAGE_BYTES;
    uint8_t* store = ring + Sh::RING * Sh::SLOT_BYTES;
    Control* ctl = reinterpret_cast<Control*>(store + Sh::STORE_BYTES);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t cta_rank = cluster_ctarank();
    volatile int* abort_flag = &ctl->abort;

    if (tid == 0) {
        for (int s = 0; s < Sh::RING; ++s) {
            mbar_init(&ctl->ring_full[s], 1);
            mbar_init(&ctl->ring_empty[s], kSplit);
        }
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&ctl->full[s], 2 * kSplit);
            mbar_init(&ctl->done[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&ctl->sum_full[b], 1);
            mbar_init(&ctl->sum_empty[b], 2 * kDrain);
        }
        ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&ctl->tmem_base)), "r"(Sh::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    pdl_trigger();
    for (int i = tid; i <= g.nLx; i += kThreads) ctl->le_start[i] = g.le_start[i];
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // both blocks' barriers exist before anything remote touches them
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;

    const int NT = (g.N + BN - 1) / BN;
    const int total = total_pair_tiles(ctl->le_start, g.le_begin, g.le_end, NT);
    const int KB = g.Kd / BK;
    const int n_clusters = (int)gridDim.x >> 1, cluster_id = (int)blockIdx.x >> 1;
    const int my_tiles = total > cluster_id ? (total - cluster_id + n_clusters - 1) / n_clusters : 0;
    const int slices = my_tiles * KB, steps = KB / kStep;  // (a row is a multiple of 64 long)

    if (warp == kTmaWarp) {
        // ------------------------------------------------------------ TMA producer (both blocks)
        if (lane == 0) {
            // dispatched rows and y1 rows were written with ordinary stores
            asm volatile("fence.proxy.async;" ::: "memory");
            Turn slot(Sh::RING);
            bool ok = true;
            for (int t = cluster_id; ok && t < total; t += n_clusters) {
                PairTile pt;
                if (!decode_pair_tile(t, ctl->le_start, g.le_begin, g.le_end, NT, &pt)) break;
                // the block without a panel of its own re-reads the first one and discards
                const PanelEntry p = g.panels[pt.panel0 + ((int)cta_rank < pt.n_panels_left ? (int)cta_rank : 0)];
                const int brow = pt.le * g.N + pt.nt * BN + (int)cta_rank * Sh::HALF;
                for (int k = 0; k < g.Kd; k += BK) {
                    if (!mbar_spin(&ctl->ring_empty[slot.at], slot.parity ^ 1, g.wait_cycles, abort_flag)) {
                        report_error(g.status, KLEOS_AT_GEMM_PRODUCER, t, (int)g.epoch);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    unsigned long long* bar = &ctl->ring_full[slot.at];
                    uint8_t* dst = ring + slot.at * Sh::SLOT_BYTES;
                    mbar_expect_tx(bar, Sh::SLOT_BYTES);
                    tma_load_2d(dst, &map_a, k, p.row_base, bar);
                    tma_load_2d(dst + BM * BK * 4, &map_b, k, brow, bar);
                    slot.next();
                }
            }
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------ MMA issuer (leader only)
        if (cta_rank == 0) {
            // parts of the panel and of the weight rows whose products are summed apart from h*h, smallest first
            constexpr int kPartA[7] = {2, 1, 2, 0, 1, 1, 0}, kPartB[7] = {1, 2, 0, 2, 1, 0, 1};
            const uint32_t elected = elect_one(), tmem = (uint32_t)uniform((int)tmem_base);
            const uint32_t bars = smem_u32(ctl), parts = smem_u32(stages);
            const int n = uniform(my_tiles * steps), n_steps = uniform(steps);
            auto multiply = [&](int s, int pa, int pb, uint32_t d, bool more) {
                const uint32_t ta = tmem + Sh::A_COL0 + s * A_COLS + pa * (BK / 2);
                const uint64_t db = part_desc(parts + s * Sh::STAGE_BYTES + pb * Sh::PLANE);
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k)
                    umma_bf16_pair_ta(elected, d, ta + k * (UMMA_K / 2), db + 2 * k, kInstrDesc, (more || k > 0) ? 1u : 0u);
            };
            auto wait = [&](unsigned long long* bar, uint32_t parity) {
                const bool ok = mbar_spin(bar, parity, g.wait_cycles, abort_flag);
                tc_fence_after();
                return ok;
            };
            int s = 0, kd = 0;                // stage; step of the tile
            uint32_t sp = 0, hp = 0, lp = 0;  // parities: stages, h*h sums, small sums
            bool ok = true;
            for (int i = 0; i < n; ++i) {
                ok = wait(&ctl->sum_empty[0], hp ^ 1);
                hp ^= 1;
#pragma unroll
                for (int j = 0; j < kStep; ++j) {
                    ok = ok && wait(&ctl->full[s + j], sp);
                    if (ok) multiply(s + j, 0, 0, tmem, j > 0);
                }
                if (!ok) break;
                umma_commit_both_if(elected, bars + (uint32_t)offsetof(Control, sum_full));
                const bool first = kd % kGroup == 0;
                if (first) {
                    if (!(ok = wait(&ctl->sum_empty[1], lp ^ 1))) break;
                    lp ^= 1;
                }
#pragma unroll
                for (int j = 0; j < kStep; ++j) {
#pragma unroll
                    for (int t = 0; t < 7; ++t) multiply(s + j, kPartA[t], kPartB[t], tmem + BN, !first || (j | t) != 0);
                    umma_commit_both_if(elected, bars + (uint32_t)offsetof(Control, done) + 8 * (s + j));
                }
                if (++kd == n_steps) kd = 0;
                if (kd % kGroup == 0) umma_commit_both_if(elected, bars + (uint32_t)offsetof(Control, sum_full) + 8);
                s += kStep;
                if (s == kStages) {
                    s = 0;
                    sp ^= 1;
                }
            }
            if (!ok) {
                if (lane == 0) report_error(g.status, KLEOS_AT_GEMM_MMA, kd, (int)g.epoch);
                *abort_flag = 1;
            }
        }
        __syncwarp();
    } else if (warp >= kDrain) {
        // ------------------------------------------------------------ split (both blocks)
        const bool panel = warp < kDrain + kSplitA;
        // panel: lane = row of the warp's quadrant.  Weight rows: four columns of every eighth row; the
        // eight lanes of a shared-memory phase read one 128-byte row, sixteen lanes store two 64-byte rows
        const int q = warp & 3, row = q * 32 + lane;
        constexpr int STEP = kSplitB * 32 / 8;
        static_assert(STEP % 8 == 0, "the swizzle is the same for all of a thread's rows");
        const int r0 = (tid - (kDrain + kSplitA) * 32) >> 3, c4 = tid & 7;
        const uint32_t in = (uint32_t)(BM + r0) * 128 + (uint32_t)((c4 ^ (r0 & 7)) << 4);
        const uint32_t part = (uint32_t)r0 * ROW + (uint32_t)((((c4 >> 1) ^ ((r0 >> 1) & 3)) << 4) + ((c4 & 1) << 3));
        Turn stage(kStages), slot(Sh::RING);
        for (int i = 0; i < slices; ++i) {
            // the stage is free once the MMAs of slice i - kStages have completed
            if (!mbar_spin(&ctl->done[stage.at], stage.parity ^ 1, g.wait_cycles, abort_flag) ||
                !mbar_spin(&ctl->ring_full[slot.at], slot.parity, g.wait_cycles, abort_flag)) {
                if (lane == 0) report_error(g.status, KLEOS_AT_GEMM_MMA, i, (int)g.epoch);
                *abort_flag = 1;
                break;
            }
            const uint8_t* src = ring + slot.at * Sh::SLOT_BYTES;
            if (panel) {
                uint32_t h[16], m[16], l[16];
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    split4(*reinterpret_cast<const float4*>(src + row * 128 + ((c ^ (row & 7)) << 4)),
                           reinterpret_cast<uint2*>(h + 2 * c), reinterpret_cast<uint2*>(m + 2 * c),
                           reinterpret_cast<uint2*>(l + 2 * c));
                tc_fence_after();
                const uint32_t ta = tmem_base + Sh::A_COL0 + stage.at * A_COLS + (static_cast<uint32_t>(q * 32) << 16);
                tmem_st_32x16(ta, h);
                tmem_st_32x16(ta + BK / 2, m);
                tmem_st_32x16(ta + BK, l);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
            } else {
                uint8_t* dst = stages + stage.at * Sh::STAGE_BYTES + part;
#pragma unroll
                for (int r = 0; r < Sh::HALF; r += STEP) {
                    uint2 h, m, l;
                    split4(*reinterpret_cast<const float4*>(src + in + r * 128), &h, &m, &l);
                    *reinterpret_cast<uint2*>(dst + r * ROW) = h;
                    *reinterpret_cast<uint2*>(dst + r * ROW + Sh::PLANE) = m;
                    *reinterpret_cast<uint2*>(dst + r * ROW + 2 * Sh::PLANE) = l;
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_pair(map_to_cta(smem_u32(&ctl->full[stage.at]), 0));
                mbar_arrive(&ctl->ring_empty[slot.at]);
            }
            stage.next();
            slot.next();
        }
    } else {
        // ------------------------------------------------------------ drain (both blocks)
        const float* bias = static_cast<const float*>(g.bias);
        const int q = warp & 3, half = warp >> 2;
        uint4* stg = reinterpret_cast<uint4*>(store + warp * 1024);
        float acc[CW];
#pragma unroll
        for (int j = 0; j < CW; ++j) acc[j] = 0.f;
        // Adds an accumulator to the registers and hands it back to the MMA issuer.  Small sums are NaN or
        // infinite only beside h*h sums that are not finite either: limited, they leave those as they are.
        auto add = [&](int which, uint32_t parity, auto small) -> bool {
            if (!mbar_spin(&ctl->sum_full[which], parity, g.wait_cycles, abort_flag)) return false;
            tc_fence_after();
            const uint32_t taddr = tmem_base + which * BN + half * CW + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll
            for (int c = 0; c < CW / 32; ++c) {
                uint32_t v[32];
                tmem_ld_32x32(taddr + c * 32, v);
                tmem_ld_wait();
                if (c + 1 == CW / 32) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_pair(map_to_cta(smem_u32(&ctl->sum_empty[which]), 0));
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    float x = __uint_as_float(v[j]);
                    if (decltype(small)::value) x = fmaxf(fminf(x, FLT_MAX), -FLT_MAX);
                    acc[c * 32 + j] += x;
                }
            }
            return true;
        };
        int tile = cluster_id, kd = 0;  // tile the sums belong to, its steps added up so far
        uint32_t hp = 0, lp = 0;
        for (int i = 0; i < my_tiles * steps; ++i) {
            bool ok = add(0, hp, std::false_type());
            hp ^= 1;
            if (++kd == steps || kd % kGroup == 0) {
                ok = ok && add(1, lp, std::true_type());
                lp ^= 1;
            }
            if (!ok) {
                if (lane == 0) report_error(g.status, KLEOS_AT_GEMM_EPILOGUE, tile, (int)g.epoch);
                *abort_flag = 1;
                break;
            }
            if (kd < steps) continue;
            kd = 0;
            // the tile is complete: transpose 32 columns at a time, so that each store instruction
            // writes whole 128-byte lines (the destination may be a peer's cell)
            PairTile pt;
            if (!decode_pair_tile(tile, ctl->le_start, g.le_begin, g.le_end, NT, &pt)) break;
            tile += n_clusters;
            const bool have = (int)cta_rank < pt.n_panels_left;
            const PanelEntry p = g.panels[pt.panel0 + (have ? (int)cta_rank : 0)];
            const int rows_w = min(32, (have ? p.rows : 0) - q * 32);
            const int n0 = pt.nt * BN + half * CW;
            float* obase = out_ptr<float>(g, p, q * 32, n0);
            // (the result of a dense layer lies where the caller put it)
            const bool aligned = (reinterpret_cast<uintptr_t>(obase) & 15) == 0;
            const float* bq = bias + (size_t)pt.le * g.N + n0;
#pragma unroll
            for (int c = 0; c < CW / 32; ++c) {
#pragma unroll 1
                for (int hr = 0; hr < 32; hr += 8) {  // eight rows at a time
                    if (hr >= rows_w || n0 + c * 32 >= g.N) break;
                    if ((lane & 24) == hr) {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            stg[(lane & 7) * 8 + (j ^ (lane & 7))] = make_uint4(
                                __float_as_uint(acc[c * 32 + 4 * j]), __float_as_uint(acc[c * 32 + 4 * j + 1]),
                                __float_as_uint(acc[c * 32 + 4 * j + 2]), __float_as_uint(acc[c * 32 + 4 * j + 3]));
                    }
                    __syncwarp();
                    const int j = lane & 7, col = c * 32 + 4 * j;
                    const float4 bf = *reinterpret_cast<const float4*>(bq + col);
#pragma unroll 1
                    for (int r = lane >> 3; r < 8 && hr + r < rows_w; r += 4) {
                        const uint4 raw = stg[r * 8 + (j ^ r)];
                        float v[4] = {__uint_as_float(raw.x), __uint_as_float(raw.y), __uint_as_float(raw.z), __uint_as_float(raw.w)};
                        const float b4[4] = {bf.x, bf.y, bf.z, bf.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            v[k] += b4[k];
                            if (g.mode == 0) v[k] = apply_act(v[k], g.hidden_act);
                        }
                        float* o = obase + (size_t)(hr + r) * g.N + col;
                        if (aligned) {
                            *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
                        } else {
#pragma unroll
                            for (int k = 0; k < 4; ++k) o[k] = v[k];
                        }
                    }
                    __syncwarp();
                }
            }
#pragma unroll
            for (int j = 0; j < CW; ++j) acc[j] = 0.f;
        }
    }

    // teardown: neither block may leave while its partner can still touch its shared memory,
    // barriers or tensor memory
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) settle_after_abort();
    cluster_sync_all();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Sh::TMEM_COLS)
                     : "memory");
    }
    if (g.mode == 1 && g.ret.world > 0) publish_return_flags(g.ret, &ctl->last_block);
}

}  // namespace kleos
