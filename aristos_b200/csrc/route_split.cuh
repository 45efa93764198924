// Router of 16-bit and TF32 layers of up to 128 experts in ONE launch: gate GEMM on the tensor cores,
// softmax, top-k, near-tie re-evaluation, slots, counts and, on one rank, the rows' way into the cells.
//
// What bounds it is latency: the bytes and multiply-adds take 5 us at most on the largest layers and
// next to nothing on the others, while 128 tokens a block, then thread by thread over the experts of its tokens,
// then through grid barriers, take 30 to 40.  So every step is spread:
//   * 16-bit layers: a block has 32, 64 or 128 tokens to itself, the fewest with which the chip holds all blocks, and
//     walks all of K for them with up to fourteen slices in flight.  Every logit is one sum over K, and the
//     softmax sum goes by experts, so a token's results do not depend on the size of the layer, and they are the bits
//     of the persistent kernel (moe_flow.cuh);
//   * TF32 layers and kleos_route_static (kSplit): a cluster of C = 1, 2 or 4 blocks shares 128 tokens, each block
//     multiplying its part of K (Args::parts), and exchanges partial logits through distributed shared memory,
//     one bulk copy per pair of blocks (16-byte stores from tensor memory to the other block took 4 us): block r
//     gets all parts of the tokens [r, r + 1) * 128 / C and adds them in order of K.  (16-bit layers did so
//     too, and took 20.9 instead of 23.9 us in a decode step, 47.5 instead of 54.1 at H = 4096, 30.2 instead of
//     29.4 at 8192 tokens, H = 2048: with bits that changed with the number of tokens.)
//   * four threads per token, each with a quarter of the experts, do softmax and top-k;
//   * slots without a grid barrier: place_tokens(), route.cuh.
// Measured, router and row copy, alone and cold (before: the persistent kernel's routing phase and a copy kernel): 256
// tokens, 8 experts 28 us -> 15; 8192 tokens, 64 experts 54 -> 43 (29 where GEMM1 gathers the rows); 16384 tokens,
// 128 experts 67 -> 60 (40); of the 128 tokens of a decode step, 64 experts, 39 -> 24 with 64 MB of weights brought
// into L2 meanwhile.
// A block only waits for blocks of lower index and for its own cluster; the host launches no more
// blocks than the device holds at once.
//
// Selection rules are those of route.cuh / moe/gate.cuh:556-718: softmax over the E real experts, the k
// largest with ties to the lowest id, mCw = sum of the k winning probabilities; tokens whose k-th and
// (k+1)-th logits are closer than fp32 summation error can move them have the experts in that
// distance of the k-th re-evaluated in fp64.
#pragma once

#include <cuda.h>

#include "route.cuh"
#include "tc_common.cuh"

namespace kleos {
namespace route_split {

constexpr int BM = 128, kThreads = 512, kWarps = kThreads / 32, kMaxParts = 4, kMaxStages = 14;

template <int PXT>
struct Shape {
    static constexpr int STAGE_BYTES = BM * 128 + PXT * 128;  // one 128-byte K slice of 128 tokens and of the gate weight
    static constexpr int STAGES = PXT == 64 ? 7 : 4;
    static constexpr int LD = PXT + 4;                          // floats of a row of partial logits
    static constexpr int RECV_BYTES = BM * LD * 4;              // [parts][128 / parts][LD]
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + RECV_BYTES + 1024 + 8192;  // 8192: Control
};

struct Args {
    RouteArgs r;               // refine_* unused; col_partial [S * parts / 128][PX]
    PlaceArgs place;           // slots, counts and, on one rank, the rows' way into the cells
    DeviceStatus* status;
    const char* ahead;         // expert weights to bring into L2 while the memory is idle, or null
    size_t ahead_bytes;        // ... a multiple of 16
    int own;                   // layers: tokens per block, 32, 64 or 128
    int parts;                 // kFine: blocks per cluster
    // kFine: K slices that one accumulator sums before the next one takes over.  When tensor memory is full of
    // accumulators they are read, and the first ones start again.
    int acc_slices;
    int withhold;              // kFine, test hook: a cluster's first block keeps its partial logits, so that the others' waits run out
};

struct Control {
    unsigned long long full[kMaxStages], empty[kMaxStages], acc_full;  // acc_full: once per filling of tensor memory
    unsigned long long acc_read;                       // a filling's accumulators have been read, eight warps
    unsigned long long got;                            // the other blocks' parts of this block's logits have arrived
    uint32_t tmem_base;
    int abort;
    unsigned launch;                                   // PlaceArgs::launch[0]
    __align__(16) float bias[128];
    int hist[128];
    int top[BM * kMaxTopK];                            // chosen experts of this block's tokens
};
// Lies over the operand stages, which are free once the block's accumulator is complete.
struct Scratch {
    PlaceScratch place;
    float sel_v[BM][kMaxTopK + 1];                     // the K + 1 largest logits of every token
    int sel_i[BM][kMaxTopK + 1];
    double band_v[kWarps][128];                        // per warp, for the near-tie re-evaluation: fp64 logits
    short band_id[kWarps][128];                        // and ids of the experts near the k-th logit
};

constexpr int kSendAt = 63488;  // partial logits on their way out lie behind Scratch in the operand stages

// shared memory -> another block's shared memory, completing on that block's mbarrier
__device__ __forceinline__ void bulk_to_block(uint32_t dst_cluster, uint32_t src, uint32_t bytes, uint32_t bar_cluster) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst_cluster), "r"(src), "r"(bytes), "r"(bar_cluster)
                 : "memory");
}

// a + b - fl(a + b), exactly (Knuth's two-sum); 0 beside a sum that is not finite
__device__ __forceinline__ float add_rest(float a, float b) {
    const float s = a + b, t = s - a;
    return fabsf(s) < INFINITY ? (a - (s - t)) + (b - t) : 0.f;
}

// fp64 dot product of a token row and a gate-weight row, by the whole warp
template <typename TE>
__device__ __forceinline__ double dot64(const TE* x, const TE* w, int H, int lane) {
    constexpr int VEC = 16 / (int)sizeof(TE);
    double s = 0.0;
#pragma unroll 4
    for (int h = lane * VEC; h < H; h += 32 * VEC) {
        const uint4 xr = *reinterpret_cast<const uint4*>(x + h), wr = *reinterpret_cast<const uint4*>(w + h);
        const TE* xv = reinterpret_cast<const TE*>(&xr);
        const TE* wv = reinterpret_cast<const TE*>(&wr);
#pragma unroll
        for (int q = 0; q < VEC; ++q) s += (double)Elem<TE>::to_f(xv[q]) * (double)Elem<TE>::to_f(wv[q]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Near-ties, by a whole warp (eight tokens, four lanes each; rare, so it stays out of line): the experts
// within eps of the k-th logit are re-evaluated in fp64 and the open places of the top-k are filled from
// them (larger value first, equal values to the lower id).  Experts further above are in the set and
// experts further below are out of it whatever the summation order.  keep64: the band's logits are replaced by
// the fp64 ones, from which the probabilities and mCw then come (kleos_route_static and 16-bit training layers; 16-bit
// inference gives the bits of the persistent kernel, and TF32 layers keep the fp32 logits' too).
template <typename TE>
__device__ __noinline__ void settle_near_ties(unsigned flagged, float* logits, int ld, int E, int K, float kth, float eps,
                                              const TE* A, int t, const TE* Wg, int H, const float* bias, Scratch* scr,
                                              int tok, bool keep64) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    short* band_id = scr->band_id[warp];
    double* band_v = scr->band_v[warp];
    while (flagged) {
        const int src = __ffs(flagged) - 1;  // first lane of the token's four
        flagged &= flagged - 1;
        const float kth_s = __shfl_sync(0xffffffffu, kth, src), eps_s = __shfl_sync(0xffffffffu, eps, src);
        const int tok_s = __shfl_sync(0xffffffffu, tok, src), t_s = __shfl_sync(0xffffffffu, t, src);
        float* l = logits + (size_t)tok_s * ld;
        int nb = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const unsigned in = __ballot_sync(0xffffffffu, e0 + lane < E && fabsf(l[e0 + lane] - kth_s) <= eps_s);
            if ((in >> lane) & 1u) band_id[nb + __popc(in & ((1u << lane) - 1u))] = (short)(e0 + lane);
            nb += __popc(in);
        }
        __syncwarp();
        for (int b = 0; b < nb; ++b) {
            const int e = band_id[b];
            const double dot = dot64<TE>(A + (size_t)t_s * H, Wg + (size_t)e * H, H, lane);
            if (lane == 0) {
                band_v[b] = dot + (double)bias[e];
                if (keep64) l[e] = (float)band_v[b];
            }
        }
        __syncwarp();
        if (lane == 0) {
            // Chosen without doubt: the same subtraction as above, so that every chosen expert is either here or in
            // the band.  (kth + eps rounds to another value: an expert at 1.0001f with kth = 1 was in neither.)
            int c_in = 0;
            for (int j = 0; j < K; ++j) c_in += scr->sel_v[tok_s][j] - kth_s > eps_s;
            for (int j = c_in; j < K; ++j) {
                int best = -1;
                for (int b = 0; b < nb; ++b) {
                    if (band_id[b] < 0) continue;
                    if (best < 0 || band_v[b] > band_v[best]) best = b;  // (ids ascend)
                }
                if (best < 0) break;  // (the band holds every open place's expert)
                scr->sel_i[tok_s][j] = band_id[best];
                scr->sel_v[tok_s][j] = l[band_id[best]];
                band_id[best] = -1;
            }
        }
        __syncwarp();
    }
}

}  // namespace route_split

// PXT: padded expert count; KT: compile-time top-k (0: read it from the arguments); kFine: kleos_route_static, whose
// mCw is a 32-bit result: Args::acc_slices, compensated sums (a layer's router sums a block's slices in one accumulator: the
// code for more cost 256 tokens 0.6 of 30 us).
template <typename TE, int PXT, int KT, bool kFine = false>
__global__ void __launch_bounds__(route_split::kThreads, 1)
route_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_wg, route_split::Args a) {
    using namespace tc;
    using namespace route_split;
    using Sh = Shape<PXT>;
    constexpr int STAGES = Sh::STAGES, LD = Sh::LD, PER = PXT / 4;  // experts per thread
    constexpr int KC = KT > 0 ? KT : kMaxTopK;
    static_assert(sizeof(Control) <= 8192 && sizeof(Scratch) <= kSendAt && kSendAt + Sh::RECV_BYTES <= STAGES * Sh::STAGE_BYTES, "shared memory set aside");
    constexpr bool kWide = sizeof(TE) == 4;            // tf32: fp32 words
    constexpr bool kSplit = kWide || kFine;            // K split over a cluster
    constexpr int BKE = 128 / (int)sizeof(TE);         // elements per K slice
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    float* recv = reinterpret_cast<float*>(tiles + STAGES * Sh::STAGE_BYTES);
    Control* ctl = reinterpret_cast<Control*>(reinterpret_cast<uint8_t*>(recv) + Sh::RECV_BYTES);
    Scratch* scr = reinterpret_cast<Scratch*>(tiles);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // own: tokens this block decides on, all alone or (kSplit) after its part of K for the 128 of its cluster
    const int C = kSplit ? a.parts : 1, me = kSplit ? (int)cluster_ctarank() : 0, own = a.own;
    const uint32_t rows = kSplit ? BM : own;           // token rows of a K slice
    const uint32_t stage_bytes = rows * 128 + PXT * 128;
    const int stages = min(kMaxStages, (int)(STAGES * Sh::STAGE_BYTES / stage_bytes));
    const int S = a.r.S, E = a.r.E, H = a.r.H, K = KT > 0 ? KT : a.r.K;
    const long long wait_cycles = a.place.wait_cycles;
    const uint32_t epoch = a.place.epoch;
    volatile int* abort_flag = &ctl->abort;
    const uint32_t tmem_cols = kFine ? 512u : (uint32_t)PXT;
    uint32_t idesc;
    if constexpr (kWide) idesc = make_instr_desc_tf32(BM, PXT);
    else idesc = make_instr_desc_16b(BM, PXT, Pack2<TE>::kMmaFormat);

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&ctl->full[s], 1);
            mbar_init(&ctl->empty[s], 1);
        }
        mbar_init(&ctl->acc_full, 1);
        mbar_init(&ctl->acc_read, 8);
        mbar_init(&ctl->got, 1);
        ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&ctl->tmem_base)), "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    pdl_trigger();
    if (tid < 128) ctl->bias[tid] = tid < E ? a.r.bias[tid] : 0.f;
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the cluster's blocks all run before anyone stores into their shared memory
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    if (tid == 64 && a.place.slots != nullptr) ctl->launch = ld_relaxed_u32(a.place.launch);  // (read after later barriers)

    const int KS = H / BKE, kb0 = me * KS / C, kb1 = (me + 1) * KS / C;  // this block's part of K
    const int n_rt = (S + (int)rows - 1) / (int)rows, n_clusters = (int)gridDim.x / C, cluster_id = (int)blockIdx.x / C;
    const int acc_slices = kFine ? a.acc_slices : KS, n_acc = kFine ? (kb1 - kb0 + acc_slices - 1) / acc_slices : 1;
    constexpr int kAccs = 512 / PXT, kSums = kFine ? PXT / 2 : 1;
    const int fills = kFine ? (n_acc + kAccs - 1) / kAccs : 1;
    const uint32_t part_bytes = (uint32_t)own * LD * 4;
    const TE* A = static_cast<const TE*>(a.r.A);
    const TE* Wg = static_cast<const TE*>(a.r.Wg);
    // Until the first expert GEMM starts there is little to load beside the gate's operands: meanwhile every
    // block brings its share of the first expert weights into L2, blocks with tokens once their operands
    // are here.
    auto bring_ahead = [&]() {
        const size_t share = ((a.ahead_bytes / 16 + gridDim.x - 1) / gridDim.x) * 16, from = blockIdx.x * share;
        for (size_t o = from; o < from + share && o < a.ahead_bytes; o += 16384)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;"
                         ::"l"(a.ahead + o), "r"((uint32_t)min(min((size_t)16384, from + share - o), a.ahead_bytes - o))
                         : "memory");
    };
    if (tid == 96 && a.ahead != nullptr && cluster_id >= n_rt) bring_ahead();
    uint32_t round = 0, s = 0, ph = 0;  // s, ph: stage and parity of the producer, and of the MMA issuer
    for (int rt = cluster_id; rt < n_rt; rt += n_clusters, ++round) {
        if (tid < PXT) ctl->hist[tid] = 0;
        if (tid == 0 && C > 1) mbar_expect_tx(&ctl->got, (uint32_t)(C - 1) * part_bytes);
        // (after a failed wait the block still runs through its barriers, with the abort flag up, so that
        // the blocks of a cluster meet at the same ones)
        if (warp == 0) {
            if (lane == 0 && !*abort_flag) {
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(&ctl->empty[s], ph ^ 1, wait_cycles, abort_flag)) {
                        report_error(a.status, KLEOS_AT_GEMM_PRODUCER, -100 - rt, (int)epoch);
                        *abort_flag = 1;
                        break;
                    }
                    mbar_expect_tx(&ctl->full[s], stage_bytes);
                    uint8_t* sa = tiles + s * stage_bytes;
                    tma_load_2d(sa, &map_a, kb * BKE, rt * (int)rows, &ctl->full[s]);
                    tma_load_2d(sa + rows * 128, &map_wg, kb * BKE, 0, &ctl->full[s]);
                    if (++s == (uint32_t)stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            __syncwarp();
        } else if (warp == 1) {
            if (lane == 0 && !*abort_flag) {
                bool ok = true;
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(&ctl->full[s], ph, wait_cycles, abort_flag)) {
                        report_error(a.status, KLEOS_AT_GEMM_MMA, -100 - rt, (int)epoch);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    // (the instruction has 128 token rows; those after `rows` are whatever lies there, and so are their logits)
                    const uint32_t sa = smem_u32(tiles + s * stage_bytes);
                    const uint64_t da = make_smem_desc(sa), db = make_smem_desc(sa + rows * 128);
                    const int acc = kFine ? (kb - kb0) / acc_slices : 0;
                    const bool first = kb - kb0 == acc * acc_slices;
                    const uint32_t d = tmem_base + (uint32_t)(acc % kAccs * PXT);
                    if (kFine && first && acc > 0 && acc % kAccs == 0) {
                        umma_commit(&ctl->acc_full);
                        if (!mbar_wait(&ctl->acc_read, (round * (fills - 1) + acc / kAccs - 1) & 1, wait_cycles, abort_flag)) {
                            report_error(a.status, KLEOS_AT_GEMM_MMA, -300 - rt, (int)epoch);
                            *abort_flag = 1;
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {  // four 32-byte steps per slice
                        if constexpr (kWide) umma_tf32(d, da + 2 * k, db + 2 * k, idesc, (!first || k != 0) ? 1u : 0u);
                        else umma_bf16(d, da + 2 * k, db + 2 * k, idesc, (!first || k != 0) ? 1u : 0u);
                    }
                    umma_commit(&ctl->empty[s]);
                    if (++s == (uint32_t)stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (ok) umma_commit(&ctl->acc_full);
            }
            __syncwarp();
        }
        if (tid == 96 && round == 0 && a.ahead != nullptr && mbar_wait(&ctl->acc_full, 0, wait_cycles, abort_flag)) bring_ahead();
        __syncwarp();
        // ---------------------------------------------------------- logits, or partial ones to the blocks that own the tokens
        if (warp >= 4 && warp < 12) {
            const int q = warp & 3, half = (warp - 4) >> 2;
            const int row = q * 32 + lane, owner = row / own;
            // the rows of one owner lie one after the other on both sides
            float* dst = (owner == me ? recv + (size_t)me * own * LD : reinterpret_cast<float*>(tiles + kSendAt) + (size_t)owner * own * LD) +
                         (size_t)(row % own) * LD + half * (PXT / 2);
            const uint32_t taddr = tmem_base + half * (PXT / 2) + (static_cast<uint32_t>(q * 32) << 16);
            float sum[kSums];  // of the fillings before the last
#pragma unroll
            for (int j = 0; j < kSums; ++j) sum[j] = 0.f;
            bool ok = true;
#pragma unroll 1
            for (int f = 0; f < fills; ++f) {
                ok = mbar_wait(&ctl->acc_full, (round * fills + f) & 1, wait_cycles, abort_flag);
                if (!ok) {
                    if (lane == 0) report_error(a.status, KLEOS_AT_GEMM_EPILOGUE, -100 - rt, (int)epoch);
                    *abort_flag = 1;
                }
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const int accs = min(kAccs, n_acc - f * kAccs);
                // (the operand stages, where the rows on their way out go, are free after the last filling only)
                const bool last = f + 1 == fills;
#pragma unroll (kFine ? PXT / 32 : 1)
                for (int c = 0; c < PXT / 2 && (kSplit || q * 32 < own); c += 16) {
                    uint32_t v[16];
                    tmem_ld_32x16(taddr + c, v);
                    tmem_ld_wait();
#pragma unroll 1
                    for (int acc = 1; acc < accs; ++acc) {
                        uint32_t w[16];
                        tmem_ld_32x16(taddr + acc * PXT + c, w);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
                    }
                    if (kSums > 1) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            sum[(c + j) % kSums] += __uint_as_float(v[j]);
                            v[j] = __float_as_uint(sum[(c + j) % kSums]);
                        }
                    }
                    if (last) {
#pragma unroll
                        for (int j = 0; j < 16; j += 4) *reinterpret_cast<uint4*>(dst + c + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                    }
                }
                if (!last) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctl->acc_read);
                }
            }
            tc_fence_before();
            if (kSplit) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                asm volatile("bar.sync 1, 256;" ::: "memory");
            }
            if (tid == 128 && !*abort_flag && !(kFine && a.withhold && me == 0))
                for (int p = 1; p < C; ++p) {
                    const int to = (me + p) % C;
                    bulk_to_block(map_to_cta(smem_u32(recv + (size_t)me * own * LD), (uint32_t)to),
                                  smem_u32(tiles + kSendAt) + (uint32_t)to * part_bytes, part_bytes,
                                  map_to_cta(smem_u32(&ctl->got), (uint32_t)to));
                }
        }
        __syncthreads();
        if (C > 1 && !mbar_wait(&ctl->got, round & 1, wait_cycles, abort_flag)) {
            if (!*abort_flag) report_error(a.status, KLEOS_AT_GEMM_EPILOGUE, -200 - rt, (int)epoch);
            *abort_flag = 1;
        }
        __syncwarp();
        // ---------------------------------------------------------- softmax and top-k, four threads per token
        // (Loops that are short in code: this runs once per launch, and the time of straight-line code
        // is that of fetching it.  With the four threads' logits in registers and all loops unrolled
        // the step took 4.0 us at 64 experts and 8.5 at 128.)
        const int tok = tid >> 2, sub = tid & 3, tok0 = rt * (int)rows + me * own, t = tok0 + tok;
        if (warp < own / 8) {  // whole warps: eight tokens each
            float* l = recv + (size_t)tok * LD + sub * PER;  // first part of K; the token's logits from here on
            float val[KC + 1];
            int idx[KC + 1];
#pragma unroll
            for (int j = 0; j <= KC; ++j) {
                val[j] = -INFINITY;
                idx[j] = 0x7fffffff;
            }
#pragma unroll 1
            for (int i = 0; i < PER; i += 4) {
                float4 v = *reinterpret_cast<const float4*>(l + i);
#pragma unroll 1
                for (int p = 1; p < C; ++p) {
                    const float4 w = *reinterpret_cast<const float4*>(l + (size_t)p * own * LD + i);
                    v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
                }
                const int e0 = sub * PER + i;
                const float4 b = *reinterpret_cast<const float4*>(ctl->bias + e0);
                float x4[4] = {v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w};
                *reinterpret_cast<float4*>(l + i) = make_float4(x4[0], x4[1], x4[2], x4[3]);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    // insertion into the K + 1 largest; strict '>' keeps the lower id in front
                    float x = e0 + q < E ? x4[q] : -INFINITY;
                    int id = e0 + q;
#pragma unroll
                    for (int j = 0; j <= KC; ++j)
                        if (x > val[j]) {
                            const float tv = val[j];
                            const int ti = idx[j];
                            val[j] = x;
                            idx[j] = id;
                            x = tv;
                            id = ti;
                        }
                }
            }
            // the four threads' lists, merged from the front: equal values to the lower id; a value that
            // compares greater than nothing is never chosen and leaves id 0
            float m = 0.f, kth = 0.f, next = 0.f;
#pragma unroll 1
            for (int j = 0; j <= K; ++j) {
                float bv = val[0];
                int be = idx[0];
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                    const int oe = __shfl_xor_sync(0xffffffffu, be, o);
                    if (ov > bv || (ov == bv && oe < be)) {
                        bv = ov;
                        be = oe;
                    }
                }
                if (be == idx[0]) {  // (ids differ between the threads unless all have none left)
#pragma unroll
                    for (int q = 0; q < KC; ++q) {
                        val[q] = val[q + 1];
                        idx[q] = idx[q + 1];
                    }
                    val[KC] = -INFINITY;
                    idx[KC] = 0x7fffffff;
                }
                if (j == 0) m = bv;
                if (j == K - 1) kth = bv;
                next = bv;
                if (sub == 0) {
                    scr->sel_v[tok][j] = bv;
                    scr->sel_i[tok][j] = be == 0x7fffffff ? 0 : be;
                }
            }
            __syncwarp();
            const float eps = a.r.tie_eps * fmaxf(1.f, fabsf(kth));
            const unsigned flagged = __ballot_sync(0xffffffffu, sub == 0 && t < S && K < E && (kth - next) < eps && !*abort_flag);
            if (flagged)
                settle_near_ties<TE>(flagged, recv, LD, E, K, kth, eps, A, t, Wg, H, ctl->bias, scr, tok,
                                     kFine || (!kWide && a.r.col_partial != nullptr));
            float d = 0.f, d_rest = 0.f;
#pragma unroll 1
            for (int i = 0; i < PER; i += 4) {
                const int e0 = sub * PER + i;
                float4 v = *reinterpret_cast<const float4*>(l + i);
                v.x = e0 < E ? __expf(v.x - m) : 0.f;
                v.y = e0 + 1 < E ? __expf(v.y - m) : 0.f;
                v.z = e0 + 2 < E ? __expf(v.z - m) : 0.f;
                v.w = e0 + 3 < E ? __expf(v.w - m) : 0.f;
                if (kSplit) {
                    const float four = (v.x + v.y) + (v.z + v.w);
                    if (kFine) d_rest += add_rest(d, four);
                    d += four;
                }
                *reinterpret_cast<float4*>(l + i) = v;
            }
            if (kSplit) {
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    const float other = __shfl_xor_sync(0xffffffffu, d, o);
                    if (kFine) d_rest += __shfl_xor_sync(0xffffffffu, d_rest, o) + add_rest(d, other);
                    d += other;
                }
                if (kFine) d += d_rest;  // (mCw is a 32-bit result: its sums and its quotient are rounded once each)
            } else {
                // in the order of the experts, as the persistent kernel adds them
                __syncwarp();
                const float* x = l - sub * PER;
#pragma unroll 4
                for (int i = 0; i < PXT; i += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(x + i);
                    d += v.x; d += v.y; d += v.z; d += v.w;
                }
            }
            const float inv = 1.f / d;
            if (sub == 0 && t < S && !*abort_flag) {
                float w[KC], in_order = 0.f;
#pragma unroll
                for (int j = 0; j < KC; ++j) {
                    w[j] = j < K ? __expf(scr->sel_v[tok][j] - m) : 0.f;
                    if (!kSplit && j < K) in_order = __fmaf_rn(w[j], inv, in_order);
                    if (kWide) w[j] = __fmul_rn(w[j], inv);
                }
                a.r.mcw[t] = kFine ? __fdiv_rn(pair_sum(w), d) : kWide ? pair_sum(w) : in_order;
#pragma unroll 1
                for (int j = 0; j < K; ++j) {
                    const int e = scr->sel_i[tok][j];
                    a.r.topk[(size_t)t * K + j] = e;
                    ctl->top[tok * K + j] = e;
                    atomicAdd(&ctl->hist[e], 1);
                }
            } else if (kFine && sub == 0 && t < S) {
                // no host code asks for a status here: a token whose logits did not come says so itself
                a.r.mcw[t] = __int_as_float(0x7fc00000);
#pragma unroll 1
                for (int j = 0; j < K; ++j) a.r.topk[(size_t)t * K + j] = -1;
            }
            // probabilities, padding columns zero
            TE* dst = static_cast<TE*>(a.r.probs) + (size_t)t * PXT + sub * PER;
            constexpr int VEC = 16 / (int)sizeof(TE);
            const bool aligned = (reinterpret_cast<uintptr_t>(a.r.probs) & 15) == 0;  // (a caller's pointer)
#pragma unroll 1
            for (int i = 0; i < PER; i += VEC) {
                float p[VEC];
#pragma unroll
                for (int q = 0; q < VEC; q += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(l + i + q);
                    p[q] = v.x; p[q + 1] = v.y; p[q + 2] = v.z; p[q + 3] = v.w;
                }
                uint32_t packed[4];
#pragma unroll
                for (int q = 0; q < VEC; ++q) p[q] = sub * PER + i + q < E ? p[q] * inv : 0.f;
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    if constexpr (kWide) {
                        packed[h] = __float_as_uint(round_tf32(p[h]));
                    } else {
                        const auto two = Pack2<TE>::from_f2(p[2 * h], p[2 * h + 1]);
                        packed[h] = *reinterpret_cast<const uint32_t*>(&two);
                    }
                }
                if (t < S && !*abort_flag) {
                    if (aligned) {
                        *reinterpret_cast<uint4*>(dst + i) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                    } else {
#pragma unroll
                        for (int q = 0; q < VEC; ++q) dst[i + q] = Elem<TE>::from_f(p[q]);
                    }
                }
                if (a.r.col_partial != nullptr) {
#pragma unroll
                    for (int q = 0; q < VEC; ++q) l[i + q] = p[q];  // for the column sums
                }
            }
        }
        __syncthreads();
        const int row = rt * C + me;  // block of `own` tokens this block decides on
        if (a.r.col_partial != nullptr && tid >= 128 && tid < 128 + PXT && !*abort_flag) {
            float sum = 0.f;
            for (int i = 0; i < own; ++i) sum += recv[(size_t)i * LD + tid - 128];
            a.r.col_partial[(size_t)row * PXT + tid - 128] = sum;
        }
        if (a.place.slots != nullptr)
            place_tokens(a.place, ctl->launch, row, n_rt * C, tok0, own, ctl->top, ctl->hist, &scr->place, abort_flag, a.status);
        if (rt + n_clusters < n_rt) {
            // another round: every block of the cluster is done with the partial logits it received, and the
            // operand stages are handed back to the TMA
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            cluster_sync_all();
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) settle_after_abort();
    cluster_sync_all();
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(tmem_cols)
                     : "memory");
    }
}

}  // namespace kleos
