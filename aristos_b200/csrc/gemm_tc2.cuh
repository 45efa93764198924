// Expert-FFN GEMM with paired blocks (tcgen05 cta_group::2), weight rows on the MMA's M side and token
// rows on its N side: a cluster of two blocks on neighbouring SMs computes 256 output columns of up to
// 288 rows of one local expert.  M is fixed at 256 by the instruction and an FFN has hundreds or
// thousands of columns; the rows an expert gets are any number, and N takes any multiple of 32.  So
// the work done for padding is below 32 rows of an expert, and an expert's weights are read once for
// every 256 or 288 of its rows.  With the rows on M, 128 a block, every tile cost as much as one of 256 rows.
// (That is with one source rank.  With several, a tile is two panels of up to 128 rows of one or two sources, and takes
// twice the rows of the larger one; an expert's odd last panel is one tile, half of which is discarded.)
// What bounds it: the weight stream from HBM up to about 256 rows an expert (128 tokens, 64 experts,
// H = I = 2048: 537 MB of weights in 85 us = 6.3 TB/s, where plain loads reach 6.2; before 106 and 115 us
// a launch), above that the tensor pipe, in steady state at the clock the power limit leaves (4096 tokens,
// H = 4096, I = 14336, 8 experts: 600 us = 1.6 PFLOP/s alone; forwards one after the other take 1520 to 1580, as
// they did with the rows on M).  16384 tokens on 128 experts of Zipf popularity: 135 + 143 us -> 96 + 95.
//
// Tile = (local expert, 256 columns, up to 288 rows).  Each block TMA-loads 128 weight rows (A) and half
// of the token rows (B), 64 wide K slices through a ring of six.  Accumulators are a ring in
// tensor memory, 16 slots of 32 columns: a tile takes as many as its rows need, and the next tile's
// follow, so that the read-back of one tile runs beside the main loop of the next whatever their sizes.
// A tile of more than 256 rows, or one whose slots wrap around, is two instructions per K step.
// No load is multicast: every block fetches exactly the bytes it keeps.
//
// Tiles are claimed from a global counter, one ahead, and handed to all roles of both blocks through a
// ring in shared memory: their sizes differ by up to nine times, so no fixed split is even.
//
// Per block, 384 threads:
//   warp 0      TMA producer of the token rows (one lane)
//   warp 1      leader only: issues tcgen05.mma.cta_group::2, commits to `empty` and
//               `acc_full` of BOTH blocks
//   warp 2      tensor-memory allocation / release (both blocks, cta_group::2 forms); in the leader
//               also the scheduler, which claims the tiles
//   warp 3      TMA producer of the weight rows (one lane)
//   warps 4..11 read-back of the block's 128 columns of all the tile's rows: two groups of four warps,
//               16 rows at a time in turn; arrive on the LEADER's `slot_empty`
//   warps 12..15  gathering form only: token rows by index
// Work and epilogue semantics follow the reference's tile worker (os/processor/processor.cuh:
// 350-489,706-741).  Every wait is bounded.  This kernel runs one GEMM over rows whose places are
// known when it starts: those of each expert by count (one source rank, and the dense single-expert layer, whose
// rows are all of one expert), or a list of panels (several ranks).
//
// Element types: bf16, fp16, and TF32 words (kind::tf32, torch_dtype 1; the reference's mma.sync
// m16n8k8 block GEMM, os/processor/mmaConfig.cuh:73-81).  A K slice is 128 bytes of a row and four
// instructions in either case: 64 16-bit or 32 4-byte elements.
#pragma once

#include <cuda.h>

#include "gemm_common.cuh"
#include "tc_common.cuh"

namespace kleos {
namespace gemm_tc2 {

constexpr int BM = 128;                             // output columns (weight rows) per block
constexpr int kMaxHalf = 144;                       // token rows per block, a multiple of 16
constexpr int kMaxRows = 2 * kMaxHalf;              // ... per tile
constexpr int kSlices = 6;                          // K slices of shared memory
constexpr int W_BYTES = BM * 128;                   // one K slice of the weight rows
constexpr int SLICE_BYTES = W_BYTES + kMaxHalf * 128;
constexpr int kSteps = 4;                           // instructions per K slice, 32 bytes of a row each
constexpr int kBackWarps = 8, kThreads = (4 + kBackWarps) * 32;
constexpr int kGatherWarps = 4;
template <bool kGather> constexpr int kBlock = kThreads + (kGather ? kGatherWarps * 32 : 0);
constexpr int TMEM_COLS = 512, kSlotCols = 32, kSlots = TMEM_COLS / kSlotCols;
// tiles on their way: at most six in the K ring, two ahead of it, sixteen in tensor memory
constexpr int kTasks = 32;
constexpr int STG_ROW = BM * 2 + 16;                // bytes of a staged row: padded, so that eight rows meet no bank conflict
constexpr int kCtlBytes = 22528;
constexpr int SMEM_BYTES = kSlices * SLICE_BYTES + 1024 + kCtlBytes;
static_assert(SMEM_BYTES <= 232448, "227 KiB of shared memory per block");
static_assert(SLICE_BYTES % 1024 == 0, "the swizzle repeats every 1024 bytes");

// Token rows as boxes, 128 bytes wide, of the heights below: a K slice of a tile is one copy, of the lowest box
// that holds the block's rows.  (Made up of boxes of 32 and 16 rows, 96 rows took three copies a slice, and
// a layer of 384 rows and K = 8192 ran 0.72 times as fast as with one of 128.)
constexpr int kBoxes = 6;
struct RowMaps {
    CUtensorMap box[kBoxes];
};
__host__ __device__ constexpr int box_rows(int i) { return i == 0 ? 16 : i == 1 ? 32 : i == 2 ? 64 : i == 3 ? 96 : i == 4 ? 128 : kMaxHalf; }
__device__ __forceinline__ int box_of(int rows) {
    int i = 0;
    while (box_rows(i) < rows) ++i;
    return i;
}

// A tile, as the scheduler hands it to the other roles.  Block r of the pair loads rows[r] token rows from
// row_base[r] on; `half` of them, a multiple of 16, go into the MMA from each block.
constexpr int kReadOnce = 1 << 16;
struct __align__(16) Task {
    int half;          // 0: no more tiles
    int le, mt;        // local expert, 256-column tile
    int src;           // source ranks, eight bits each, and kReadOnce when no other tile reads these weights
    int row_base[2], rows[2];
};

struct Control {
    unsigned long long full[kSlices];    // used on the leader
    unsigned long long empty[kSlices];   // one per block
    unsigned long long acc_full[kSlots];     // one per block, tile i uses [i % kSlots]
    unsigned long long slot_empty[kSlots];   // used on the leader, 16 arrivals (8 warps x 2 blocks)
    unsigned long long task_full[kTasks];    // one per block
    unsigned long long begun[2];             // leader: the loads of tile i have begun, [i % 2]
    uint32_t tmem_base;
    int abort;
    bool last_block;
    Task task[kTasks];
    int rows[256];        // contiguous: rows of every local expert
    int splits[256];      // tiles along the rows of every local expert
    int first[257];       // tiles before every local expert
    __align__(16) unsigned char stage[2][2][16 * STG_ROW];  // per read-back group, two turns: 16 rows x 256 bytes
};
static_assert(sizeof(Control) <= kCtlBytes, "control block must fit the shared memory set aside for it");
constexpr int kBarriers = offsetof(Control, tmem_base) / 8;
static_assert(kBarriers <= kThreads, "a thread per barrier");

// Tiles along the rows of an expert.  A K slice of a tile of n rows takes the larger of 2 n cycles of the
// tensor pipe and n + 256 of shared memory (32 KiB + 128 n bytes of operand reads and TMA writes);
// one of more than 256 rows is two instructions a step, which read the weights twice: 672 cycles at 288
// rows.  So 257 to 288 rows are best taken as one tile, and more of them 256 at a time.
__device__ __forceinline__ int row_splits(int rows) {
    return rows <= kMaxRows ? (rows + kMaxRows - 1) / kMaxRows : (rows + 255) / 256;
}
// A dense layer is one expert, so its tiles are all alike and take whole rounds over the block pairs: as many
// (and as small) ones as fit the same number of rounds.  (Of several experts' tiles a pair that is done
// early takes another.)
__device__ __forceinline__ int dense_splits(int rows, int column_tiles, int pairs) {
    const int least = row_splits(rows), rounds = (least * column_tiles + pairs - 1) / pairs;
    return max(least, min(rounds * pairs / column_tiles, (rows + 31) >> 5));
}

// Tiles in order of local expert, column tile, rows: tiles that run together read the same weights.
// `le` is the caller's place in the list (its tiles only grow).
__device__ __forceinline__ Task decode_task(int t, const Control* ctl, const GemmArgs& g, int* le) {
    int e = *le;
    while (ctl->first[e + 1] <= t) ++e;
    *le = e;
    const int splits = ctl->splits[e], r = t - ctl->first[e];
    Task x;
    x.le = e;
    x.mt = r / splits;
    const int j = r - x.mt * splits;
    if (g.contiguous) {
        // 32 rows are the unit, and the tiles of an expert differ by one at most
        const int rows = ctl->rows[e], units = (rows + 31) >> 5, share = units / splits, more = units - share * splits;
        const int at = j * share + min(j, more), n = share + (j < more ? 1 : 0);
        const int left = min(32 * n, rows - 32 * at);
        x.half = 16 * n;
        x.row_base[0] = e * g.pEC + 32 * at;
        x.rows[0] = min(x.half, left);
        x.row_base[1] = x.row_base[0] + x.half;
        x.rows[1] = left - x.rows[0];
        x.src = g.rank | (g.rank << 8);
    } else {
        const int p0 = g.le_start[e] + 2 * j;
        const bool second = p0 + 1 < g.le_start[e + 1];
        const PanelEntry a = g.panels[p0], b = g.panels[second ? p0 + 1 : p0];
        x.row_base[0] = a.row_base;
        x.row_base[1] = b.row_base;  // (without a second panel its block re-reads the first one and discards)
        x.rows[0] = a.rows;
        x.rows[1] = second ? b.rows : 0;
        x.src = a.src | (b.src << 8);
        x.half = (max(x.rows[0], x.rows[1]) + 15) >> 4 << 4;
    }
    if (splits == 1) x.src |= kReadOnce;
    return x;
}

// The slots of a tile that starts at ring position `at`: as one run, or as two when they wrap around or
// are more than the 256 columns of an instruction.
struct Runs {
    int n0, n1;       // slots
    int slot0, slot1;
    __device__ __forceinline__ Runs(uint32_t at, int half) {
        const int n = half >> 4, room = kSlots - (int)(at % kSlots);
        slot0 = (int)(at % kSlots);
        n0 = n > room ? room : n > 8 ? (n + 1) >> 1 : n;
        n1 = n - n0;
        slot1 = (slot0 + n0) % kSlots;
    }
};

template <typename TE>
__host__ __device__ constexpr uint32_t instr_desc() {  // N = 0
    if constexpr (sizeof(TE) == 4) return tc::make_instr_desc_tf32(2 * BM, 0);
    else return tc::make_instr_desc_16b(2 * BM, 0, Pack2<TE>::kMmaFormat);
}

// 16 lanes x 16 columns as two 16 x 8 fragments: register 4 x + 2 h + i of thread t is lane t / 4 + 8 h,
// column 8 x + 2 (t % 4) + i
__device__ __forceinline__ void tmem_ld_16x256_x2(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
// Four 8 x 8 blocks of 16-bit elements, transposed: thread 8 i + j gives the address of column j of block i.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t* r) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(unsigned long long* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(tc::smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Whether all 128 threads that meet at the barrier say yes.
__device__ __forceinline__ bool all_of_group(bool yes, int barrier) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %1, 0;\n\t"
        "bar.red.and.pred q, %2, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"((uint32_t)yes), "r"(barrier)
        : "memory");
    return all != 0;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t cluster_addr, uint4 v) {
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}
// An arrival that announces nothing in memory: the tensor-memory reads before it have completed (tcgen05.wait::ld).
// With release semantics it would wait for the thread's result rows on their way to global memory.
__device__ __forceinline__ void arrive_relaxed(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

}  // namespace gemm_tc2

// kEpi selects the fused epilogue at compile time (0: bias + ReLU, 1: bias + GELU, 2: bias only)
// so the read-back loop stays a short straight-line sequence.
// (Six stages of one K slice: three of two slices, with half the barrier round trips, took 1516 us instead of 1505
// on the layer of 4096 tokens, H = 4096, I = 14336, 8 experts, and 65.3 instead of 64.3 on the dense layer of
// 4096 tokens, H = I = 2048.)
// kGather: the token rows are fetched from the activations by token index, four rows a copy, instead of from
// the cells, so that on one rank nobody copies them there (a layer of 8192 tokens, k = 2, 4 KiB rows: 13 us
// of the router's 43, and 64 MB written and read back).  Four warps issue the copies: 128 rows take 0.33 us,
// which a weight stream from HBM hides (0.4 us a slice) and the tensor pipe at 256 rows a tile does not
// (0.26 us); one warp took 1.06.  Up to 256 rows an expert it pays all the same, by what the router then does not copy:
// see State::gather.
template <typename TE, int kEpi, bool kGather>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(gemm_tc2::kBlock<kGather>, 1)
ffn_gemm_tc2(const __grid_constant__ gemm_tc2::RowMaps map_x, const __grid_constant__ CUtensorMap map_w, GemmArgs g) {
    using namespace tc;
    using namespace gemm_tc2;
    constexpr bool kWide = sizeof(TE) == 4;           // TF32
    constexpr int BKE = 128 / (int)sizeof(TE);        // elements of a K slice
    const long long t_kernel = clock64();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    Control* ctl = reinterpret_cast<Control*>(tiles + kSlices * SLICE_BYTES);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t cta_rank = cluster_ctarank();
    const bool leader = cta_rank == 0;
    volatile int* abort_flag = &ctl->abort;

    if (tid < kBarriers) {  // one each: they lie one after the other at the start of Control
        const int first_slot = (int)(offsetof(Control, slot_empty) / 8);
        mbar_init(reinterpret_cast<unsigned long long*>(ctl) + tid, tid >= first_slot && tid < first_slot + kSlots ? 2 * kBackWarps : 1);
        if (tid == 0) ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&ctl->tmem_base)), "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    // What the second GEMM of a forward needs to know of the plan was written before the first one began
    // (whose blocks let this launch start only once they had waited for it), and no kernel writes the
    // weights: its first weight slices are on their way before the first GEMM has ended.
    if (!g.plan_ready) pdl_wait();
    const int MT = (g.N + 2 * BM - 1) / (2 * BM);
    for (int e = tid; e < g.nLx; e += kBlock<kGather>) {
        const bool in = e >= g.le_begin && e < g.le_end;
        if (g.contiguous) {
            ctl->rows[e] = !in ? 0 : g.counts ? (int)min(g.counts[e], (unsigned)g.EC) : g.pEC;
            ctl->splits[e] = g.counts ? row_splits(ctl->rows[e]) : dense_splits(ctl->rows[e], MT, (int)gridDim.x >> 1);
        } else {
            ctl->splits[e] = in ? (g.le_start[e + 1] - g.le_start[e] + 1) >> 1 : 0;
        }
    }
    __syncthreads();
    const int n_clusters = (int)gridDim.x >> 1, cluster_id = blockIdx.x >> 1;
    if (warp == 0) {
        warp_scan([&](int e) { return ctl->splits[e] * MT; }, ctl->first, g.nLx);
        __syncwarp();
        // the pair's first tile needs no claim: each block decodes it for itself
        if (lane == 0) {
            int le = 0;
            Task x{};
            if (cluster_id < ctl->first[g.nLx]) x = decode_task(cluster_id, ctl, g, &le);
            ctl->task[0] = x;
        }
    }
    __syncwarp();
    tc_fence_before();
    cluster_sync_all();  // (a barrier of both blocks; their mbarriers exist before anything remote touches them)
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    if (g.stats && tid == 0) g.stats[blockIdx.x * kStatSlots + 8] = clock64() - t_kernel;
    if (warp != 3 || !g.plan_ready) pdl_wait();
    if (warp == 0) pdl_trigger();

    const int KS = g.Kd / BKE;                // K slices

    // Tile i of this pair.  The ring needs no "empty" signal, see kTasks.  After a failed wait: no more tiles.
    auto take = [&](uint32_t i, int where) -> Task {
        if (i == 0) return ctl->task[0];
        unsigned long long* bar = &ctl->task_full[(i - 1) % kTasks];
        const uint32_t parity = ((i - 1) / kTasks) & 1u;
        bool ok = try_wait_cluster(bar, parity);
        if (!ok) {
            const long long t0 = clock64();
            uint32_t polls = 0;
            while (!(ok = try_wait_cluster(bar, parity))) {
                __nanosleep(40);
                if ((++polls & 31u) == 0) {
                    if (*abort_flag) break;
                    if (clock64() - t0 > g.wait_cycles) {
                        report_error(g.status, where, -2 - (int)i, (int)g.epoch);
                        *abort_flag = 1;
                        break;
                    }
                }
            }
        }
        Task x = ctl->task[i % kTasks];
        if (!ok) x.half = 0;
        return x;
    };

    if (warp == 0) {
        // ------------------------------------------------------------ token rows (both blocks)
        if (lane == 0) {
            asm volatile("fence.proxy.async;" ::: "memory");
            uint32_t it = 0;
            long long w_empty = 0;
            const long long t_begin = clock64();
            for (uint32_t i = 0;; ++i) {
                const Task x = take(i, KLEOS_AT_GEMM_PRODUCER);
                if (x.half == 0) break;
                if (leader) mbar_arrive(&ctl->begun[i & 1]);
                const int row = leader ? x.row_base[0] : x.row_base[1];
                const int box = kGather ? 0 : box_of(x.half);
                const CUtensorMap* map = &map_x.box[box];
                const uint32_t bytes = 2u * (uint32_t)(W_BYTES + (kGather ? x.half : box_rows(box)) * 128);
                bool ok = true;
                for (int kb = 0; kb < KS; ++kb, ++it) {
                    const int s = it % kSlices;
                    const uint32_t ph = (it / kSlices) & 1;
                    if (!mbar_wait_timed(&ctl->empty[s], ph ^ 1, g.wait_cycles, abort_flag, &w_empty)) {
                        report_error(g.status, KLEOS_AT_GEMM_PRODUCER, (int)i, (int)g.epoch);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    // the leader announces the bytes of both blocks on its own barrier
                    if (leader) mbar_expect_tx(&ctl->full[s], bytes);
                    if (!kGather)
                        tma_load_2d_pair(tiles + s * SLICE_BYTES + W_BYTES, map, kb * BKE, row, map_to_cta(smem_u32(&ctl->full[s]), 0));
                }
                if (!ok) break;
            }
            if (g.stats) {
                g.stats[blockIdx.x * kStatSlots + 0] = w_empty;
                g.stats[blockIdx.x * kStatSlots + 1] = clock64() - t_begin;
            }
        }
        __syncwarp();
    } else if (warp == 3) {
        // ------------------------------------------------------------ weight rows (both blocks)
        // They wait for the same free-stage barrier as the token rows and complete on the same full
        // barrier; the byte count announced by warp 0 covers both, and a slice landing before
        // that announcement only makes the barrier's byte count negative for a moment (the phase
        // cannot complete before warp 0 has arrived).
        if (lane == 0) {
            asm volatile("fence.proxy.async;" ::: "memory");
            uint32_t it = 0;
            long long w_unused = 0;
            // weights that one tile reads leave L2 first, so that the rows between the kernels stay there
            uint64_t stream;
            asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(stream));
            for (uint32_t i = 0;; ++i) {
                const Task x = take(i, KLEOS_AT_GEMM_PRODUCER);
                if (x.half == 0) break;
                // past the last column the block loads its partner's rows again and discards the results
                const int col = x.mt * 2 * BM + (int)cta_rank * BM;
                const int brow = x.le * g.N + (col < g.N ? col : x.mt * 2 * BM);
                bool ok = true;
                for (int kb = 0; kb < KS; ++kb, ++it) {
                    const int s = it % kSlices;
                    const uint32_t ph = (it / kSlices) & 1;
                    if (!mbar_wait_timed(&ctl->empty[s], ph ^ 1, g.wait_cycles, abort_flag, &w_unused)) {
                        ok = false;  // the first producer reports the failure
                        break;
                    }
                    const uint32_t full_leader = map_to_cta(smem_u32(&ctl->full[s]), 0);
                    uint8_t* dst = tiles + s * SLICE_BYTES;
                    if (x.src & kReadOnce) tma_load_2d_pair_hint(dst, &map_w, kb * BKE, brow, full_leader, stream);
                    else tma_load_2d_pair(dst, &map_w, kb * BKE, brow, full_leader);
                }
                if (!ok) break;
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        // ------------------------------------------------------------ scheduler (leader only)
        // Claims a tile when the loads of the tile before it have begun, and hands it, decoded, to
        // all roles of both blocks.
        if (leader && lane == 0 && ctl->task[0].half != 0) {
            const int total = ctl->first[g.nLx];
            int le = 0;
            bool ok = true;
            long long w_unused = 0;
            for (uint32_t i = 1; ok; ++i) {
                ok = mbar_wait_timed(&ctl->begun[(i - 1) & 1], ((i - 1) >> 1) & 1, g.wait_cycles, abort_flag, &w_unused);
                if (!ok) break;  // (the roles report what they wait for)
                const unsigned t = (unsigned)n_clusters + atomicAdd(g.next_tile, 1u);
                Task x{};
                if (t < (unsigned)total) x = decode_task((int)t, ctl, g, &le);
                ctl->task[i % kTasks] = x;
                const uint32_t peer = map_to_cta(smem_u32(&ctl->task[i % kTasks]), 1);
                st_cluster_v4(peer, *reinterpret_cast<const uint4*>(&x));
                st_cluster_v4(peer + 16, *(reinterpret_cast<const uint4*>(&x) + 1));
                const uint32_t bar = smem_u32(&ctl->task_full[(i - 1) % kTasks]);
                mbar_arrive_cluster(map_to_cta(bar, 0));
                mbar_arrive_cluster(map_to_cta(bar, 1));
                ok = x.half != 0;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader only)
        // (the whole warp runs the loop and the elected lane issues, see tc::elect_one)
        if (leader) {
            const uint32_t elected = elect_one();
            const uint32_t slices = smem_u32(tiles), bars = smem_u32(ctl), tmem = (uint32_t)uniform((int)tmem_base);
            uint32_t s = 0, ph = 0, at = 0;
            long long w_acc = 0, w_full = 0;
            const long long t_begin = clock64();
            for (uint32_t i = 0;; ++i) {
                const int half = uniform(take(i, KLEOS_AT_GEMM_MMA).half);
                if (half == 0) break;
                const Runs runs(at, half);
                bool ok = true;
                {
                    // a lane per slot
                    const uint32_t slot = at + (uint32_t)lane;
                    if (lane < runs.n0 + runs.n1)
                        ok = mbar_wait_timed(&ctl->slot_empty[slot % kSlots], ((slot / kSlots) & 1) ^ 1, g.wait_cycles, abort_flag, &w_acc);
                    ok = __all_sync(0xffffffffu, ok);
                }
                if (!ok) {
                    if (lane == 0) report_error(g.status, KLEOS_AT_GEMM_MMA, (int)i, (int)g.epoch);
                    *abort_flag = 1;
                    break;
                }
                at += runs.n0 + runs.n1;
                tc_fence_after();
                // N of a run: 32 columns a slot, 16 rows of each block
                const uint32_t idesc0 = instr_desc<TE>() | ((uint32_t)runs.n0 << 19), idesc1 = instr_desc<TE>() | ((uint32_t)runs.n1 << 19);
                const uint32_t d0 = tmem + runs.slot0 * kSlotCols, d1 = tmem + runs.slot1 * kSlotCols;
                const uint32_t off1 = (uint32_t)runs.n0 * 2048;  // token rows of the second run
                for (int kb = 0; kb < KS; ++kb) {
                    if (!mbar_wait_timed(&ctl->full[s], ph, g.wait_cycles, abort_flag, &w_full)) {
                        if (lane == 0) report_error(g.status, KLEOS_AT_GEMM_MMA, (int)i, (int)g.epoch);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = slices + s * SLICE_BYTES;
                    const uint64_t da = make_smem_desc(sa), db = make_smem_desc(sa + W_BYTES);
                    auto multiply = [&](uint32_t d, uint64_t db_run, uint32_t idesc) {
#pragma unroll
                        for (int k = 0; k < kSteps; ++k) {
                            const uint32_t more = k != 0 ? 1u : (uint32_t)(kb != 0);
                            if constexpr (kWide) umma_tf32_pair_if(elected, d, da + 2 * k, db_run + 2 * k, idesc, more);
                            else umma_bf16_pair_if(elected, d, da + 2 * k, db_run + 2 * k, idesc, more);
                        }
                    };
                    multiply(d0, db, idesc0);
                    if (runs.n1 > 0) multiply(d1, make_smem_desc(sa + W_BYTES + off1), idesc1);
                    // the stage is free in both blocks once these MMAs have read it
                    umma_commit_both_if(elected, bars + (uint32_t)offsetof(Control, empty) + 8 * s);
                    if (++s == kSlices) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (!ok) break;
                umma_commit_both_if(elected, bars + (uint32_t)offsetof(Control, acc_full) + 8 * (i % kSlots));
            }
            if (g.stats && lane == 0) {
                g.stats[blockIdx.x * kStatSlots + 2] = w_acc;
                g.stats[blockIdx.x * kStatSlots + 3] = w_full;
                g.stats[blockIdx.x * kStatSlots + 4] = clock64() - t_begin;
            }
        }
        __syncwarp();
    } else if (kGather && warp >= 4 + kBackWarps) {
        // ------------------------------------------------------------ token rows by index (both blocks)
        // A lane per four rows; warp 0 of the leader announces the bytes.
        asm volatile("fence.proxy.async;" ::: "memory");
        uint32_t it = 0;
        long long w_unused = 0;
        for (uint32_t i = 0;; ++i) {
            const Task x = take(i, KLEOS_AT_GEMM_PRODUCER);
            if (!__all_sync(0xffffffffu, x.half != 0)) break;
            const int per = (x.half / 4 + kGatherWarps - 1) / kGatherWarps, at = 4 * ((warp - 4 - kBackWarps) * per + lane);
            const bool mine = lane < per && at < x.half;
            const int row = (leader ? x.row_base[0] : x.row_base[1]) + at;
            int4 rows = make_int4(0, 0, 0, 0);
            if (mine) rows = *reinterpret_cast<const int4*>(g.row_token + row);  // (past the last row: some earlier forward's tokens)
            bool ok = true;
            for (int kb = 0; kb < KS; ++kb, ++it) {
                const int s = it % kSlices;
                ok = mbar_wait_timed(&ctl->empty[s], ((it / kSlices) & 1) ^ 1, g.wait_cycles, abort_flag, &w_unused);
                if (!__all_sync(0xffffffffu, ok)) break;  // the first producer reports the failure
                if (mine)
                    tma_gather4_pair(tiles + s * SLICE_BYTES + W_BYTES + at * 128, &map_x.box[0], kb * BKE, rows,
                                     map_to_cta(smem_u32(&ctl->full[s]), 0));
                __syncwarp();
            }
            if (!__all_sync(0xffffffffu, ok)) break;
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------ read-back (both blocks)
        // Tensor-memory lane = output column, column = token row.  Group 0 takes the first 16 columns of
        // every slot, group 1 the others; a warp reads the 32 lanes of its quadrant.
        const int q = warp & 3, grp = (warp - 4) >> 2;
        const int tg = tid - 128 - grp * 128;  // thread of the group
        const TE* bias = static_cast<const TE*>(g.bias);
        uint32_t at = 0, turn = 0;
        long long w_accfull = 0;
        const long long t_begin = clock64();
        for (uint32_t i = 0;; ++i) {
            // The warps of a group meet at barriers below, so all of them go on or none: whatever one of
            // them gave up on, they find out here.
            const Task x = take(i, KLEOS_AT_GEMM_EPILOGUE);
            if (!all_of_group(x.half != 0, 1 + grp)) break;
            const Runs runs(at, x.half);
            const int n0 = x.mt * 2 * BM + (int)cta_rank * BM;  // this block's first output column
            // bias of the columns this thread reads back, loaded while the main loop is still running
            float bv[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int n = n0 + q * 32 + (kWide ? lane : 8 * k + (lane >> 2));
                bv[k] = n < g.N && (k == 0 || !kWide) ? Elem<TE>::to_f(bias[(size_t)x.le * g.N + n]) : 0.f;
            }
            TE* obase[2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
                obase[h] = out_ptr<TE>(g, PanelEntry{x.row_base[h], x.rows[h], x.le, (x.src >> (8 * h)) & 0xff}, 0, n0);
            const bool ok = mbar_wait_timed(&ctl->acc_full[i % kSlots], (i / kSlots) & 1, g.wait_cycles, abort_flag, &w_accfull);
            if (!ok) {
                if (lane == 0) report_error(g.status, KLEOS_AT_GEMM_EPILOGUE, (int)i, (int)g.epoch);
                *abort_flag = 1;
            }
            if (!all_of_group(ok, 1 + grp)) break;
            tc_fence_after();
            const int n_slots = runs.n0 + runs.n1;
            // A turn is 16 columns: 16 rows of one block's share.  Two turns' loads are in flight together.
            auto fetch = [&](uint32_t slot, uint32_t* r) {
                const uint32_t taddr = tmem_base + (slot % kSlots) * kSlotCols + grp * 16 + (static_cast<uint32_t>(q * 32) << 16);
                if constexpr (kWide) {
                    tmem_ld_32x16(taddr, r);
                } else {
                    tmem_ld_16x256_x2(taddr, r);
                    tmem_ld_16x256_x2(taddr + (16u << 16), r + 8);
                }
            };
            auto store = [&](int k, const uint32_t* r) {
                const bool run1 = k >= runs.n0;
                const int len = (run1 ? runs.n1 : runs.n0) * 16, off = run1 ? runs.n0 * 16 : 0;
                const int c = (k - (run1 ? runs.n0 : 0)) * kSlotCols + grp * 16;
                const int h = c >= len, r0 = off + c - (h ? len : 0);
                const int valid = min(16, (h ? x.rows[1] : x.rows[0]) - r0);
                if (valid <= 0) return;  // (the same for all warps of the group)
                TE* o = (h ? obase[1] : obase[0]) + (size_t)r0 * g.N;
                auto finish = [&](uint32_t bits, float b) {
                    float v = __uint_as_float(bits) + b;
                    if constexpr (kEpi == 0) v = fmaxf(v, 0.f);
                    else if constexpr (kEpi == 1) v = apply_act(v, 1);
                    return v;
                };
                if constexpr (kWide) {
                    // 32 consecutive columns of a row: one 128-byte line per store instruction
                    if (n0 + q * 32 < g.N) {
                        float* of = reinterpret_cast<float*>(o) + q * 32 + lane;
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (j < valid) of[(size_t)j * g.N] = round_tf32(finish(r[j], bv[0]));
                    }
                } else {
                    // transposed through shared memory: the group's four warps put the block's 128 columns of
                    // 16 rows there, and every store instruction writes 256 bytes of two rows
                    const uint32_t stg = smem_u32(ctl->stage[grp][turn & 1]);
                    ++turn;
#pragma unroll
                    for (int x8 = 0; x8 < 2; ++x8) {
                        uint32_t m[4];
#pragma unroll
                        for (int b = 0; b < 4; ++b) {  // columns 8 b .. 8 b + 7 of the warp's 32
                            const uint32_t* f = r + (b >> 1) * 8 + x8 * 4 + (b & 1) * 2;
                            const auto p = Pack2<TE>::from_f2(finish(f[0], bv[b]), finish(f[1], bv[b]));
                            m[b] = *reinterpret_cast<const uint32_t*>(&p);
                        }
                        stmatrix_x4_trans(stg + (uint32_t)((8 * x8 + (lane & 7)) * STG_ROW + q * 64 + (lane >> 3) * 16), m);
                    }
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
                    const int col = (tg & 15) * 8;
#pragma unroll
                    for (int j = tg >> 4; j < 16; j += 8)
                        if (j < valid && n0 + col < g.N) {
                            uint4 v;
                            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                                         : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                                         : "r"(stg + (uint32_t)(j * STG_ROW + col * 2)));
                            *reinterpret_cast<uint4*>(o + (size_t)j * g.N + col) = v;
                        }
                }
            };
#pragma unroll 1
            for (int k = 0; k < n_slots; k += 2, at += 2) {
                uint32_t r0[16], r1[16];
                const bool two = k + 1 < n_slots;
                fetch(at, r0);
                if (two) fetch(at + 1, r1);
                tmem_ld_wait();
                // this warp's part of the slots is in registers: hand it back to the MMA issuer
                tc_fence_before();
                __syncwarp();
                if (lane < (two ? 2 : 1)) arrive_relaxed(map_to_cta(smem_u32(&ctl->slot_empty[(at + lane) % kSlots]), 0));
                store(k, r0);
                if (two) store(k + 1, r1);
            }
            at -= n_slots & 1;
        }
        if (g.stats && warp == 4 && lane == 0) {
            g.stats[blockIdx.x * kStatSlots + 5] = w_accfull;
            g.stats[blockIdx.x * kStatSlots + 6] = clock64() - t_begin;
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
    // the last pair to finish leaves the counters as it found them
    if (leader && tid == 0 && atomicInc(g.next_tile + 1, (unsigned)n_clusters - 1) == (unsigned)n_clusters - 1) g.next_tile[0] = 0;
    if (g.mode == 1 && g.ret.world > 0) publish_return_flags(g.ret, &ctl->last_block);
}

}  // namespace kleos
