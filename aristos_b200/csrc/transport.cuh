// Token dispatch into the expert ranks' cells, the tile plan built from the arrived counts,
// and the gate-weighted combine of the returned rows.
//
// Roles follow the reference: packet::dispatch (os/packet.cuh:35-286) copies the routed,
// unscaled rows into cell [source rank][local expert] on the expert's rank and raises one
// flag per (source, expert) carrying the routed count, also when the count is zero
// (:240-259); the decoder turns arrived packets into 128-row tasks (:304-398); combine
// (os/processor/processor.cuh:27-205) scales returned rows and accumulates them per token.
// Here every peer is reached with plain 16-byte stores into its mapped cells over NVLink and
// the combine is a deterministic gather-sum instead of element-wise atomics.
#pragma once

#include "common.cuh"

namespace kleos {

// Offsets of the regions inside each rank's symmetric arena (identical on every rank).
struct ArenaLayout {
    size_t xcell;  // [world*nLx][pEC][H] dispatched token rows, by (source rank, local expert)
    size_t ycell;  // [E][pEC][H] returned FFN rows, by global expert
    size_t xflag;  // [world*nLx] u64: (epoch<<32)|routed count, raised when the cell's rows are stored
    size_t cflag;  // [world*nLx] u64: (epoch<<32)|routed count, raised as soon as the count is known
    size_t yflag;  // [world] u64: (epoch<<32)|1 when that expert rank has returned everything
    size_t ypflag; // [E][pEC/128] u64: (epoch<<32)|1 when that 128-row panel of results has arrived
    size_t bytes;
};

struct DispatchArgs {
    const void* A;             // [S,H]
    const int* cell_tokens;    // [E,pEC]
    const unsigned* counts;    // [E]
    PeerTable peers;
    ArenaLayout lay;
    unsigned* done_counter;    // zero between launches
    int H, E, EC, pEC, nLx, rank, world;
    uint32_t epoch;
    int elem_bytes;
    int le_begin, le_end;      // only experts whose local index is in [le_begin, le_end) are moved
};

// Warp per routed row; rows are spread over the whole grid.
__global__ void __launch_bounds__(256) dispatch_kernel(DispatchArgs a) {
    __shared__ unsigned prefix[257];  // E <= 256
    __shared__ bool last_block;
    const int tid = threadIdx.x;
    pdl_trigger();
    pdl_wait();
    // Rows are sent in this order: local expert index first, and for each of them the owner
    // ranks starting with the one after this rank.  At any moment the source ranks therefore
    // write to DIFFERENT owners, instead of all pushing into the same GPU's NVLink ingress.
    // prefix[i] = rows before order position i (zero-length outside this launch's range).
    for (int i = tid; i < a.E; i += blockDim.x) {
        const int le = i / a.world, owner = (a.rank + 1 + i % a.world) % a.world;
        const int e = owner * a.nLx + le;
        prefix[i + 1] = (le >= a.le_begin && le < a.le_end) ? min(a.counts[e], (unsigned)a.EC) : 0u;
    }
    __syncthreads();
    if (tid == 0) {
        unsigned run = 0;
        for (int e = 0; e < a.E; ++e) {
            const unsigned n = prefix[e + 1];
            prefix[e] = run;
            run += n;
        }
        prefix[a.E] = run;
    }
    __syncthreads();
    const unsigned total = prefix[a.E];
    const int lane = tid & 31;
    const unsigned warps = gridDim.x * (blockDim.x >> 5);
    const unsigned row_chunks = (unsigned)((size_t)a.H * a.elem_bytes / 16);
    for (unsigned g = blockIdx.x * (blockDim.x >> 5) + (tid >> 5); g < total; g += warps) {
        int lo = 0, hi = a.E;  // last order position with prefix[] <= g
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (prefix[mid] <= g) lo = mid; else hi = mid;
        }
        const unsigned slot = g - prefix[lo];
        const int le = lo / a.world, owner = (a.rank + 1 + lo % a.world) % a.world;
        const int e = owner * a.nLx + le;
        const int tok = a.cell_tokens[(size_t)e * a.pEC + slot];
        const uint4* src = reinterpret_cast<const uint4*>(
            static_cast<const char*>(a.A) + (size_t)tok * a.H * a.elem_bytes);
        uint4* dst = reinterpret_cast<uint4*>(
            a.peers.arena[owner] + a.lay.xcell +
            (((size_t)a.rank * a.nLx + le) * a.pEC + slot) * a.H * a.elem_bytes);
        // eight 16-byte loads in flight per lane before the first store is issued
        for (unsigned c0 = lane; c0 < row_chunks; c0 += 256) {
            uint4 v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (c0 + 32 * q < row_chunks) v[q] = src[c0 + 32 * q];
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (c0 + 32 * q < row_chunks) dst[c0 + 32 * q] = v[q];
        }
    }
    // publish: every block fences its peer stores, the last block to finish raises the flags
    __threadfence_system();
    __syncthreads();
    if (tid == 0) {
        const unsigned prev = atomicAdd(a.done_counter, 1u);
        last_block = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if (last_block) {
        __threadfence_system();
        for (int e = tid; e < a.E; e += blockDim.x) {
            const int owner = e / a.nLx, le = e - owner * a.nLx;
            if (le < a.le_begin || le >= a.le_end) continue;
            unsigned long long* f = reinterpret_cast<unsigned long long*>(
                a.peers.arena[owner] + a.lay.xflag) + ((size_t)a.rank * a.nLx + le);
            st_release_sys(f, make_flag(a.epoch, min(a.counts[e], (unsigned)a.EC)));
        }
        if (tid == 0) *a.done_counter = 0u;
    }
}

// One 128-row panel of one cell: what a GEMM m-tile works on.
struct PanelEntry {
    int row_base;  // first row in the xcell / y1cell row space
    int rows;      // valid rows (1..128)
    int le;        // local expert
    int src;       // source rank
};

// off[i] = f(0) + .. + f(i-1) for i = 0 .. n, by one warp.
template <typename F>
__device__ __forceinline__ void warp_scan(F f, int* off, int n) {
    const int lane = threadIdx.x & 31;
    int run = 0;
    for (int i0 = 0; i0 < n; i0 += 32) {
        const int v = i0 + lane < n ? f(i0 + lane) : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (i0 + lane < n) off[i0 + lane] = run + incl - v;
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) off[n] = run;
}

// The panel list when every expert is this rank's own, by a whole block that knows the routed rows
// of every expert (cnt, off: shared memory, off has n + 1 entries).  The router does this in passing,
// so that a one-rank forward has no plan launch.
__device__ __forceinline__ void write_local_plan(const int* cnt, int* off, int n, int pEC, int rank,
                                                 PanelEntry* panels, int* le_start) {
    __syncthreads();
    if (threadIdx.x < 32) warp_scan([&](int e) { return (cnt[e] + kTileM - 1) / kTileM; }, off, n);
    __syncthreads();
    for (int e = threadIdx.x; e <= n; e += blockDim.x) {
        le_start[e] = off[e];
        if (e == n) break;
        for (int r = 0, i = off[e]; r < cnt[e]; r += kTileM, ++i)
            panels[i] = PanelEntry{e * pEC + r, min(kTileM, cnt[e] - r), e, rank};
    }
}

struct PlanArgs {
    const char* arena;       // this rank's arena
    ArenaLayout lay;
    PanelEntry* panels;      // [world*nLx*pEC/128]
    int* le_start;           // [nLx+1] panels of local expert le are [le_start[le], le_start[le+1])
    unsigned* cell_counts;   // [world*nLx] routed count per (source, local expert)
    DeviceStatus* status;
    int world, nLx, pEC;
    uint32_t epoch;
    long long wait_cycles;
    int le_begin, le_end;    // local experts planned by this launch; panels are appended
    int rank;
};

// Single block.  Waits (bounded) for the count flag of every (source, local expert) cell, then
// lists the panels grouped by local expert so that tiles sharing a weight tile run together.
__global__ void __launch_bounds__(1024) plan_kernel(PlanArgs a) {
    __shared__ int failed;
    __shared__ int cnt_s[2048];  // world * nLx <= 8 * 256; a count can reach pEC, which has no 16-bit limit
    const int cells = a.world * a.nLx;
    pdl_trigger();
    pdl_wait();
    if (threadIdx.x == 0) failed = 0;
    __syncthreads();
    const unsigned long long* flags =
        reinterpret_cast<const unsigned long long*>(a.arena + a.lay.xflag);
    for (int c = threadIdx.x; c < cells; c += blockDim.x) {
        const int cle = c % a.nLx;
        if (cle < a.le_begin || cle >= a.le_end) continue;
        unsigned long long v = 0;
        if (!wait_flag(flags + c, a.epoch, a.wait_cycles, &v)) {
            report_error(a.status, KLEOS_AT_PLAN_WAIT, c, (int)a.epoch);
            atomicExch(&failed, 1);
            a.cell_counts[c] = 0;
            cnt_s[c] = 0;
        } else {
            const unsigned n = min((unsigned)(v & 0xffffffffu), (unsigned)a.pEC);
            a.cell_counts[c] = n;
            cnt_s[c] = (int)n;
        }
    }
    __syncthreads();
    // plan order: local expert by local expert, sources starting with the rank after this one
    // (so that the expert ranks' result stores fan out over different source ranks instead of
    // converging on one).  A warp scans the panel counts of the cells in that order, then
    // every cell writes its own panels.
    __shared__ int off_s[2049];
    const int ncell = (a.le_end - a.le_begin) * a.world;
    const int n0 = a.le_begin == 0 ? 0 : a.le_start[a.le_begin];  // continue the previous launch's list
    if (threadIdx.x < 32)
        warp_scan(
            [&](int o) {
                const int le = a.le_begin + o / a.world, src = (a.rank + 1 + o % a.world) % a.world;
                return failed ? 0 : (cnt_s[src * a.nLx + le] + kTileM - 1) / kTileM;
            },
            off_s, ncell);
    __syncthreads();
    for (int le = threadIdx.x; le <= a.le_end - a.le_begin; le += blockDim.x)
        if (le > 0 || a.le_begin == 0) a.le_start[a.le_begin + le] = n0 + off_s[le * a.world];
    if (failed) return;
    for (int o = threadIdx.x; o < ncell; o += blockDim.x) {
        const int le = a.le_begin + o / a.world, src = (a.rank + 1 + o % a.world) % a.world;
        const int c = src * a.nLx + le;
        const int cnt = cnt_s[c];
        int n = n0 + off_s[o];
        for (int r = 0; r < cnt; r += kTileM)
            a.panels[n++] = PanelEntry{c * a.pEC + r, min(kTileM, cnt - r), le, src};
    }
}

// Training-mode gate statistics of one rank's tokens, as the reference keeps them in its
// bookkeeping (types.cuh:944-960): mean probability per expert (moe/gate.cuh:607-635), fraction
// of the tokens that chose each expert (unclamped, :698-705) and the auxiliary loss
// sum_e mean_prob[e] * mean_count[e] / E (:763-773).  One block of 256 threads; all sums in a fixed order.
// out = [mean_prob E][mean_count E][loss 1].
struct GateStatsArgs {
    const float* col_partial;  // [blocks][PX] column sums of the router's blocks, or null
    const unsigned* counts;    // [E]
    float* out;
    int blocks, PX, S, E;
};
__device__ __forceinline__ void gate_stats(const GateStatsArgs& a) {
    __shared__ float part[256], term[256];
    // 256 / PX threads per expert (PX = 192: one), each with its own run of blocks
    const int groups = 256 / a.PX, e = threadIdx.x % a.PX, grp = threadIdx.x / a.PX, per = (a.blocks + groups - 1) / groups;
    float sum = 0.f;
    if (grp < groups) {
#pragma unroll 8
        for (int b = grp * per; b < min((grp + 1) * per, a.blocks); ++b) sum += a.col_partial[(size_t)b * a.PX + e];
    }
    part[threadIdx.x] = sum;
    __syncthreads();
    float t = 0.f;
    if ((int)threadIdx.x < a.E) {
        for (int i = 1; i < groups; ++i) sum += part[i * a.PX + e];
        const float mp = sum / (float)a.S, mc = (float)a.counts[e] / (float)a.S;
        a.out[e] = mp;
        a.out[a.E + e] = mc;
        t = mp * mc / (float)a.E;
    }
    term[threadIdx.x] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        float loss = 0.f;
        for (int i = 0; i < a.E; ++i) loss += term[i];
        a.out[2 * a.E] = loss;
    }
}
__global__ void __launch_bounds__(256) gate_stats_kernel(GateStatsArgs a) {
    pdl_trigger();
    pdl_wait();
    gate_stats(a);
}

struct CombineArgs {
    GateStatsArgs stats;  // training mode: a last block beside those of the combine computes them
    const char* arena;   // this rank's arena (ycell, yflag)
    ArenaLayout lay;
    const void* probs;   // [S,PX] element-rounded gate probabilities
    const int* topk;     // [S,K]
    const int* slots;    // [S,K]
    const float* mcw;    // [S]
    void* out;           // [S,H]
    DeviceStatus* status;
    int S, H, K, PX, pEC;
    int world;           // return flags to wait for (0: the results are this rank's own, stored by the kernel before)
    uint32_t epoch;
    long long wait_cycles;
};

// out[t] = sum_j Element(prob[t,e_j]) * Element(y2[e_j][slot_j] / mCw[t]) over kept choices
// (reference processor.cuh:110-168); with k == 1 the row is copied unscaled (:170-204).
// Rows of tokens whose every choice was dropped are written as zeros.  Warp per token; KT is
// the compile-time top-k (0 = read it from the arguments), which lets the k row loads of
// several 16-byte chunks be issued together.
template <typename T, int KT>
__global__ void __launch_bounds__(256) combine_kernel(CombineArgs a) {
    __shared__ int failed;
    pdl_trigger();
    pdl_wait();
    const int blocks = (int)gridDim.x - (a.stats.col_partial != nullptr ? 1 : 0);
    if ((int)blockIdx.x == blocks) {
        gate_stats(a.stats);
        return;
    }
    if (threadIdx.x == 0) failed = 0;
    __syncthreads();
    if (threadIdx.x < a.world) {
        const unsigned long long* f =
            reinterpret_cast<const unsigned long long*>(a.arena + a.lay.yflag) + threadIdx.x;
        unsigned long long v;
        if (!wait_flag(f, a.epoch, a.wait_cycles, &v)) {
            report_error(a.status, KLEOS_AT_COMBINE_WAIT, threadIdx.x, (int)a.epoch);
            atomicExch(&failed, 1);
        }
    }
    __syncthreads();
    if (failed) return;

    constexpr int VEC = 16 / sizeof(T);
    constexpr int KMAX = KT > 0 ? KT : kMaxTopK;
    constexpr int UNR = KT > 0 && KT <= 2 ? 4 : 1;
    const int K = KT > 0 ? KT : a.K;
    const int lane = threadIdx.x & 31;
    const int warps = blocks * (blockDim.x >> 5);
    const T* probs = static_cast<const T*>(a.probs);
    const T* ycell = reinterpret_cast<const T*>(a.arena + a.lay.ycell);
    const int chunks = a.H / VEC;
    for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < a.S; t += warps) {
        const T* yrow[KMAX];
        float p[KMAX];
#pragma unroll
        for (int j = 0; j < KMAX; ++j) {
            yrow[j] = nullptr;
            p[j] = 0.f;
            if (j < K) {
                const int e = a.topk[(size_t)t * K + j];
                const int sl = a.slots[(size_t)t * K + j];
                p[j] = Elem<T>::to_f(probs[(size_t)t * a.PX + e]);
                if (sl != kDropped) yrow[j] = ycell + ((size_t)e * a.pEC + sl) * a.H;
            }
        }
        const float w = a.mcw[t];
        const float inv_w = 1.f / w;
        T* orow = static_cast<T*>(a.out) + (size_t)t * a.H;
        for (int c0 = lane; c0 < chunks; c0 += 32 * UNR) {
            uint4 raw[UNR][KMAX];
#pragma unroll
            for (int u = 0; u < UNR; ++u)
#pragma unroll
                for (int j = 0; j < KMAX; ++j)
                    if (j < K && yrow[j] != nullptr && c0 + 32 * u < chunks)
                        raw[u][j] = ld_cg_v4(yrow[j] + (size_t)(c0 + 32 * u) * VEC);
#pragma unroll
            for (int u = 0; u < UNR; ++u) {
                const int c = c0 + 32 * u;
                if (c >= chunks) break;
                uint4 o;
                if constexpr (sizeof(T) == 2) {
                    // 16-bit elements: Element(y / mCw) is one fp32 multiply and a packed round; the product
                    // with the bf16 probability and the running sum are single-rounding bf16x2
                    // instructions, which is exactly the element-type arithmetic of the
                    // reference's combine
                    using P2 = Pack2<T>;
                    typename P2::type acc2[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc2[i] = P2::from_f2(0.f, 0.f);
#pragma unroll
                    for (int j = 0; j < KMAX; ++j)
                        if (j < K && yrow[j] != nullptr) {
                            const typename P2::type* y2 = reinterpret_cast<const typename P2::type*>(&raw[u][j]);
                            const typename P2::type pj = P2::from_f2(p[j], p[j]);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                if (K > 1) {
                                    const float2 yf = P2::to_f2(y2[i]);
                                    const typename P2::type v = P2::from_f2(yf.x * inv_w, yf.y * inv_w);
                                    acc2[i] = P2::add(acc2[i], P2::mul(pj, v));
                                } else {
                                    acc2[i] = y2[i];
                                }
                            }
                        }
                    o = *reinterpret_cast<const uint4*>(acc2);
                } else {
                    float acc[VEC];
#pragma unroll
                    for (int i = 0; i < VEC; ++i) acc[i] = 0.f;
#pragma unroll
                    for (int j = 0; j < KMAX; ++j)
                        if (j < K && yrow[j] != nullptr) {
                            const T* yv = reinterpret_cast<const T*>(&raw[u][j]);
#pragma unroll
                            for (int i = 0; i < VEC; ++i) {
                                if (K > 1) {
                                    const float v = Elem<T>::round(Elem<T>::to_f(yv[i]) / w);
                                    const float sc = Elem<T>::round(p[j] * v);
                                    acc[i] = Elem<T>::round(acc[i] + sc);
                                } else {
                                    acc[i] = Elem<T>::to_f(yv[i]);
                                }
                            }
                        }
                    T* ov = reinterpret_cast<T*>(&o);
#pragma unroll
                    for (int i = 0; i < VEC; ++i) ov[i] = Elem<T>::from_f(acc[i]);
                }
                *reinterpret_cast<uint4*>(orow + (size_t)c * VEC) = o;
            }
        }
    }
}

// Flag raised by the last GEMM2 block: tells every source rank that this expert rank has
// stored all of its result rows.
struct ReturnFlagArgs {
    PeerTable peers;
    ArenaLayout lay;
    unsigned* done_counter;
    int rank, world;   // world 0: all results stay on this rank, whose next kernel needs no flag (8 to 12 us)
    uint32_t epoch;
    int suppress;  // test hook: do not raise the flags (exercises the bounded wait in combine)
};

template <typename Flag>
__device__ __forceinline__ void publish_return_flags(const ReturnFlagArgs& r, Flag* smem_last) {
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned prev = atomicAdd(r.done_counter, 1u);
        *smem_last = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if (*smem_last) {
        __threadfence_system();
        if ((int)threadIdx.x < r.world && !r.suppress) {
            unsigned long long* f = reinterpret_cast<unsigned long long*>(
                r.peers.arena[threadIdx.x] + r.lay.yflag) + r.rank;
            st_release_sys(f, make_flag(r.epoch, 1u));
        }
        if (threadIdx.x == 0) *r.done_counter = 0u;
    }
}

}  // namespace kleos
