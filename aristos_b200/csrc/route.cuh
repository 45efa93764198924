// Router: gate GEMM + softmax + top-k, near-tie refinement, slot assignment.
//
// Semantics follow the reference gate (moe/gate.cuh:470-720): logits = A * Wg^T with fp32
// accumulation, softmax over the E real experts, k rounds of masked arg-max with ties to the
// lowest expert id (:654-670), mCw = sum of the k winning probabilities (:669), slot per
// (expert, token) kept iff slot < EC (:689-718).  Two deliberate differences: slots are
// handed out in ascending token order (the reference uses atomicAdd arrival order,
// :698-700), and tokens whose k-th / (k+1)-th logits are closer than fp32 summation error
// are re-evaluated in fp64 so the selected set does not depend on accumulation order.
#pragma once

#include "transport.cuh"

namespace kleos {

struct RouteArgs {
    const void* A;        // [S,H] activations
    const void* Wg;       // [PX,H] gate weight, row e = expert e
    const float* bias;    // [E] logit bias (zeros when unused)
    void* probs;          // [S,PX] gate probabilities (element type)
    int* topk;            // [S,K]
    float* mcw;           // [S]
    int* refine_list;     // token ids needing fp64 re-evaluation
    int* refine_count;
    double* refine_logits;  // [S,E] fp64 logits of listed tokens
    int* refine_done;       // [S] per listed token: logits finished (zero between forwards)
    int S, H, E, K, PX;
    float tie_eps;
    // training mode only, else null: [router blocks][PX] column sums of the fp32 probabilities
    // of each block's tokens, summed in a fixed order (the reference accumulates the same
    // per-expert mean with atomicAdd, moe/gate.cuh:607-635)
    float* col_partial;
};

// ---------------------------------------------------------------- router on the FP32 pipes
// Float layers, layers of more than 128 experts, and kleos_route_static on float.  Bound by the FP32
// FMA rate and L2: S * H * PX multiply-adds (4096 tokens, H = 2048, 64 experts: 15 us on all SMs).  One
// block per 32 tokens; the K dimension is split over its eight warps, each with its own 16-wide K
// slices of the tokens and of 64 gate-weight rows, double-buffered by asynchronous copies, so the
// main loop has no block barrier; a lane keeps 8 tokens x 8 experts and reads four K values at a time
// (16 shared-memory loads per 256 multiply-adds, no bank conflicts).  The eight partial sums are added
// in a fixed order, then a warp per token does softmax and top-k.
// Measured, 4096 tokens, H = 2048, 64 experts: float 42 us, bf16 45; one block per 64 tokens with
// scalar loads and one thread per token in the selection took 139 and 141.  256 tokens, H = 512: 37
// -> 14 us.  (Sixteen warps of 128 registers: 48 and 60.)
namespace route_fma {
constexpr int TM = 32, TE = 64, KC = 16, WARPS = 8, PART_LD = 72;
template <typename T> constexpr int kLd = sizeof(T) == 4 ? 20 : 24;  // elements a row of a slice takes
template <typename T> constexpr int kSliceBytes = (TM + TE) * kLd<T> * (int)sizeof(T);
template <typename T, int PXT> constexpr int smem_bytes() {
    return WARPS * 2 * kSliceBytes<T> + TM * (PXT + 1) * 4;
}
static_assert(WARPS * 2 * kSliceBytes<float> >= WARPS * TM * PART_LD * 4 &&
              WARPS * 2 * kSliceBytes<__half> >= WARPS * TM * PART_LD * 4, "the partial sums reuse the slices");

__device__ __forceinline__ void copy16_async(void* smem, const void* global) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                 ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))), "l"(global)
                 : "memory");
}
template <typename T> __device__ __forceinline__ float4 load4(const T* p) {
    if constexpr (sizeof(T) == 4) {
        return *reinterpret_cast<const float4*>(p);
    } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(p);
        const float2 a = Pack2<T>::to_f2(*reinterpret_cast<const typename Pack2<T>::type*>(&raw.x));
        const float2 b = Pack2<T>::to_f2(*reinterpret_cast<const typename Pack2<T>::type*>(&raw.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
}
}  // namespace route_fma

template <typename T, int PXT>
__global__ void __launch_bounds__(256) route_kernel(RouteArgs a) {
    using namespace route_fma;
    constexpr int LD = kLd<T>, LDL = PXT + 1, VEC = 16 / (int)sizeof(T), PIECES = KC / VEC;
    extern __shared__ __align__(16) unsigned char route_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    T* mine = reinterpret_cast<T*>(route_smem + warp * 2 * kSliceBytes<T>);
    float* part = reinterpret_cast<float*>(route_smem);  // [WARPS][TM][PART_LD], after the K loop
    float* Ls = reinterpret_cast<float*>(route_smem + WARPS * 2 * kSliceBytes<T>);  // [TM][LDL]
    const T* A = static_cast<const T*>(a.A);
    const T* Wg = static_cast<const T*>(a.Wg);
    const int row0 = blockIdx.x * TM, H = a.H, slices = H / KC;
    const int ty = lane >> 3, tx = lane & 7;
    pdl_trigger();
    pdl_wait();

    for (int e0 = 0; e0 < PXT; e0 += TE) {
        float acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
        auto fetch = [&](int sl, int buf) {
            T* dst = mine + buf * (TM + TE) * LD;
#pragma unroll
            for (int i = 0; i < (TM + TE) * PIECES / 32; ++i) {
                const int r = (i * 32 + lane) / PIECES, c = (i * 32 + lane) % PIECES;
                // rows past the last token repeat it; their results are not used
                const T* row = r < TM ? A + (size_t)min(row0 + r, a.S - 1) * H : Wg + (size_t)(e0 + r - TM) * H;
                copy16_async(dst + r * LD + c * VEC, row + sl * KC + c * VEC);
            }
        };
        if (warp < slices) fetch(warp, 0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        int buf = 0;
        for (int sl = warp; sl < slices; sl += WARPS, buf ^= 1) {
            if (sl + WARPS < slices) fetch(sl + WARPS, buf ^ 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            const T* As = mine + buf * (TM + TE) * LD + ty * LD;
            const T* Bs = mine + buf * (TM + TE) * LD + (TM + tx) * LD;
#pragma unroll
            for (int k = 0; k < KC; k += 4) {
                float4 x[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] = load4(As + 4 * i * LD + k);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 w = load4(Bs + 8 * j * LD + k);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        acc[i][j] = fmaf(x[i].w, w.w, fmaf(x[i].z, w.z, fmaf(x[i].y, w.y, fmaf(x[i].x, w.x, acc[i][j]))));
                }
            }
            __syncwarp();  // every lane is done with the slice before it is overwritten
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) part[(warp * TM + ty + 4 * i) * PART_LD + tx + 8 * j] = acc[i][j];
        __syncthreads();
        for (int o = tid; o < TM * TE; o += 256) {
            const int r = o / TE, e = o % TE;
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) s += part[(w * TM + r) * PART_LD + e];
            Ls[r * LDL + e0 + e] = s + (e0 + e < a.E ? a.bias[e0 + e] : 0.f);
        }
        __syncthreads();  // the slices may be filled again; the logits are complete after the last round
    }

    // Selection, a warp per token: k + 1 rounds of arg-max over the logits (equal values to the lower
    // expert id, the reference's tie rule, moe/gate.cuh:662-667; a value that compares greater than
    // nothing is never chosen and leaves id 0), softmax over the E real experts.
    constexpr int PER = PXT / 32;
    T* probs = static_cast<T*>(a.probs);
    for (int r = warp; r < TM && row0 + r < a.S; r += WARPS) {
        const int t = row0 + r;
        float l[PER];
        unsigned taken = 0;
#pragma unroll
        for (int q = 0; q < PER; ++q) l[q] = lane + 32 * q < a.E ? Ls[r * LDL + lane + 32 * q] : -INFINITY;
        float m = 0.f, kth = 0.f, margin = INFINITY, top = 0.f;  // top: lane j keeps the j-th chosen logit
        for (int j = 0; j <= a.K && j < a.E; ++j) {
            float bv = -INFINITY;
            int be = 0x7fffffff;
#pragma unroll
            for (int q = 0; q < PER; ++q)
                if (!((taken >> q) & 1u) && l[q] > bv) {
                    bv = l[q];
                    be = lane + 32 * q;
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oe = __shfl_xor_sync(0xffffffffu, be, o);
                if (ov > bv || (ov == bv && oe < be)) {
                    bv = ov;
                    be = oe;
                }
            }
            if (be != 0x7fffffff && (be & 31) == lane) taken |= 1u << (be >> 5);
            if (j == 0) m = bv;
            if (j == a.K) {
                margin = kth - bv;
            } else {
                kth = bv;
                if (lane == j) top = bv;
                if (lane == 0) a.topk[(size_t)t * a.K + j] = be == 0x7fffffff ? 0 : be;
            }
        }
        float p[PER], d = 0.f;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            p[q] = lane + 32 * q < a.E ? __expf(l[q] - m) : 0.f;
            d += p[q];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        const float inv = 1.f / d;
        float w = lane < a.K ? __expf(top - m) * inv : 0.f;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);  // k <= 8
        if (lane == 0) {
            a.mcw[t] = w;
            if (margin < a.tie_eps * fmaxf(1.f, fabsf(kth))) {
                const int pos = atomicAdd(a.refine_count, 1);
                a.refine_list[pos] = t;  // list has room for every token
            }
        }
        // probabilities, padding columns zero (PX == PXT: both are E rounded up to 64)
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const float pq = p[q] * inv;
            probs[(size_t)t * PXT + lane + 32 * q] = Elem<T>::from_f(pq);
            if (a.col_partial != nullptr) Ls[r * LDL + lane + 32 * q] = pq;
        }
    }
    if (a.col_partial != nullptr) {
        __syncthreads();
        if (tid < PXT) {
            float sum = 0.f;
            for (int r = 0; r < TM && row0 + r < a.S; ++r) sum += Ls[r * LDL + tid];
            a.col_partial[(size_t)blockIdx.x * PXT + tid] = sum;
        }
    }
}

// fp64 re-evaluation of the tokens on the refine list.  One warp per (listed token, expert)
// dot product; the warp that completes a token's last logit redoes that token's selection.
template <typename T>
__global__ void __launch_bounds__(256) refine_kernel(RouteArgs a) {
    constexpr int VEC = 16 / sizeof(T);
    const T* A = static_cast<const T*>(a.A);
    const T* Wg = static_cast<const T*>(a.Wg);
    pdl_trigger();
    pdl_wait();
    const int n = *a.refine_count;
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < n * a.E;
         item += warps) {
        const int i = item / a.E, e = item - i * a.E;
        const int t = a.refine_list[i];
        const T* x = A + (size_t)t * a.H;
        const T* w = Wg + (size_t)e * a.H;
        double s = 0.0;
#pragma unroll 4
        for (int h = lane * VEC; h < a.H; h += 32 * VEC) {
            const uint4 xr = *reinterpret_cast<const uint4*>(x + h);
            const uint4 wr = *reinterpret_cast<const uint4*>(w + h);
            const T* xv = reinterpret_cast<const T*>(&xr);
            const T* wv = reinterpret_cast<const T*>(&wr);
#pragma unroll
            for (int q = 0; q < VEC; ++q)
                s += (double)Elem<T>::to_f(xv[q]) * (double)Elem<T>::to_f(wv[q]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        int done = 0;
        if (lane == 0) {
            a.refine_logits[(size_t)i * a.E + e] = s + (double)a.bias[e];
            __threadfence();
            done = atomicAdd(a.refine_done + i, 1);
        }
        done = __shfl_sync(0xffffffffu, done, 0);
        if (done != a.E - 1) continue;
        // last logit of token i: the whole warp redoes the selection on the fp64 logits
        // (k rounds of warp arg-max, ties to the lowest expert id) and the fp32 softmax
        __threadfence();
        constexpr int PER_LANE = 8;  // E <= 256
        const double* l64 = a.refine_logits + (size_t)i * a.E;
        double cand[PER_LANE];
        float lf[PER_LANE];
#pragma unroll
        for (int q = 0; q < PER_LANE; ++q) {
            const int ee = lane + 32 * q;
            cand[q] = ee < a.E ? __ldcg(l64 + ee) : -INFINITY;
            lf[q] = (float)cand[q];
        }
        float m = -INFINITY;
#pragma unroll
        for (int q = 0; q < PER_LANE; ++q) m = fmaxf(m, lf[q]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float d = 0.f;
#pragma unroll
        for (int q = 0; q < PER_LANE; ++q)
            if (lane + 32 * q < a.E) d += __expf(lf[q] - m);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        const float inv = 1.f / d;
        float wsum = 0.f;
        for (int j = 0; j < a.K; ++j) {
            double bv = -INFINITY;
            int be = 0x7fffffff;
#pragma unroll
            for (int q = 0; q < PER_LANE; ++q) {
                const int ee = lane + 32 * q;  // ascending per lane, so '>' keeps the lower id
                if (cand[q] > bv) {
                    bv = cand[q];
                    be = ee;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oe = __shfl_xor_sync(0xffffffffu, be, o);
                if (ov > bv || (ov == bv && oe < be)) {
                    bv = ov;
                    be = oe;
                }
            }
            // every lane now agrees on (bv, be); its owner retires the candidate
#pragma unroll
            for (int q = 0; q < PER_LANE; ++q)
                if (lane + 32 * q == be) cand[q] = -INFINITY;
            if (lane == 0) a.topk[(size_t)t * a.K + j] = be;
            wsum += __expf((float)bv - m) * inv;
        }
        if (lane == 0) {
            a.mcw[t] = wsum;
            a.refine_done[i] = 0;  // ready for the next forward
        }
        T* probs = static_cast<T*>(a.probs);
#pragma unroll
        for (int q = 0; q < PER_LANE; ++q) {
            const int ee = lane + 32 * q;
            if (ee < a.E) probs[(size_t)t * a.PX + ee] = Elem<T>::from_f(__expf(lf[q] - m) * inv);
        }
    }
}

// Slots in ascending token order (the reference hands them out in atomicAdd arrival order,
// moe/gate.cuh:689-718; ascending order is one of its possible outcomes and is reproducible).
struct PlaceArgs {
    const int* topk;        // [S,K], place_kernel only
    const void* A;          // [S,H]
    int* slots;             // [S,K] slot or kDropped
    int* cell_tokens;       // [E,pEC] token id held by each slot
    unsigned* counts;       // [E] unclamped
    // [rows][place_words(PX)]: every block's histogram of chosen experts, four counts of 12 bits and a tag of 16 bits
    // in a word, so that a reader knows from the word itself that it is this launch's.  (A count
    // reaches 128 * k = 1024: a token of NaN logits chooses expert 0 k times.)
    unsigned long long* hist;
    // {launches so far, rows placed by this one}: the tag comes from here and not from the epoch, which is an
    // argument and the same in every replay of a captured forward
    unsigned* launch;
    // publish: count flags, cflag[owner][rank*nLx + le] = (epoch<<32)|routed, one 8-byte peer store
    // per expert (the reference's first-stage signal carries the same count, types.cuh:300-317)
    PeerTable peers;
    size_t cflag;
    int publish;
    // one rank, GEMMs that read the cells: the token rows go to this rank's own cells [E][pEC][H] (else null)
    char* xcell;
    unsigned row_chunks;    // 16-byte chunks of a token row
    // one rank, GEMMs that work through a panel list: the last block writes it (else null)
    PanelEntry* panels;
    int* le_start;
    DeviceStatus* status;
    long long wait_cycles;
    int S, K, E, PX, EC, pEC, nLx, rank;
    uint32_t epoch;
};

constexpr int kPlaceThreads = 512, kPlaceWarps = kPlaceThreads / 32;
constexpr int kPlaceMaxE = 256;
__host__ __device__ constexpr int place_words(int px) { return px / 4; }  // px is a multiple of 64
struct PlaceScratch {
    int wcount[kPlaceWarps][kPlaceMaxE];
    int part[kPlaceThreads * 4];
    int base[kPlaceMaxE], total[kPlaceMaxE], off[kPlaceMaxE + 1];
};

__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Slots, counts and (one rank) the way of the rows into the cells for one block's `own` <= 128 tokens, from tok0
// on, row `row` of n_rows: 512 threads, all of them.  top[own * K] and hist[PX] are the chosen experts and
// their histogram, in shared memory.  The block publishes its histogram and adds up those of the rows
// before it as they come, without a fence, a flag or a grid barrier: it only waits for blocks of lower
// index.  A wait that runs out raises *abort_flag.  `launch`: PlaceArgs::launch[0], read before.
__device__ __forceinline__ void place_tokens(const PlaceArgs& a, unsigned launch, int row, int n_rows, int tok0, int own, int* top,
                                             const int* hist, PlaceScratch* s, volatile int* abort_flag, DeviceStatus* status) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, K = a.K, E = a.E, words = place_words(a.PX);
    const uint32_t tag = (launch + 1) & 0xffffu;  // (the words are zero at first)
    if (tid < words && !*abort_flag) {
        unsigned long long w = (unsigned long long)tag << 48;
        for (int j = 0; j < 4; ++j) w |= (unsigned long long)hist[4 * tid + j] << (12 * j);
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(a.hist + (size_t)row * words + tid), "l"(w) : "memory");
    }
    // The row is counted, also after a failed wait: with the last one, every block has read launch[0].  (By a thread
    // that has no row to wait for in a small layer: at the block's end the count took 0.3 of 31 us.)
    if (tid == kPlaceThreads - 1 && atomicInc(a.launch + 1, (unsigned)n_rows - 1) == (unsigned)n_rows - 1) a.launch[0] = launch + 1;
    for (int i = tid; i < kPlaceWarps * kPlaceMaxE; i += kPlaceThreads) (&s->wcount[0][0])[i] = 0;
    // `width` threads per row, a word each; four rows in flight
    const int width = words <= 16 ? 16 : words <= 32 ? 32 : 64, groups = kPlaceThreads / width;
    const int word = tid % width, grp = tid / width;
    int run[4] = {0, 0, 0, 0};
    if (word < words) {
        const long long t0 = clock64();
#pragma unroll 1
        for (int r0 = grp; r0 < row && !*abort_flag; r0 += 4 * groups) {
            unsigned long long v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                v[j] = r0 + j * groups < row ? ld_relaxed_u64(a.hist + (size_t)(r0 + j * groups) * words + word) : 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (r0 + j * groups >= row) break;
                while ((uint32_t)(v[j] >> 48) != tag) {
                    __nanosleep(100);
                    v[j] = ld_relaxed_u64(a.hist + (size_t)(r0 + j * groups) * words + word);
                    if (*abort_flag) break;
                    if (clock64() - t0 > a.wait_cycles) {
                        report_error(status, KLEOS_AT_GRID_BARRIER, row, (int)a.epoch);
                        *abort_flag = 1;
                        break;
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) run[q] += (int)((v[j] >> (12 * q)) & 0xfff);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) s->part[(grp * width + word) * 4 + q] = run[q];
    }
    __syncthreads();
    for (int e = tid; e < a.PX; e += kPlaceThreads) {
        int sum = 0;
#pragma unroll 4
        for (int i = 0; i < groups; ++i) sum += s->part[i * width * 4 + e];
        s->base[e] = sum;
        s->total[e] = sum + hist[e];
    }
    __syncthreads();
    if (*abort_flag) return;  // (the same for all threads: nothing raises it from here on)
    // Rank of every (token, choice) entry among the earlier entries of the block that chose the same
    // expert: inside a warp from a match mask, across the warps from a per-warp count table.
    const int n_own = own * K;
#pragma unroll 1
    for (int i0 = 0; i0 < n_own; i0 += kPlaceThreads) {
        const int i = i0 + tid;
        const int e = i < n_own ? top[i] : -1;
        const unsigned same = __match_any_sync(0xffffffffu, e);
        const int before = __popc(same & ((1u << lane) - 1u));
        const bool lead = e >= 0 && before == 0;
        if (lead) s->wcount[warp][e] = __popc(same);
        __syncthreads();
        if (e >= 0) {
            int pos = s->base[e] + before;
            for (int w = 0; w < warp; ++w) pos += s->wcount[w][e];
            const bool kept = pos < a.EC;
            a.slots[(size_t)tok0 * K + i] = kept ? pos : kDropped;
            if (kept) a.cell_tokens[(size_t)e * a.pEC + pos] = tok0 + i / K;
            top[i] = kept ? e * a.pEC + pos : -1;  // from here on: the entry's row in the cells
        }
        __syncthreads();
        if (lead) {
            atomicAdd(&s->base[e], s->wcount[warp][e]);
            s->wcount[warp][e] = 0;
        }
        __syncthreads();
    }
    if (row == n_rows - 1) {
        // totals of every expert: unclamped count for this rank, clamped count to the owner
        for (int e = tid; e < E; e += kPlaceThreads) {
            const int total = s->total[e];
            a.counts[e] = (unsigned)total;
            s->total[e] = min(total, a.EC);
            if (a.publish) {
                const int owner = e / a.nLx, le = e - owner * a.nLx;
                st_release_sys(reinterpret_cast<unsigned long long*>(a.peers.arena[owner] + a.cflag) + ((size_t)a.rank * a.nLx + le),
                               make_flag(a.epoch, (unsigned)min(total, a.EC)));
            }
        }
        if (a.panels != nullptr) write_local_plan(s->total, s->off, E, a.pEC, a.rank, a.panels, a.le_start);
    }
    if (a.xcell != nullptr) {
        // a warp per token, which is read once and stored to each expert that kept it
#pragma unroll 1
        for (int tk = warp; tk < own; tk += kPlaceWarps) {
            const uint4* src = static_cast<const uint4*>(a.A) + (size_t)(tok0 + tk) * a.row_chunks;
#pragma unroll 1
            for (unsigned c0 = lane; c0 - lane < a.row_chunks; c0 += 256) {
                uint4 v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (c0 + 32 * q < a.row_chunks) v[q] = src[c0 + 32 * q];
#pragma unroll 1
                for (int j = 0; j < K; ++j) {
                    const int to = top[tk * K + j];
                    if (to < 0) continue;
                    uint4* dst = reinterpret_cast<uint4*>(a.xcell) + (size_t)to * a.row_chunks;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (c0 + 32 * q < a.row_chunks) dst[c0 + 32 * q] = v[q];
                }
            }
        }
    }
}

// The same on its own, behind the routers whose blocks do not have 512 threads or whose choices the near-tie
// kernel may change: one block per 32, 64 or 128 tokens (place_own()).  Blocks wait for lower ones, which are placed on
// the chip first.  It stands for three kernels (histogram 2.8 us, slots 5.9, rows 3.9 at 256 tokens, 8 float experts,
// where the forward went from 97.5 to 85 with the return flags gone too).
constexpr int kPlaceOwn = 32, kPlaceOwnMost = 128;
__global__ void __launch_bounds__(kPlaceThreads) place_kernel(PlaceArgs a, int tokens) {
    __shared__ PlaceScratch s;
    __shared__ int hist[kPlaceMaxE], top[kPlaceOwnMost * kMaxTopK], abort;
    __shared__ unsigned launch;
    pdl_wait();
    pdl_trigger();
    const int tid = threadIdx.x, tok0 = blockIdx.x * tokens, own = min(tokens, a.S - tok0);
    for (int e = tid; e < kPlaceMaxE; e += kPlaceThreads) hist[e] = 0;
    if (tid == 0) abort = 0;
    if (tid == kPlaceThreads - 1) launch = ld_relaxed_u32(a.launch);
    __syncthreads();
    for (int i = tid; i < own * a.K; i += kPlaceThreads) {
        top[i] = a.topk[(size_t)tok0 * a.K + i];
        atomicAdd(&hist[top[i]], 1);
    }
    __syncthreads();
    place_tokens(a, launch, blockIdx.x, gridDim.x, tok0, own, top, hist, &s, &abort, a.status);
}

}  // namespace kleos
