// kleos_route_static: the router for callers that must not allocate device memory.
//
// Some hosts of this library cannot call cudaMalloc at the point where they need a routing
// decision: code running inside a framework's memory-pool callback, a real-time serving loop
// that has pinned its memory budget up front, or a process whose allocator is owned by another
// runtime.  The regular path (kleos_initialize + kleos_forward) allocates its bookkeeping once
// at initialise time; this entry point needs no initialise call at all.  The float router's scratch
// (the list of near-tie tokens, their fp64 logits, completion counters) and a zero bias live in
// the fixed array below, which every GPU that loads the library holds until the process exits.  The bf16
// router keeps everything else on the chip.
//
// This file is compiled as part of kleos_api.cu (one translation unit), so the array, the
// cudaGetSymbolAddress call and the launches below all see the same symbol.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>

#include "route_split.cuh"

namespace {

constexpr int kStaticMaxTokens = 4096;  // S limit
constexpr int kStaticMaxExperts = 64;   // E limit (one 64-wide gate tile)
constexpr int kMaxDevices = 64;

// Layout of the scratch array (byte offsets, all 256-byte aligned).
constexpr size_t kOffCount = 0;                                                // int
constexpr size_t kOffStatus = 64;                                              // DeviceStatus, bf16: the tokens say it too
constexpr size_t kOffDone = 256;                                               // int[S]
constexpr size_t kOffList = kOffDone + sizeof(int) * kStaticMaxTokens;         // int[S]
constexpr size_t kOffZeroBias = kOffList + sizeof(int) * kStaticMaxTokens;     // float[E], stays 0
constexpr size_t kClearBytes = kOffZeroBias + 256;                             // cleared by every float call
constexpr size_t kOffLogits = kClearBytes;                                     // double[S*E]
constexpr size_t kScratchBytes =
    kOffLogits + sizeof(double) * kStaticMaxTokens * kStaticMaxExperts;
static_assert(kScratchBytes == 2130432, "the size quoted in kleos_b200.h and in the documentation");

// In host code this name is only a handle for cudaGetSymbolAddress, never a device address.
static __device__ __align__(256) unsigned char g_route_scratch[kScratchBytes];

struct StaticDevice {
    unsigned char* scratch = nullptr;
    long long wait_cycles = 20000000000LL;  // about ten seconds; KLEOS_WAIT_MS at the first call
    int withhold = 0;                       // KLEOS_DEBUG_STATIC_WITHHOLD=1 at the first call: see route_split::Args
};
StaticDevice g_static[kMaxDevices];

int complain(int code, const char* what) {
    std::fprintf(stderr, "[kleos_b200] kleos_route_static: %s\n", what);
    return code;
}

}  // namespace

extern "C" int kleos_route_static(const void* A, const void* Wg, const float* gate_bias, int S,
                                  int H, int E, int K, int torch_dtype, void* probs,
                                  int32_t* topk, float* mcw, void* stream) {
    using namespace kleos;
    if (!A || !Wg || !probs || !topk || !mcw) return complain(KLEOS_E_ARG, "null device pointer");
    // the near-tie re-evaluation reads rows of A and Wg sixteen bytes at a time
    if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(Wg)) & 15)
        return complain(KLEOS_E_ARG, "A and Wg must be 16-byte aligned");
    if (S < 1 || S > kStaticMaxTokens)
        return complain(KLEOS_E_ARG, "S exceeds the 4096-token limit of the fixed scratch array");
    if (E < 1 || E > kStaticMaxExperts)
        return complain(KLEOS_E_ARG, "E exceeds the 64-expert limit of the fixed scratch array");
    if (K < 1 || K > E || K > kMaxTopK) return complain(KLEOS_E_ARG, "top-k out of range");
    if (H < 64 || H % 64) return complain(KLEOS_E_ARG, "H must be a positive multiple of 64");
    if (torch_dtype != 0 && torch_dtype != 2)
        return complain(KLEOS_E_UNSUPPORTED, "torch_dtype must be 0 (float) or 2 (bf16)");  // fp16: use the layer API

    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return complain(KLEOS_E_CUDA, "no current CUDA device");
    StaticDevice& here = g_static[dev];
    if (!here.scratch) {
        // one-time set-up for this device (do the first call outside any stream capture)
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_route_scratch);
        const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
        if (e == cudaSuccess) e = cudaFuncSetAttribute(route_kernel<float, 64>, dyn, route_fma::smem_bytes<float, 64>());
        if (e == cudaSuccess) e = cudaFuncSetAttribute(route_split_kernel<__nv_bfloat16, 64, 2, true>, dyn, route_split::Shape<64>::SMEM_BYTES);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(route_split_kernel<__nv_bfloat16, 64, 0, true>, dyn, route_split::Shape<64>::SMEM_BYTES);
        if (e != cudaSuccess || !p) {
            std::fprintf(stderr, "[kleos_b200] setting up kleos_route_static failed: %s\n",
                         cudaGetErrorString(e));
            return KLEOS_E_CUDA;
        }
        if (const char* w = std::getenv("KLEOS_WAIT_MS")) {
            int khz = 0;
            if (cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, dev) == cudaSuccess)
                here.wait_cycles = (long long)(std::atof(w) * khz);
        }
        const char* wh = std::getenv("KLEOS_DEBUG_STATIC_WITHHOLD");
        here.withhold = wh && wh[0] == '1';
        here.scratch = static_cast<unsigned char*>(p);
    }
    unsigned char* scratch = here.scratch;
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : cudaStreamPerThread;

    RouteArgs ra{};
    ra.A = A;
    ra.Wg = Wg;
    ra.bias = gate_bias ? gate_bias : reinterpret_cast<const float*>(scratch + kOffZeroBias);
    ra.probs = probs;
    ra.topk = topk;
    ra.mcw = mcw;
    ra.refine_count = reinterpret_cast<int*>(scratch + kOffCount);
    ra.refine_done = reinterpret_cast<int*>(scratch + kOffDone);
    ra.refine_list = reinterpret_cast<int*>(scratch + kOffList);
    ra.refine_logits = reinterpret_cast<double*>(scratch + kOffLogits);
    ra.S = S;
    ra.H = H;
    ra.E = E;
    ra.K = K;
    ra.PX = 64;
    ra.tie_eps = 1e-4f;
    if (torch_dtype == 0) {
        // the counter, the completion flags and the zero bias must start at zero; the previous
        // call (or an aborted one) may have left anything there
        if (cudaMemsetAsync(scratch, 0, kClearBytes, st) != cudaSuccess)
            return complain(KLEOS_E_CUDA, "cudaMemsetAsync on the scratch array failed");
        const int grid = (S + route_fma::TM - 1) / route_fma::TM;
        route_kernel<float, 64><<<grid, 256, route_fma::smem_bytes<float, 64>(), st>>>(ra);
        refine_kernel<float><<<148, 256, 0, st>>>(ra);
    } else {
        // bf16 goes to the tensor cores (route_split.cuh): four blocks per 128 tokens, or as many as there
        // are 64-wide slices of K.  mCw is a 32-bit result, so the running sums stay short: an accumulator per
        // slice, added up in fp32 registers eight at a time.  4096 tokens, H = 2048, 64 experts: 18.5 us; the two
        // kernels on the FP32 pipes took 58.
        CUtensorMap map_a, map_wg;
        const char* err = encode_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, (uint64_t)S, (uint64_t)H, route_split::BM, 64);
        if (!err) err = encode_map(&map_wg, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, Wg, 64, (uint64_t)H, 64, 64);
        if (err) return complain(KLEOS_E_CUDA, err);
        route_split::Args sp{};
        sp.r = ra;
        sp.status = reinterpret_cast<DeviceStatus*>(scratch + kOffStatus);
        sp.place.wait_cycles = here.wait_cycles;
        sp.withhold = here.withhold;
        const int slices = H / 64;
        sp.parts = slices >= 4 ? 4 : slices >= 2 ? 2 : 1;
        sp.own = route_split::BM / sp.parts;
        sp.acc_slices = 1;
        cudaLaunchConfig_t lc{};
        lc.gridDim = dim3((unsigned)((S + route_split::BM - 1) / route_split::BM * sp.parts));
        lc.blockDim = dim3(route_split::kThreads);
        lc.dynamicSmemBytes = route_split::Shape<64>::SMEM_BYTES;
        lc.stream = st;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)sp.parts;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        lc.attrs = &at;
        lc.numAttrs = 1;
        if (K == 2) cudaLaunchKernelEx(&lc, route_split_kernel<__nv_bfloat16, 64, 2, true>, map_a, map_wg, sp);
        else cudaLaunchKernelEx(&lc, route_split_kernel<__nv_bfloat16, 64, 0, true>, map_a, map_wg, sp);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        std::fprintf(stderr, "[kleos_b200] kleos_route_static launch failed: %s\n",
                     cudaGetErrorString(e));
        return KLEOS_E_CUDA;
    }
    return KLEOS_OK;
}
