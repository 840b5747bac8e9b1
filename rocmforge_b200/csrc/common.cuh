// Shared device helpers for the hand-written sm_100a kernels.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#define RF_PAGE 64            // tokens per cache page; the Python cache uses the same number

// The first key position that a query at position pos sees; it always sees up to pos itself.  The attention kernels
// take the rule as one number: span > 0, the last span positions (a sliding window); span < 0, the positions of the
// query's own chunk of -span positions, chunks counted from position 0 of the sequence; 0, every position.  The bound
// never falls as pos grows.
__host__ __device__ __forceinline__ int rf_first_key(int pos, int span) {
    if (span > 0) return pos - span + 1 > 0 ? pos - span + 1 : 0;
    if (span < 0) return pos / (-span) * (-span);
    return 0;
}

// Every exported launcher returns 0, a cudaError_t (> 0) or one of these (< 0).
#define RF_ERR_BAD_ARG (-1)
#define RF_ERR_UNSUPPORTED (-2)

// ---------------------------------------------------------------- programmatic dependent launch
// Kernels of a step run back to back on one stream.  With the launch attribute below a kernel may be
// scheduled while its predecessor is still running: it executes its set-up (and whatever does not
// depend on the predecessor, above all streaming weights into shared memory) and then blocks in
// pdl_wait() until the predecessor has completed and its writes are visible.  Every kernel of this
// library calls pdl_wait() before it reads anything another kernel of the step wrote and before it
// writes anything at all; what it touches earlier is only weights, the step descriptor and block
// tables, which no kernel of a step writes.  Launched without the attribute, both calls do nothing.
//
// Pointers to what another kernel of the step wrote are named in the call (or are not __restrict__): the compiler takes loads
// through a const __restrict__ parameter for loads of what nobody writes, and may move them up across the wait.  The call hands the
// pointer back as a new one that it knows nothing of but that it is global, so what is read through it is read after the wait; the
// parameters that kernels write through keep their __restrict__.  A pointer formed from the parameter before the wait is named itself.
// What it costs (ms a step, before and after): 7B decoding 2.45, 2.45 at batch 1 and 3.35, 3.35 at batch 64, Rifizen at batch 64 0.737,
// 0.749, a Vilulorn prompt of 2,048 tokens 2.78, 2.89 (width 2,048).
template <typename T>
__device__ __forceinline__ void rf_read_from_here(T*& p) {
    size_t g = __cvta_generic_to_global(p);
    asm volatile("" : "+l"(g));
    p = static_cast<T*>(__cvta_global_to_generic(g));
}
template <typename T>
__device__ __forceinline__ void rf_read_from_here(const T* __restrict__& p) {
    size_t g = __cvta_generic_to_global(p);
    asm volatile("" : "+l"(g));
    p = static_cast<const T*>(__cvta_global_to_generic(g));
}
template <typename... P>
__device__ __forceinline__ void pdl_wait(P&... written_before) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    (rf_read_from_here(written_before), ...);
}
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

static int g_rf_pdl = 0;
extern "C" void rf_set_pdl(int on) { g_rf_pdl = on; }

template <typename... KArgs, typename... Args>
static cudaError_t rf_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                             Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (g_rf_pdl) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// The same with a thread-block cluster of `cluster` CTAs along x (grid.x a multiple of it).
template <typename... KArgs, typename... Args>
static cudaError_t rf_launch_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                     int cluster, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_rf_pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// A host-side note of what has been set on each device: a kernel's attributes (its limit of shared memory, the cluster sizes it may
// have) hold for the device that was current when they were set, and a process may run models on several.
template <typename T>
struct PerDevice {
    T at[64] = {};
    T& here() {
        int dev = 0;
        cudaGetDevice(&dev);
        return at[dev & 63];
    }
};

#define RF_LAUNCH_CHECK()                         \
    do {                                          \
        cudaError_t e__ = cudaGetLastError();     \
        if (e__ != cudaSuccess) return (int)e__;  \
    } while (0)

template <typename T> struct Cvt;
template <> struct Cvt<float> {
    static __device__ __forceinline__ float to_f32(float v) { return v; }
    static __device__ __forceinline__ float from_f32(float v) { return v; }
};
template <> struct Cvt<__nv_bfloat16> {
    static __device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
    static __device__ __forceinline__ __nv_bfloat16 from_f32(float v) { return __float2bfloat16_rn(v); }
};

// A norm weight or bias may be stored in 32-bit or in bfloat16 whatever the compute dtype.
__device__ __forceinline__ float load_vec(const void* p, int is_f32, int i) {
    return is_f32 ? reinterpret_cast<const float*>(p)[i]
                  : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Four numbers of each of the lanes l, l ^ 8, l ^ 16, l ^ 24: out[k] = number r of the lane 8 k + l % 8, where r = lane / 8.
__device__ __forceinline__ void quad_trade(const float* x, float* out, int r) {
    const bool up1 = r & 1, up2 = r & 2;
    // lanes 8 apart trade odd against even numbers: e[i] is number 2 i + (r & 1) of the even lane, o[i] of the odd one
    float e[2], o[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float got = __shfl_xor_sync(0xffffffffu, up1 ? x[2 * i] : x[2 * i + 1], 8);
        e[i] = up1 ? got : x[2 * i];
        o[i] = up1 ? x[2 * i + 1] : got;
    }
    const float ge = __shfl_xor_sync(0xffffffffu, up2 ? e[0] : e[1], 16), go = __shfl_xor_sync(0xffffffffu, up2 ? o[0] : o[1], 16);
    out[0] = up2 ? ge : e[0]; out[1] = up2 ? go : o[0];
    out[2] = up2 ? e[1] : ge; out[3] = up2 ? o[1] : go;
}

// Block-wide sum; every thread gets the result. `red` is shared scratch of >= 33 floats.
// The tree is fixed by blockDim alone, so the value does not depend on what else runs.
__device__ __forceinline__ float block_sum(float v, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < nwarp ? red[lane] : 0.f;
        t = warp_sum(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}
__device__ __forceinline__ float block_max(float v, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < nwarp ? red[lane] : -INFINITY;
        t = warp_max(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}
