// Shared device helpers for the sm_100a decode kernels.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>

#define B200_WARP 32

// ---- programmatic dependent launch -------------------------------------
// A kernel launched with the programmatic-stream-serialization attribute may
// begin while its predecessor drains. Everything before pdl_wait() must touch
// only memory no earlier kernel writes (here: weights); pdl_wait() returns once
// the predecessor grid has completed and its stores are visible.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch of a kernel that calls pdl_wait() before it touches anything an earlier kernel writes: it may be scheduled while its
// predecessor drains, if that one says so (pdl_launch_dependents), and otherwise starts after it as usual.
template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// ---- order of blocks ---------------------------------------------------
// Blocks of a one-dimensional grid take items that are numbered from the heaviest to the lightest. Two that start on an SM together never wait for
// one another's end: with `two`, the second round counts from its light end, so that every SM gets about the same (rows of a causal
// attention: 9 tiles of 64 an SM at most for 509 rows of 32 heads, 12 in order of heads and tiles).
__device__ __forceinline__ int rank_by_weight(bool two)
{
    constexpr int SMS = 148;
    const int id = blockIdx.x, second = two ? min(2 * SMS, (int)gridDim.x) - SMS : 0;
    return id >= SMS && id < SMS + second ? 2 * SMS + second - 1 - id : id;
}

// ---- memory ------------------------------------------------------------
// Streaming 16-byte load that does not allocate in L1 (weights are read once).
__device__ __forceinline__ uint4 ldg_stream_16(const void *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned short ldg_stream_u16(const void *p) {
    unsigned short v;
    asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned ld_acquire_sys(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_sys(unsigned *p, unsigned v) {
    asm volatile("st.release.sys.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

// ---- pairs of fp32 values in one instruction ------------------------------
__device__ __forceinline__ void add_pair(float &a, float &b, float x, float y) {
    asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\tadd.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}"
        : "+f"(a), "+f"(b) : "f"(x), "f"(y));
}
__device__ __forceinline__ void mul_pair(float &a, float &b, float x, float y) {
    asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\tmul.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}"
        : "+f"(a), "+f"(b) : "f"(x), "f"(y));
}

// ---- reductions --------------------------------------------------------
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
// Sum over the whole block; every thread gets the result. `red` holds >= 33 floats.
__device__ __forceinline__ float block_sum(float v, float *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();                       // protect `red` from a previous use
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < nw ? red[lane] : 0.0f;
        t = warp_sum(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

// ---- clusters ------------------------------------------------------------
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Sum, in rank order, of the four floats at shared-memory address `addr` (16-byte aligned) of n <= 8 blocks of the cluster: ranks
// first, first + step, ... All loads are in flight at once: one by one they cost a round trip of 0.25 us each.
__device__ __forceinline__ float4 sum_ranks4(uint32_t addr, int n, int first, int step) {
    float4 v[8];
#pragma unroll
    for (int z = 0; z < 8; ++z) {
        if (z < n) {
            uint32_t at;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(first + z * step));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[z].x), "=f"(v[z].y), "=f"(v[z].z), "=f"(v[z].w) : "r"(at));
        }
    }
    float4 s = v[0];
#pragma unroll
    for (int z = 1; z < 8; ++z)
        if (z < n) { s.x += v[z].x; s.y += v[z].y; s.z += v[z].z; s.w += v[z].w; }
    return s;
}

// Bounded wait for a flag another GPU writes. Returns false when it gave up.
#define B200_SPIN_LIMIT 4000000
__device__ __forceinline__ bool wait_flag_ge(const unsigned *flag, unsigned want, int limit = B200_SPIN_LIMIT) {
    for (int it = 0; it < limit; ++it) {
        // signed distance so that a wrapped counter still compares correctly
        if ((int)(ld_acquire_sys(flag) - want) >= 0) return true;
        __nanosleep(20);
    }
    return false;
}
