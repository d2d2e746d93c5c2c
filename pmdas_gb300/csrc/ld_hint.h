// ld_hint.h — 16-byte global loads with an L2 prefetch-size hint.
//
// PTX `ld .L2::64B / .L2::128B / .L2::256B` (HINT 0: no qualifier).  A leaf
// record's head (node and box: 48 bytes at D = 4) read with the 64-byte hint
// fetches its two sectors only; without a hint, streams over the 128-byte
// records fetched more.  The "memory" clobber keeps the load ordered with the
// thread's own stores.
#pragma once

#include <cuda_runtime.h>

template <int HINT>
__device__ __forceinline__ float4 ld4_hint(const float* p) {
    float4 v;
    if constexpr (HINT == 64)
        asm volatile("ld.global.L2::64B.v4.f32 {%0,%1,%2,%3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    else if constexpr (HINT == 128)
        asm volatile("ld.global.L2::128B.v4.f32 {%0,%1,%2,%3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    else if constexpr (HINT == 256)
        asm volatile("ld.global.L2::256B.v4.f32 {%0,%1,%2,%3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    else
        v = *reinterpret_cast<const float4*>(p);
    return v;
}

// The value of sample idx (3 floats at 4-byte alignment), gathered at random; for words
// that the calling kernel does not write (read-only loads, and nothing orders them with
// its stores; it may write other words of the same buffer, as render_sample does).  Without the hint L2 fetches
// 128 bytes for the 12; with it the errors pass moves a third less DRAM traffic:
// 87.5 -> 82.3 us per pass on a 4-D 4K frame at 16 spp, 15.5 -> 13.7 us on 4-D
// 1024x1024, and integrate 4.60 -> 4.50 ms and 0.240 -> 0.237 ms.  Measured and
// slower (84-88 us, 14-15.6 us): the same loads kept in program order (volatile),
// and one or two aligned 16-byte loads in place of the three.
__device__ __forceinline__ float3 ld_value64(const float* __restrict__ values, int idx) {
    const float* p = values + 3 * (size_t)idx;
    float3 v;
    asm("ld.global.nc.L2::64B.f32 %0, [%1];" : "=f"(v.x) : "l"(p));
    asm("ld.global.nc.L2::64B.f32 %0, [%1];" : "=f"(v.y) : "l"(p + 1));
    asm("ld.global.nc.L2::64B.f32 %0, [%1];" : "=f"(v.z) : "l"(p + 2));
    return v;
}

// The first NF floats of a 16-byte aligned record (rounded up to 16-byte
// chunks: the record must extend that far) with the 64-byte hint.
template <int NF>
__device__ __forceinline__ void ld_head64(const float* p, float (&out)[(NF + 3) / 4 * 4]) {
#pragma unroll
    for (int k = 0; k < (NF + 3) / 4; ++k) {
        const float4 v = ld4_hint<64>(p + 4 * k);
        out[4 * k] = v.x;
        out[4 * k + 1] = v.y;
        out[4 * k + 2] = v.z;
        out[4 * k + 3] = v.w;
    }
}

// The first H4 16-byte chunks of the 32 consecutive records [first, first + 32) (of
// L; `stride` floats apart), read by the warp into wbuf (record r's at wbuf + r * H4)
// with each load covering consecutive chunks: a third of the lines that 32 lanes
// each reading their own record touch.
template <int H4>
__device__ __forceinline__ void warp_heads64(const float* __restrict__ nb, size_t stride, int first, int L,
                                             float4* wbuf) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < H4; ++q) {
        const int c = q * 32 + lane;
        const int rec = c / H4;
        if (first + rec < L) wbuf[c] = ld4_hint<64>(nb + (size_t)(first + rec) * stride + 4 * (c - rec * H4));
    }
    __syncwarp();
}
