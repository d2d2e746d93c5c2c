// shade.cuh — the integrand over the culled disc lists, for every kernel that
// evaluates samples (the integrand kernels, and the values kernels that follow place in
// the render loops).
#pragma once

#include "integrand.h"

// Disc culling: the image is cut into MDAS_CULL_TILES x MDAS_CULL_TILES tiles
// and every tile keeps a list of the discs that may cover a sample in it, with a
// margin that absorbs rounding, in the order in which the full scan tests them.
// Shading then tests only those discs, so the first covering disc (and every
// value) is the one the full scan finds.
//
// A tile's list: 32-bit words; word 0 the number of discs n, word 1 + j the discs
// 2j (low half) and 2j + 1 (high half) of the list.
#define MDAS_CULL_TILES 64
__host__ __device__ inline int mdas_cull_stride(int count) { return 1 + (count + 1) / 2; }  // words per tile

__device__ __forceinline__ int cull_tile(float px, float py) {
    constexpr int T = MDAS_CULL_TILES;
    const int tx = min(max((int)mdas_mul(px, (float)T), 0), T - 1);
    const int ty = min(max((int)mdas_mul(py, (float)T), 0), T - 1);
    return ty * T + tx;
}

// The first disc of a tile's list that covers(p) holds for, or -1; p: the disc's
// first 8 floats.  Two discs are tested at a time: their loads are in flight
// together (a chain of list word and disc for every test is what bounded this).
// Against bit masks of the tile's discs, a word and a disc at a time with 4-byte
// loads: integrand per pass 42.4 -> 29.5 us on 5-D 1920x1080 frames of 256 discs,
// 14.0 -> 12.2 us on 4-D 1024x1024.
template <class Covers>
__device__ __forceinline__ int first_cover(const float* __restrict__ prims, const unsigned* __restrict__ list,
                                           Covers covers) {
    const int n = (int)list[0];
    const float4* __restrict__ discs = reinterpret_cast<const float4*>(prims);
    static_assert(MDAS_PRIM_STRIDE == 12, "three 16-byte chunks per disc");
    for (int j = 0; j < n; j += 2) {
        const unsigned pair = list[1 + (j >> 1)];
        const int k0 = (int)(pair & 0xffffu), k1 = j + 1 < n ? (int)(pair >> 16) : k0;
        const float4 a0 = discs[3 * k0], b0 = discs[3 * k0 + 1];
        const float4 a1 = discs[3 * k1], b1 = discs[3 * k1 + 1];
        const float p0[8] = {a0.x, a0.y, a0.z, a0.w, b0.x, b0.y, b0.z, b0.w};
        const float p1[8] = {a1.x, a1.y, a1.z, a1.w, b1.x, b1.y, b1.z, b1.w};
        const bool h0 = covers(p0), h1 = covers(p1);
        if (h0) return k0;
        if (h1) return k1;
    }
    return -1;
}

// mdas_shade over the tile's candidate discs: the same tests in the same order
// as the full scans of integrand.h (the direct-light kind is not culled).
__device__ __forceinline__ void shade_culled(const MdasScene& sc, const float* __restrict__ prims,
                                             const unsigned* __restrict__ cull, const float* c, float* out) {
    const float px = mdas_div(c[0], sc.scaleX);
    const float py = mdas_div(c[1], sc.scaleY);
    const unsigned* list = cull + (size_t)cull_tile(px, py) * mdas_cull_stride(sc.count);
    int k = -1;
    if (sc.kind == MDAS_SCENE_DISCS_MB) {
        const float t = c[2];
        k = first_cover(prims, list, [&](const float* p) { return mdas_disc_mb_covers(p, px, py, t) != 0; });
    } else if (sc.kind == MDAS_SCENE_DISCS_DOF || sc.kind == MDAS_SCENE_DISCS_MBDOF) {
        const int moving = sc.kind == MDAS_SCENE_DISCS_MBDOF;
        float t, lx, ly, wx, wy;
        mdas_dof_ray(&sc, c, moving, &t, &lx, &ly, &wx, &wy);
        k = first_cover(prims, list,
                        [&](const float* p) { return mdas_disc_dof_covers(p, lx, ly, wx, wy, t, moving) != 0; });
    } else {
        mdas_shade(&sc, prims, c, out);
        return;
    }
    out[0] = out[1] = out[2] = sc.background;
    if (k >= 0) {
        const float4 rgb = reinterpret_cast<const float4*>(prims)[3 * k + 2];
        out[0] = rgb.x;
        out[1] = rgb.y;
        out[2] = rgb.z;
    }
}
