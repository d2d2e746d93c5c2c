// integrand.cu — the analytic integrand kernel and the seeded scene generators.
//
// Stands in for the reference's OptiX launch over the sample buffer
// (launchSubframe, SDK/optixMotionBlur/optixMotionBlur.cpp:420-470): evaluates
// samples [offset, offset + count) of a grid's coordinate buffer into its value
// buffer.  Compiled with strict IEEE flags so the CPU oracle, which shares
// integrand.h, gets identical values.
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include <algorithm>
#include <atomic>
#include <vector>
#include "integrand.h"
#include "grid_types.h"
#include "scene.h"
#include "shade.cuh"

namespace {

// ---- disc culling ---------------------------------------------------------------------
bool mdas_culled_kind(int kind) {
    return kind == MDAS_SCENE_DISCS_MB || kind == MDAS_SCENE_DISCS_DOF || kind == MDAS_SCENE_DISCS_MBDOF;
}

// Can disc p cover a sample whose image point lies in [x0, x1] x [y0, y1] (in
// [0, 1] image units)?  Motion blur: the disc's centre sweeps the box between
// its positions at t = 0 and t = 1.  Depth of field: the ray meets the disc's
// plane at s * focal * (nx * filmHalfW, ny * filmHalfH) + (1 - s) * lens point,
// s = depth / focal, |lens point| <= lensRadius.  So the disc can be hit only
// if the distance between those two boxes is within r (+ |1 - s| * lensRadius).
// NaNs keep the disc (only a certain miss drops it).
__device__ bool cull_may_cover(const MdasScene& sc, const float* p, float x0, float x1, float y0, float y1) {
    const bool moving = sc.kind != MDAS_SCENE_DISCS_DOF;
    const float vx = moving ? p[4] : 0.0f, vy = moving ? p[5] : 0.0f;
    const float cx0 = p[0] + fminf(0.0f, vx), cx1 = p[0] + fmaxf(0.0f, vx);
    const float cy0 = p[1] + fminf(0.0f, vy), cy1 = p[1] + fmaxf(0.0f, vy);
    float bx0 = x0, bx1 = x1, by0 = y0, by1 = y1, reach = sqrtf(fmaxf(p[7], 0.0f));
    float scale = 1.0f;
    if (sc.kind != MDAS_SCENE_DISCS_MB) {
        const float s = p[6];
        const float ax = s * sc.focalDistance * sc.filmHalfW, ay = s * sc.focalDistance * sc.filmHalfH;
        const float ux0 = ax * (2.0f * x0 - 1.0f), ux1 = ax * (2.0f * x1 - 1.0f);
        const float uy0 = ay * (2.0f * y0 - 1.0f), uy1 = ay * (2.0f * y1 - 1.0f);
        bx0 = fminf(ux0, ux1);
        bx1 = fmaxf(ux0, ux1);
        by0 = fminf(uy0, uy1);
        by1 = fmaxf(uy0, uy1);
        reach += fabsf(1.0f - s) * fabsf(sc.lensRadius);
        scale += fabsf(ax) + fabsf(ay) + fabsf(sc.lensRadius);
    }
    scale += fabsf(cx0) + fabsf(cx1) + fabsf(cy0) + fabsf(cy1) + reach;
    const float dx = fmaxf(fmaxf(cx0 - bx1, bx0 - cx1), 0.0f);
    const float dy = fmaxf(fmaxf(cy0 - by1, by0 - cy1), 0.0f);
    const float dist = sqrtf(dx * dx + dy * dy);
    return !(dist > reach + 1.0e-3f * scale);
}

// One warp per tile: its lanes test 32 discs at a time, in the order in which the
// full scan tests them (integrand.h: motion blur from the last disc, depth of field
// from the first), and append those kept to the tile's list (shade.cuh).
__global__ void __launch_bounds__(256) k_build_cull(MdasScene sc, const float* __restrict__ prims,
                                                     unsigned* __restrict__ lists) {
    constexpr int T = MDAS_CULL_TILES;
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile < T * T; tile += warps) {
        const int tx = tile % T, ty = tile / T;
        const float pad = 1.0e-4f;
        const float x0 = (float)tx / T - pad, x1 = (float)(tx + 1) / T + pad;
        const float y0 = (float)ty / T - pad, y1 = (float)(ty + 1) / T + pad;
        unsigned* list = lists + (size_t)tile * mdas_cull_stride(sc.count);
        unsigned short* entries = reinterpret_cast<unsigned short*>(list + 1);
        int n = 0;
        for (int base = 0; base < sc.count; base += 32) {
            const int i = base + lane;
            const int k = sc.kind == MDAS_SCENE_DISCS_MB ? sc.count - 1 - i : i;
            const bool may = i < sc.count && cull_may_cover(sc, prims + MDAS_PRIM_STRIDE * k, x0, x1, y0, y1);
            const unsigned m = __ballot_sync(0xffffffffu, may);
            if (may) entries[n + __popc(m & ((1u << lane) - 1u))] = (unsigned short)k;
            n += __popc(m);
        }
        if (lane == 0) list[0] = (unsigned)n;
    }
}

template <int D>
__global__ void __launch_bounds__(256) k_evaluate(MdasScene sc, const float* __restrict__ prims,
                                                   const unsigned* __restrict__ cull, const float* __restrict__ coords,
                                                   float* __restrict__ values, const MdasCounts* __restrict__ counts,
                                                   int offset, int count) {
    // a full scan reads every primitive for every sample: staged in shared
    // memory; a culled scan reads a few, straight from the (L1-resident) table
    extern __shared__ float s_prims[];
    if (!cull) {
        const int nfl = sc.count * MDAS_PRIM_STRIDE;
        for (int k = threadIdx.x; k < nfl; k += blockDim.x) s_prims[k] = prims[k];
        __syncthreads();
    }
    if (counts) {  // the samples the last adaptive pass added
        offset = counts->N - counts->newN;
        count = counts->newN;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const size_t s = (size_t)offset + i;
        float c[D];
#pragma unroll
        for (int d = 0; d < D; ++d) c[d] = coords[s * D + d];
        float out[3];
        if (cull) shade_culled(sc, prims, cull, c, out);
        else mdas_shade(&sc, s_prims, c, out);
        values[3 * s + 0] = out[0];
        values[3 * s + 1] = out[1];
        values[3 * s + 2] = out[2];
    }
}

// Batched integrand over the images' initial samples: chunks of 256 samples across
// the images of one launch
// (same enumeration scheme as the batched MDAS kernels); primitives are read
// from global memory (L1/L2-resident), as several scenes share a launch.
template <int D>
__global__ void __launch_bounds__(256) k_evaluate_batch(const MdasBatchScene* __restrict__ scenes, int n) {
    __shared__ int s_pre[257];
    __shared__ unsigned s_warp[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned v = 0;
    if (threadIdx.x < (unsigned)n) v = (unsigned)((scenes[threadIdx.x].initialSamples + 255) / 256);
    unsigned incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        unsigned w = lane < 8 ? s_warp[lane] : 0u;
        for (int o = 1; o < 8; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < 8) s_warp[lane] = w;
    }
    __syncthreads();
    if (threadIdx.x < (unsigned)n) s_pre[threadIdx.x] = (int)((warp ? s_warp[warp - 1] : 0u) + incl - v);
    if (threadIdx.x == 0) s_pre[n] = (int)s_warp[7];
    __syncthreads();
    const int total = s_pre[n];
    for (int ch = blockIdx.x; ch < total; ch += gridDim.x) {
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_pre[mid] <= ch) lo = mid;
            else hi = mid - 1;
        }
        const MdasBatchScene& b = scenes[lo];
        const int k = (ch - s_pre[lo]) * 256 + threadIdx.x;
        if (k < b.initialSamples) {
            const size_t s = (size_t)k;
            float c[D];
#pragma unroll
            for (int d = 0; d < D; ++d) c[d] = b.coords[s * D + d];
            float out[3];
            if (b.cull) shade_culled(b.sc, b.prims, b.cull, c, out);
            else mdas_shade(&b.sc, b.prims, c, out);
            b.values[3 * s + 0] = out[0];
            b.values[3 * s + 1] = out[1];
            b.values[3 * s + 2] = out[2];
        }
    }
}

// The 64-bit LCG (Knuth's MMIX constants) that the reference image and the true
// errors draw from, 24 random bits per float.  A stream belongs to a pixel or a
// leaf; the lanes that share it each take every T-th sample and jump over the
// draws of the others (n draws take a state s to A_n s + C_n).
struct Lcg64 {
    unsigned long long s;
    __device__ float next() {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (float)(unsigned)(s >> 40) * (1.0f / 16777216.0f);
    }
};

struct Lcg64Jump {
    unsigned long long A, C;
    __device__ explicit Lcg64Jump(unsigned n) : A(1ull), C(0ull) {
        unsigned long long a = 6364136223846793005ull, c = 1442695040888963407ull;
        for (; n; n >>= 1) {  // (A, C) composed with the (a, c) of the bits of n
            if (n & 1u) {
                A = A * a;
                C = C * a + c;
            }
            c = c * a + c;
            a = a * a;
        }
    }
    __device__ void apply(Lcg64& r) const { r.s = r.s * A + C; }
};

// Sum over the T lanes that share a stream, on every one of them.
template <int T>
__device__ __forceinline__ double lanes_sum(double v) {
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Reference image of an integrand: `spp` samples per pixel, the image plane
// stratified on a sqrt(spp) x sqrt(spp) grid with jitter, the other dimensions
// uniform, radiance accumulated in FP64.  T lanes share a pixel's stream and
// its samples (reference_lanes).
// cull (may be null): the scene's culling lists; the samples' values are the full
// scan's either way.
// 4-D depth of field, 256 discs, 256 x 256 at 1024 spp: 0.85 ms; 12.8 ms with one
// thread per pixel testing every disc from the front.
template <int D, int T>
__global__ void __launch_bounds__(256) k_reference_image(MdasScene sc, const float* __restrict__ prims,
                                                          const unsigned* __restrict__ cull, int width, int height,
                                                          int strata, unsigned long long seed,
                                                          double* __restrict__ out) {
    extern __shared__ float s_prims[];
    if (!cull) {
        const int nfl = sc.count * MDAS_PRIM_STRIDE;
        for (int k = threadIdx.x; k < nfl; k += blockDim.x) s_prims[k] = prims[k];
        __syncthreads();
    }
    const int P = width * height;
    const int sub = threadIdx.x & (T - 1);
    const int spp = strata * strata;
    const Lcg64Jump start(sub * D), skip((T - 1) * D);
    const int di = T / strata, dj = T - di * strata;
    const float px = sc.scaleX / (float)width, py = sc.scaleY / (float)height;
    const int groups = gridDim.x * (blockDim.x / T);
    // (every lane of a warp runs the same iterations: the sums are exchanged by
    // whole warps)
    for (int first = (blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / T; first < P; first += groups) {
        const int p = first + ((threadIdx.x & 31) / T);
        double acc[3] = {0.0, 0.0, 0.0};
        if (p < P) {
            const int x = p % width, y = p / width;
            Lcg64 rng{seed ^ (0x9E3779B97F4A7C15ull * (unsigned long long)(p + 1))};
            start.apply(rng);
            int i = sub / strata, j = sub - i * strata;
            for (int q = sub; q < spp; q += T) {
                float c[D];
                c[0] = ((float)x + ((float)i + rng.next()) / (float)strata) * px;
                c[1] = ((float)y + ((float)j + rng.next()) / (float)strata) * py;
#pragma unroll
                for (int d = 2; d < D; ++d) c[d] = rng.next();
                if constexpr (T > 1) skip.apply(rng);
                float v[3];
                if (cull) shade_culled(sc, prims, cull, c, v);
                else mdas_shade(&sc, s_prims, c, v);
                acc[0] += (double)v[0];
                acc[1] += (double)v[1];
                acc[2] += (double)v[2];
                i += di;
                j += dj;
                if (j >= strata) {
                    j -= strata;
                    ++i;
                }
            }
        }
        const double inv = 1.0 / ((double)strata * (double)strata);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double sum = lanes_sum<T>(acc[k]);
            if (sub == 0 && p < P) out[3 * (size_t)p + k] = sum * inv;
        }
    }
}

// True reconstruction error of each leaf (the training target of the learned
// leaf priority): the leaf's mean sample value against the integrand's mean
// over the leaf's box, estimated from `samples` uniform points with FP64
// accumulation; err = volume * sum_c |mean_c - ref_c| / sqrt(ref_c^2 + 1e-2),
// in the units of the plain error (a relative deviation times the volume,
// image axes in pixels).  T lanes share a leaf's points (leaf_lanes); from 4 lanes on
// one lane per colour channel finishes it (FP64 division and square root): 16,384
// leaves x 64 points of a 5-D scene of 256 discs 0.93 -> 0.045 ms, the culling included.
// cull: as k_reference_image; a leaf that reaches out of the scene's domain (of a grid of
// another scale, of a loaded state) is scanned in full: the lists are for points inside.
template <int D, int T>
__global__ void __launch_bounds__(256) k_leaf_true_errors(MdasScene sc, const float* __restrict__ prims,
                                                           const unsigned* __restrict__ cull, MdasDeviceGrid g,
                                                           const int* __restrict__ leaves, int L, int samples,
                                                           unsigned long long seed, float* __restrict__ out) {
    extern __shared__ float s_prims[];
    if (!cull) {
        const int nfl = sc.count * MDAS_PRIM_STRIDE;
        for (int k = threadIdx.x; k < nfl; k += blockDim.x) s_prims[k] = prims[k];
        __syncthreads();
    }
    const int sub = threadIdx.x & (T - 1);
    const Lcg64Jump start(sub * D), skip((T - 1) * D);
    const int groups = gridDim.x * (blockDim.x / T);
    for (int first = (blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / T; first < L; first += groups) {
        const int row = first + ((threadIdx.x & 31) / T);
        double acc[3] = {0.0, 0.0, 0.0};
        float mean[3] = {0.0f, 0.0f, 0.0f};
        float volume = 1.0f;
        if (row < L) {
            const int i = leaves ? leaves[row] : row;
            const float* nb = g.nb + (size_t)i * g.nbFloats;
            const int idx[4] = {reinterpret_cast<const int*>(nb)[0], reinterpret_cast<const int*>(nb)[1],
                                reinterpret_cast<const int*>(nb)[2], reinterpret_cast<const int*>(nb)[3]};
            float mn[D], mx[D];
            bool inside = true;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                mn[d] = nb[4 + d];
                mx[d] = nb[4 + D + d];
                volume *= mx[d] - mn[d];
                inside = inside && mn[d] >= 0.0f && mx[d] <= (d == 0 ? sc.scaleX : d == 1 ? sc.scaleY : 1.0f);
            }
            int n = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (idx[k] < 0) continue;
#pragma unroll
                for (int c = 0; c < 3; ++c) mean[c] += g.values[3 * (size_t)idx[k] + c];
                ++n;
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) mean[c] = n ? mean[c] / (float)n : 0.0f;
            Lcg64 rng{seed ^ (0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1))};
            start.apply(rng);
            for (unsigned s = sub; s < (unsigned)samples; s += T) {  // (past 2^31 - 1 near its end)
                float c[D];
#pragma unroll
                for (int d = 0; d < D; ++d) c[d] = mn[d] + rng.next() * (mx[d] - mn[d]);
                if constexpr (T > 1) skip.apply(rng);
                float v[3];
                // (a branch for each place of the primitives: shared-memory loads stay such)
                if (!cull) mdas_shade(&sc, s_prims, c, v);
                else if (inside) shade_culled(sc, prims, cull, c, v);
                else mdas_shade(&sc, prims, c, v);
                acc[0] += (double)v[0];
                acc[1] += (double)v[1];
                acc[2] += (double)v[2];
            }
        }
        // the sum over the channels, on the leaf's first lane
        double e = 0.0;
        if constexpr (T == 1) {
            if (row < L) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const double ref = acc[c] / (double)samples;
                    e += fabs((double)mean[c] - ref) / sqrt(ref * ref + 1e-2);
                }
            }
        } else {
            static_assert(T >= 4, "a lane per channel");
#pragma unroll
            for (int c = 0; c < 3; ++c) acc[c] = lanes_sum<T>(acc[c]);
            // lanes 0..2 of the leaf: one channel each
            const double a = sub == 0 ? acc[0] : sub == 1 ? acc[1] : acc[2];
            const float m = sub == 0 ? mean[0] : sub == 1 ? mean[1] : mean[2];
            if (row < L && sub < 3) {
                const double ref = a / (double)samples;
                e = fabs((double)m - ref) / sqrt(ref * ref + 1e-2);
            }
            const double e1 = __shfl_down_sync(0xffffffffu, e, 1), e2 = __shfl_down_sync(0xffffffffu, e, 2);
            e = (e + e1) + e2;
        }
        if (row < L && sub == 0) out[row] = (float)(e * (double)volume);
    }
}

}  // namespace

uint64_t mdas_next_scene_id() {
    static std::atomic<uint64_t> last{0};
    return ++last;
}

namespace {

// splitmix64 (Steele, Lea & Flood, "Fast splittable pseudorandom number
// generators", OOPSLA 2014): the documented stream every scene is drawn from.
struct SplitMix64 {
    uint64_t s;
    uint64_t next() {
        uint64_t z = (s += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    }
    // 24 random bits -> [0, 1)
    float uniform() { return (float)(next() >> 40) * (1.0f / 16777216.0f); }
    float range(float a, float b) { return a + (b - a) * uniform(); }
};

}  // namespace

namespace {
template <int T>
cudaError_t launch_leaf_true_errors(const MdasScene& sc, const float* d_prims, const unsigned* cull,
                                    const MdasDeviceGrid& g, const int* leaves, int L, int samples,
                                    unsigned long long seed, float* out, cudaStream_t s) {
    const size_t smem = cull ? 0 : sizeof(float) * MDAS_PRIM_STRIDE * (size_t)sc.count;
    const int perBlock = 256 / T;
    const int64_t want = ((int64_t)L + perBlock - 1) / perBlock;
    const int grid = (int)(want < 65535 ? want : 65535);
    switch (g.D) {
        case 3: k_leaf_true_errors<3, T><<<grid, 256, smem, s>>>(sc, d_prims, cull, g, leaves, L, samples, seed, out); break;
        case 4: k_leaf_true_errors<4, T><<<grid, 256, smem, s>>>(sc, d_prims, cull, g, leaves, L, samples, seed, out); break;
        case 5: k_leaf_true_errors<5, T><<<grid, 256, smem, s>>>(sc, d_prims, cull, g, leaves, L, samples, seed, out); break;
        case 6: k_leaf_true_errors<6, T><<<grid, 256, smem, s>>>(sc, d_prims, cull, g, leaves, L, samples, seed, out); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Lanes per leaf of the true errors: 1, 4 or 8.  Lanes are shared
//   * as far as that is needed to fill the GPU and each has 4 samples (us with 1, 4, 8
//     lanes, 256 discs: 20,000 leaves with 16 points 66, 53, 58, with 64 points 132, 72,
//     72; 665,000 leaves with 1 point 212, 333, 643, with 64 points 804, 799, 1037; 4
//     spheres, 100,000 leaves with 16 points 107, 102, 130), 4 on the fewest leaves
//     whatever they have (5000 with 1 point 44, 38, 46);
//   * heavy: as reference_lanes (256 spheres, 629,000 leaves: with 1 point 503, 1400,
//     2472, with 4 points 1749, 1416, 2492, with 16 points 6721, 5264, 4784).
int leaf_lanes(int L, int samples, bool heavy) {
    int best = 4LL * L <= 1 << 15 ? 4 : 1;
    for (int t = 4; t <= 8; t *= 2) {
        const bool even = ((int64_t)samples + t - 1) / t * t * 8 <= (int64_t)samples * 9;
        if (heavy ? even : (int64_t)L * t <= 1 << 19 && samples / t >= 4) best = t;
    }
    return best;
}
}  // namespace

cudaError_t mdas_launch_leaf_true_errors(const MdasScene& sc, const float* d_prims, const unsigned* cull,
                                         const MdasDeviceGrid& g, const int* leaves, int L, int samples,
                                         unsigned long long seed, float* out, cudaStream_t s) {
    if (L <= 0) return cudaSuccess;
    if (!mdas_culled_kind(sc.kind)) cull = nullptr;
    switch (leaf_lanes(L, samples, !cull && sc.count >= 32)) {
        case 4: return launch_leaf_true_errors<4>(sc, d_prims, cull, g, leaves, L, samples, seed, out, s);
        case 8: return launch_leaf_true_errors<8>(sc, d_prims, cull, g, leaves, L, samples, seed, out, s);
        default: return launch_leaf_true_errors<1>(sc, d_prims, cull, g, leaves, L, samples, seed, out, s);
    }
}

size_t mdas_cull_words(const MdasScene& sc) {
    if (!mdas_culled_kind(sc.kind) || sc.count <= 0) return 0;
    return (size_t)MDAS_CULL_TILES * MDAS_CULL_TILES * (size_t)mdas_cull_stride(sc.count);
}

cudaError_t mdas_launch_build_cull(const MdasScene& sc, const float* d_prims, unsigned* lists, cudaStream_t s) {
    if (mdas_cull_words(sc) == 0) return cudaSuccess;
    if (!lists) return cudaErrorInvalidValue;
    // (8 warps per block, one tile per warp)
    k_build_cull<<<MDAS_CULL_TILES * MDAS_CULL_TILES / 8, 256, 0, s>>>(sc, d_prims, lists);
    return cudaGetLastError();
}

cudaError_t mdas_launch_evaluate(const MdasScene& sc, const float* d_prims, const unsigned* cull, const float* coords,
                                 float* values, int dim, const MdasCounts* counts, int offset, int count, int grid,
                                 cudaStream_t s) {
    if (grid <= 0) grid = 1;
    if (dim < sc.dim) return cudaErrorInvalidValue;
    if (!mdas_culled_kind(sc.kind)) cull = nullptr;
    const size_t smem = cull ? 0 : sizeof(float) * MDAS_PRIM_STRIDE * (size_t)sc.count;
    switch (dim) {
        case 3: k_evaluate<3><<<grid, 256, smem, s>>>(sc, d_prims, cull, coords, values, counts, offset, count); break;
        case 4: k_evaluate<4><<<grid, 256, smem, s>>>(sc, d_prims, cull, coords, values, counts, offset, count); break;
        case 5: k_evaluate<5><<<grid, 256, smem, s>>>(sc, d_prims, cull, coords, values, counts, offset, count); break;
        case 6: k_evaluate<6><<<grid, 256, smem, s>>>(sc, d_prims, cull, coords, values, counts, offset, count); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t mdas_launch_evaluate_batch(const MdasBatchScene* scenes, int n, int D, int grid, cudaStream_t s) {
    switch (D) {
        case 3: k_evaluate_batch<3><<<grid, 256, 0, s>>>(scenes, n); break;
        case 4: k_evaluate_batch<4><<<grid, 256, 0, s>>>(scenes, n); break;
        case 5: k_evaluate_batch<5><<<grid, 256, 0, s>>>(scenes, n); break;
        case 6: k_evaluate_batch<6><<<grid, 256, 0, s>>>(scenes, n); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

namespace {
template <int T>
cudaError_t launch_reference_image(const MdasScene& sc, const float* d_prims, const unsigned* cull, int width,
                                   int height, int strata, unsigned long long seed, double* out, int sms,
                                   cudaStream_t s) {
    const size_t smem = cull ? 0 : sizeof(float) * MDAS_PRIM_STRIDE * (size_t)sc.count;
    const int64_t want = ((int64_t)width * height * T + 255) / 256;
    const int grid = (int)(want < (int64_t)sms * 16 ? want : (int64_t)sms * 16);
    switch (sc.dim) {
        case 3: k_reference_image<3, T><<<grid, 256, smem, s>>>(sc, d_prims, cull, width, height, strata, seed, out); break;
        case 4: k_reference_image<4, T><<<grid, 256, smem, s>>>(sc, d_prims, cull, width, height, strata, seed, out); break;
        case 5: k_reference_image<5, T><<<grid, 256, smem, s>>>(sc, d_prims, cull, width, height, strata, seed, out); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Lanes per pixel of the reference image.  A pixel's sum over its lanes costs FP64
// additions, of which an SM makes few, so lanes are shared only
//   * as far as that is needed to fill the GPU (2^19 of them) and each has 8 samples
//     (us with 1, 8, 32 lanes; 4 spheres: 256x256 at 1 spp 23, 46, 128, at 64 spp 150,
//     104, 158, at 1024 spp 2086, 1076, 1064; 3840x2160 at 1 spp 184, 2362, 12335;
//     64x64 at 1024 spp 1934, 249, 114), on the smallest images (2^16) up to 8 whatever
//     they have (64x64, 256 discs, at 9 spp 34, 24, 30);
//   * up to 8 on any image where each has 256 samples: the lanes test the same few
//     discs (640x480 at 1024 spp, 256 discs, with 1, 4, 32 lanes: 4165, 3696, 3955);
//   * heavy: in a full scan of many primitives, which a warp leaves together only if its
//     samples are alike, as far as few lanes are left over in the last round (640x480,
//     64 spheres, with 1, 2, 4, 32 lanes: at 4 spp 160, 139, 142, 860, at 9 spp 333, 306,
//     353, 875, at 64 spp 2174, 1822, 1732, 1670; 1920x1080 at 9 spp 1667, 1819, 2212,
//     5864).
int reference_lanes(int64_t pixels, int spp, bool heavy) {
    int best = 1;
    for (int t = 2; t <= 32; t *= 2) {
        const int64_t lanes = pixels * t;
        const bool even = ((int64_t)spp + t - 1) / t * t * 8 <= (int64_t)spp * 9;
        const bool few = t <= 8 && lanes <= 1 << 16 && spp >= t;
        if (few || (heavy ? even && lanes <= (t <= 16 ? 1 << 21 : 1 << 20)
                          : (lanes <= 1 << 19 && spp / t >= 8) || (t <= 8 && spp / t >= 256)))
            best = t;
    }
    return best;
}
}  // namespace

cudaError_t mdas_launch_reference_image(const MdasScene& sc, const float* d_prims, const unsigned* cull, int width,
                                        int height, int strata, unsigned long long seed, double* out, int sms,
                                        cudaStream_t s) {
    if (!mdas_culled_kind(sc.kind)) cull = nullptr;
    const bool heavy = !cull && sc.count >= 32;
    switch (reference_lanes((int64_t)width * height, strata * strata, heavy)) {
        case 2: return launch_reference_image<2>(sc, d_prims, cull, width, height, strata, seed, out, sms, s);
        case 4: return launch_reference_image<4>(sc, d_prims, cull, width, height, strata, seed, out, sms, s);
        case 8: return launch_reference_image<8>(sc, d_prims, cull, width, height, strata, seed, out, sms, s);
        case 16: return launch_reference_image<16>(sc, d_prims, cull, width, height, strata, seed, out, sms, s);
        case 32: return launch_reference_image<32>(sc, d_prims, cull, width, height, strata, seed, out, sms, s);
        default: return launch_reference_image<1>(sc, d_prims, cull, width, height, strata, seed, out, sms, s);
    }
}

// Scene generators.  Draw order is part of the format: the same seed gives the
// same primitives on every machine (host code is built with -ffp-contract=off).
int mdas_generate_scene(int kind, uint64_t seed, int count, float scaleX, float scaleY, int width, int height,
                        MdasScene* sc, std::vector<float>* prims) {
    if (count < 0 || count > MDAS_MAX_PRIMS || width <= 0 || height <= 0) return MDAS_ERR_INVALID;
    *sc = MdasScene();
    sc->kind = kind;
    sc->count = count;
    sc->scaleX = scaleX;
    sc->scaleY = scaleY;
    sc->background = 0.1f;
    // fovy = 45 degrees: tan(pi/8) = sqrt(2) - 1 exactly in real arithmetic
    const float tanHalf = (float)(sqrt(2.0) - 1.0);
    sc->filmHalfH = tanHalf;
    sc->filmHalfW = tanHalf * ((float)width / (float)height);
    sc->focalDistance = 4.0f;
    sc->lensRadius = 0.1f;
    prims->assign((size_t)count * MDAS_PRIM_STRIDE, 0.0f);
    SplitMix64 rng{seed};
    float* p = prims->data();
    switch (kind) {
        case MDAS_SCENE_DISCS_MB: {
            sc->dim = 3;
            for (int k = 0; k < count; ++k) {
                float* q = p + MDAS_PRIM_STRIDE * k;
                q[0] = rng.uniform();             // center x in [0,1)
                q[1] = rng.uniform();             // center y
                q[3] = rng.range(0.02f, 0.08f);   // radius
                q[8] = rng.uniform();             // R
                q[9] = rng.uniform();             // G
                q[10] = rng.uniform();            // B
                q[4] = rng.range(-0.1f, 0.1f);    // velocity x per unit shutter time
                q[5] = rng.range(-0.1f, 0.1f);    // velocity y
                q[7] = q[3] * q[3];
            }
            break;
        }
        case MDAS_SCENE_DISCS_DOF:
        case MDAS_SCENE_DISCS_MBDOF: {
            sc->dim = kind == MDAS_SCENE_DISCS_DOF ? 4 : 5;
            for (int k = 0; k < count; ++k) {
                float* q = p + MDAS_PRIM_STRIDE * k;
                q[2] = rng.range(1.0f, 10.0f);    // depth
                q[3] = rng.range(0.05f, 0.3f);    // radius (world units)
                q[8] = rng.uniform();
                q[9] = rng.uniform();
                q[10] = rng.uniform();
                // center uniform over the view frustum's cross-section at that depth
                q[0] = (2.0f * rng.uniform() - 1.0f) * (q[2] * sc->filmHalfW);
                q[1] = (2.0f * rng.uniform() - 1.0f) * (q[2] * sc->filmHalfH);
                q[6] = q[2] / sc->focalDistance;
                q[7] = q[3] * q[3];
            }
            // list by increasing depth (stable), so that shading can stop at the first cover
            std::vector<float> sorted(prims->size());
            std::vector<int> order(count);
            for (int k = 0; k < count; ++k) order[k] = k;
            std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
                return p[MDAS_PRIM_STRIDE * a + 2] < p[MDAS_PRIM_STRIDE * b + 2];
            });
            for (int k = 0; k < count; ++k)
                for (int f = 0; f < MDAS_PRIM_STRIDE; ++f)
                    sorted[MDAS_PRIM_STRIDE * k + f] = p[MDAS_PRIM_STRIDE * order[k] + f];
            *prims = sorted;
            p = prims->data();
            if (kind == MDAS_SCENE_DISCS_MBDOF) {
                for (int k = 0; k < count; ++k) {
                    float* q = p + MDAS_PRIM_STRIDE * k;
                    q[4] = rng.range(-0.1f, 0.1f);
                    q[5] = rng.range(-0.1f, 0.1f);
                }
            }
            break;
        }
        case MDAS_SCENE_DIRECT_LIGHT: {
            sc->dim = 4;
            sc->background = 0.0f;
            for (int k = 0; k < count; ++k) {
                float* q = p + MDAS_PRIM_STRIDE * k;
                q[3] = rng.range(0.3f, 1.0f);
                q[0] = rng.range(-2.0f, 2.0f);
                q[1] = rng.range(-2.0f, 2.0f);
                q[2] = rng.range(0.5f, 2.0f);
                q[6] = 1.0f / q[3];
                q[7] = q[3] * q[3];
            }
            // pinhole at (0,-6,3) looking at the origin, up = +z
            const double eye[3] = {0.0, -6.0, 3.0};
            const double wl = sqrt(eye[0] * eye[0] + eye[1] * eye[1] + eye[2] * eye[2]);
            const double w[3] = {-eye[0] / wl, -eye[1] / wl, -eye[2] / wl};
            // u = w x up, normalised
            double u[3] = {w[1] * 1.0 - w[2] * 0.0, w[2] * 0.0 - w[0] * 1.0, w[0] * 0.0 - w[1] * 0.0};
            const double ul = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
            for (double& x : u) x /= ul;
            // v = u x w
            const double v[3] = {u[1] * w[2] - u[2] * w[1], u[2] * w[0] - u[0] * w[2], u[0] * w[1] - u[1] * w[0]};
            const double th = sqrt(2.0) - 1.0;
            const double aspect = (double)width / (double)height;
            for (int i = 0; i < 3; ++i) {
                sc->eye[i] = (float)eye[i];
                sc->W[i] = (float)w[i];
                sc->U[i] = (float)(u[i] * th * aspect);
                sc->V[i] = (float)(v[i] * th);
            }
            sc->lightCorner[0] = -0.5f;
            sc->lightCorner[1] = -0.5f;
            sc->lightCorner[2] = 4.0f;
            sc->lightSize = 1.0f;
            sc->emission = 10.0f;
            sc->albedo = 0.7f;
            break;
        }
        default:
            return MDAS_ERR_INVALID;
    }
    return MDAS_OK;
}
