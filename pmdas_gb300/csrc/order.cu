// order.cu — Morton keys, one-sweep LSD radix sort, Karras hierarchy and point
// location over the MDAS leaves (compiled with strict IEEE flags: the keys
// depend on one division and one multiplication per coordinate, which a CPU
// restatement must be able to repeat bit for bit).
#include <type_traits>
#include "order.h"
#include "ld_hint.h"

namespace mdas_order {

// ---------------------------------------------------------------------------------
// Keys.  The reference numbers its initial cells (uniformSamplingKernel,
// kdgrid.cu:144-157): bit k < bitsPerDim of the cell coordinate of dimension j is
// bit D*k + (D-1-j) of the index, and for the two image dimensions bit
// k in [bitsPerDim, bitsPerDim + extraImgBits) is bit
// D*bitsPerDim + 2*(k - bitsPerDim) + 1-j.  A key is that index at
// K = bitsPerDim + fineBits bits per dimension, so key >> (D * fineBits) is
// the reference's index of the initial cell.
// ---------------------------------------------------------------------------------

// (a cell coordinate has at most 31 bits: bitsPerDim + fineBits + extraImgBits <= 31)
int key_bits(int D, int bitsPerDim, int extraImgBits, int fineBits) {
    if (D < 1 || D > 16 || bitsPerDim < 0 || extraImgBits < 0 || fineBits < 0) return -1;
    if ((long long)bitsPerDim + fineBits + extraImgBits > 31) return -1;
    const long long b = (long long)D * (bitsPerDim + fineBits) + 2LL * extraImgBits;
    return b <= 64 ? (int)b : -1;
}

int max_fine_bits(int D, int bitsPerDim, int extraImgBits) {
    if (D < 1 || D > 16 || bitsPerDim < 0 || extraImgBits < 0) return -1;
    const int rest = 64 - D * bitsPerDim - 2 * extraImgBits;
    const int f = rest < 0 ? -1 : rest / D;
    const int cap = 31 - bitsPerDim - extraImgBits;
    return f < cap ? f : cap;
}

struct KeyParams {
    int D, K, eib;
    float scaleX, scaleY;
};

// Cell coordinate of u in [0, 1) at B bits: floor(u * 2^B), clamped to [0, 2^B - 1].
__device__ __forceinline__ uint32_t quantize(float u, int B) {
    const float top = (float)(1u << B);
    const float s = __fmul_rn(u, top);  // exact: a power-of-two scaling
    if (!(s > 0.0f)) return 0u;         // negative, zero or NaN
    if (s >= top) return (1u << B) - 1u;
    return (uint32_t)s;  // truncation = floor for s > 0
}

// The 8 bits of v spread D apart (bit i to bit D * i): one entry of the table a
// key kernel keeps in shared memory, so that a key takes one lookup per byte of
// each coordinate instead of one step per bit.
__device__ __forceinline__ uint64_t spread_byte(unsigned v, int D) {
    uint64_t r = 0;
    for (int i = 0; i < 8 && D * i < 64; ++i) r |= (uint64_t)((v >> i) & 1u) << (D * i);
    return r;
}

// The bits of x at the even positions (bit i to bit 2i).
__device__ __forceinline__ uint64_t spread_two(uint32_t x) {
    uint64_t v = x;
    v = (v | (v << 16)) & 0x0000FFFF0000FFFFull;
    v = (v | (v << 8)) & 0x00FF00FF00FF00FFull;
    v = (v | (v << 4)) & 0x0F0F0F0F0F0F0F0Full;
    v = (v | (v << 2)) & 0x3333333333333333ull;
    v = (v | (v << 1)) & 0x5555555555555555ull;
    return v;
}

// Key of point p: bit b < K of dimension j's cell coordinate goes to bit
// D * b + (D - 1 - j); the extra image bits b in [K, K + eib) of the two image
// axes go to bit D * K + 2 (b - K) + 1 - j (the initial-cell numbering of
// uniformSamplingKernel, kdgrid.cu:144-160, extended to K bits).  `spread`:
// spread_byte(v, D) for v < 256.
// DIM: k.D where it is known at compile time (0: not known).
template <int DIM = 0>
__device__ __forceinline__ uint64_t point_key(const float* p, const KeyParams& k, const uint64_t* spread) {
    uint64_t key = 0;
    const uint32_t lowMask = k.K >= 32 ? 0xffffffffu : ((1u << k.K) - 1u);
    const int D = DIM ? DIM : k.D;
#pragma unroll
    for (int j = 0; j < D; ++j) {
        float u = p[j];
        if (j == 0) u = __fdiv_rn(u, k.scaleX);
        if (j == 1) u = __fdiv_rn(u, k.scaleY);
        const int B = k.K + (j < 2 ? k.eib : 0);
        const uint32_t q = quantize(u, B);
        const uint32_t low = q & lowMask;
        for (int m = 0; 8 * m < k.K; ++m)
            key |= spread[(low >> (8 * m)) & 0xffu] << (D * 8 * m + (D - 1 - j));
        if (j < 2 && k.eib > 0) key |= spread_two(q >> k.K) << (D * k.K + 1 - j);
    }
    return key;
}

__device__ __forceinline__ void load_spread(uint64_t* s_spread, int D) {
    for (int v = threadIdx.x; v < 256; v += blockDim.x) s_spread[v] = spread_byte((unsigned)v, D);
    __syncthreads();
}

__global__ void k_morton_encode(const float* __restrict__ points, int n, KeyParams kp, uint64_t* __restrict__ keys) {
    __shared__ uint64_t s_spread[256];
    load_spread(s_spread, kp.D);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        keys[i] = point_key(points + (size_t)i * kp.D, kp, s_spread);
}

// The box of cell c at K bits per dimension, as uniformSamplingKernel
// computes it (kdgrid.cu:142-164, 191-196): mn = offset, mx = offset + extent.
__global__ void k_morton_decode(const uint64_t* __restrict__ cells, int n, KeyParams kp, float* __restrict__ boxes) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint64_t c = cells[i];
        float* box = boxes + (size_t)i * 2 * kp.D;
        for (int j = 0; j < kp.D; ++j) {
            uint32_t xq = 0, extentInv = 1u << kp.K;
            for (int b = 0; b < kp.K; ++b) xq |= (uint32_t)((c >> (kp.D * b + (kp.D - j - 1))) & 1u) << b;
            if (j < 2) {
                for (int b = kp.K; b < kp.K + kp.eib; ++b)
                    xq |= (uint32_t)((c >> (kp.D * kp.K + 2 * (b - kp.K) + 1 - j)) & 1u) << b;
                extentInv <<= kp.eib;
            }
            float extent = __fdiv_rn(1.0f, (float)extentInv);
            float offset = __fmul_rn((float)xq, extent);
            if (j == 0) {
                offset = __fmul_rn(offset, kp.scaleX);
                extent = __fmul_rn(extent, kp.scaleX);
            } else if (j == 1) {
                offset = __fmul_rn(offset, kp.scaleY);
                extent = __fmul_rn(extent, kp.scaleY);
            }
            box[j] = offset;
            box[kp.D + j] = __fadd_rn(offset, extent);
        }
    }
}

// The records' heads are read by whole warps (ld_hint.h): each lane reading its own
// touched a line or two per load and lane.  5.9 M leaves at D = 4: 115 -> 80 us.
template <int D>
__global__ void __launch_bounds__(256) k_leaf_keys(const float* __restrict__ nb, int nbFloats, int L, KeyParams kp,
                                                   uint64_t* __restrict__ keys) {
    constexpr int H4 = (4 + 2 * D + 3) / 4;
    __shared__ uint64_t s_spread[256];
    __shared__ float4 s_head[8][32 * H4];
    load_spread(s_spread, kp.D);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int base = blockIdx.x * 256; base < L; base += gridDim.x * 256) {
        const int first = base + 32 * warp;
        warp_heads64<H4>(nb, nbFloats, first, L, s_head[warp]);
        if (first + lane < L) {
            const float* h = reinterpret_cast<const float*>(s_head[warp] + lane * H4);
            float c[D];
#pragma unroll
            for (int j = 0; j < D; ++j) c[j] = __fmul_rn(0.5f, __fadd_rn(h[4 + j], h[4 + D + j]));
            keys[first + lane] = point_key<D>(c, kp, s_spread);
        }
        __syncwarp();  // the buffer is refilled
    }
}

static int blocks_for(int n, int threads) {
    const int b = (n + threads - 1) / threads;
    return b < 1 ? 1 : (b > 65535 * 4 ? 65535 * 4 : b);
}

static int sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

cudaError_t morton_encode(const float* points, int n, int D, int bpd, int eib, int F, float sx, float sy,
                          uint64_t* keys, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const KeyParams kp{D, bpd + F, eib, sx, sy};
    k_morton_encode<<<blocks_for(n, 256), 256, 0, s>>>(points, n, kp, keys);
    return cudaGetLastError();
}

cudaError_t morton_decode(const uint64_t* cells, int n, int D, int bpd, int eib, float sx, float sy, float* boxes,
                          cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const KeyParams kp{D, bpd, eib, sx, sy};
    k_morton_decode<<<blocks_for(n, 256), 256, 0, s>>>(cells, n, kp, boxes);
    return cudaGetLastError();
}

#define ORDER_SWITCH_D(D, CALL)                         \
    switch (D) {                                        \
        case 3: { constexpr int DD = 3; CALL; } break;  \
        case 4: { constexpr int DD = 4; CALL; } break;  \
        case 5: { constexpr int DD = 5; CALL; } break;  \
        case 6: { constexpr int DD = 6; CALL; } break;  \
        default: return cudaErrorInvalidValue;          \
    }

cudaError_t leaf_keys(const MdasDeviceGrid& g, int L, int F, uint64_t* keys, cudaStream_t s) {
    if (L <= 0) return cudaSuccess;
    const KeyParams kp{g.D, g.bitsPerDim + F, g.extraImgBits, g.scaleX, g.scaleY};
    ORDER_SWITCH_D(g.D, (k_leaf_keys<DD><<<min(blocks_for(L, 256), 8 * sm_count()), 256, 0, s>>>(g.nb, g.nbFloats, L, kp, keys)));
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// Radix sort: 8-bit digits, least significant first.  One histogram kernel counts
// every digit position in one read of the keys; a tiny kernel turns the counts
// into each digit's global start; then one kernel per digit position ranks a
// tile of keys in shared memory and scatters it, taking the tile's offsets from
// its predecessors' published digit counts (chained scan with look-back).
// Tiles are numbered in launch order by an atomic counter, so every tile a CTA
// waits for already runs and never waits for a later one; each wait is bounded
// and records a timeout in `status` instead of waiting on.
// ---------------------------------------------------------------------------------

constexpr int kBins = 256;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
#ifndef MDAS_SORT_ITEMS
#define MDAS_SORT_ITEMS 12
#endif
// keys per thread (5.9 M keys, whole sort, items/CTAs per SM: 8/6 561, 8/5 526, 9/5 517,
// 10/4 508, 12/4 500, 14/3 511, 16/3 496-500 us; 12 keeps the smaller tile for small inputs)
constexpr int kItems = MDAS_SORT_ITEMS;
constexpr int kTile = kThreads * kItems;  // keys per tile
constexpr unsigned kFlagAggregate = 1u << 30;
constexpr unsigned kFlagInclusive = 2u << 30;
constexpr unsigned kCountMask = (1u << 30) - 1u;
constexpr int kSpinLimit = 1 << 18;  // polls of one look-back word before giving up
constexpr int kMaxPasses = 8;
constexpr int kHistKeys = 8;  // keys a thread of the histogram reads at a time
#ifndef MDAS_SORT_WINDOW
#define MDAS_SORT_WINDOW 4
#endif
constexpr int kWindow = MDAS_SORT_WINDOW;  // predecessor words read per look-back round trip

__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(unsigned* p, unsigned v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The kernels of a sort are launched with programmatic dependence: the next one may
// be scheduled while the last CTAs of this one run, and waits here before it reads
// anything this one wrote.  Its CTAs are resident only once all of this one's have
// started, so a look-back still waits for running CTAs only.  5.9 M keys, ten launches:
// 500 -> 474 us.
__device__ __forceinline__ void start_dependents() { asm volatile("griddepcontrol.launch_dependents;" :::); }
__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static cudaError_t launch_dependent(void (*kernel)(KArgs...), int grid, int block, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

__global__ void __launch_bounds__(kThreads) k_histogram(const uint64_t* __restrict__ keys, int n, int beginBit,
                                                        int endBit, int passes, unsigned* __restrict__ hist) {
    start_dependents();
    __shared__ unsigned s_hist[kMaxPasses][kBins];
    for (int i = threadIdx.x; i < passes * kBins; i += kThreads) s_hist[i / kBins][i % kBins] = 0u;
    __syncthreads();
    // kHistKeys keys of a thread at a time, so that their loads overlap (one at a time in
    // 2 CTAs per SM, each key waited for its load: the whole sort of 5.9 M keys 473 us;
    // 4 keys in 2, 4, 8 CTAs: 459, 455, 457; 8 keys in 4: 449)
    const unsigned count = (unsigned)n, step = gridDim.x * kThreads;
    for (unsigned i0 = blockIdx.x * kThreads + threadIdx.x; i0 < count; i0 += kHistKeys * step) {
        uint64_t k[kHistKeys];
#pragma unroll
        for (int q = 0; q < kHistKeys; ++q) k[q] = i0 + q * step < count ? keys[i0 + q * step] : 0ull;
        for (int p = 0; p < passes; ++p) {
            const int shift = beginBit + 8 * p;
            const unsigned m = (1u << min(8, endBit - shift)) - 1u;
#pragma unroll
            for (int q = 0; q < kHistKeys; ++q)
                if (i0 + q * step < count) atomicAdd(&s_hist[p][(unsigned)(k[q] >> shift) & m], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * kBins; i += kThreads) {
        const unsigned c = s_hist[i / kBins][i % kBins];
        if (c) atomicAdd(&hist[i], c);
    }
}

// exclusive prefix of each pass's 256 digit counts, in place (one CTA per pass)
__global__ void __launch_bounds__(kBins) k_digit_starts(unsigned* __restrict__ hist) {
    __shared__ unsigned s_warp[kBins / 32];
    unsigned* h = hist + blockIdx.x * kBins;
    start_dependents();
    wait_predecessor();
    const unsigned v = h[threadIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    unsigned base = 0;
    for (int w = 0; w < warp; ++w) base += s_warp[w];
    h[threadIdx.x] = base + incl - v;
}

struct SweepArgs {
    const uint64_t* keysIn;
    const uint32_t* valuesIn;  // nullptr: value = index
    uint64_t* keysOut;
    uint32_t* valuesOut;
    int n;
    int shift;
    int bits;
    const unsigned* digitStart;  // [256]
    unsigned* lookback;          // [tiles * 256], zeroed
    unsigned* tileCounter;       // zeroed
    unsigned* status;
    int spinLimit;               // polls of one look-back word before giving up
};

// The look-back's poll limit (0: kSpinLimit); a test sets it small to drive the
// timeout path (set_test_wait_limit).
int g_sortSpinLimit = 0;

#ifndef MDAS_SORT_MIN_CTAS
#define MDAS_SORT_MIN_CTAS 4  // 64 registers: 4 CTAs per SM (the sweep: see kItems)
#endif
// One digit position, by the chained scan of A. Adinets and D. Merrill ("Onesweep: A
// Faster Least Significant Digit Radix Sort for GPUs", 2022): one read and one write of
// the keys, global offsets by look-back (D. Merrill and M. Garland, "Single-pass Parallel
// Prefix Scan with Decoupled Look-back", 2016).  Ranking a warp's keys through per-digit
// masks that the lanes OR into shared memory is used by the same family of sorts (CUB's
// match by atomic OR).  Cycles of a CTA's phases decide the order of the steps (5.9 M
// keys; 608 CTAs at work at once):
//   * ranking within the warp was the longest (16 K cycles of 38 K with eight ballots
//     per row): a row's lanes now leave their bits at their digit in shared memory
//     and read back the lanes that share it, the next row's bits on their way
//     meanwhile;
//   * the look-back (10-16 K: up to 600 predecessors that all publish at the same
//     time, walked a window per round trip) comes after the tile is staged in digit
//     order, which needs no global offsets: most of it is over by then (windows of 4, 8
//     and 16 words: 488, 493, 495 us for the whole sort).
__global__ void __launch_bounds__(kThreads, MDAS_SORT_MIN_CTAS) k_onesweep(SweepArgs a) {
    __shared__ unsigned s_warpHist[kWarps][kBins];  // per-warp digit counts, then per-warp offsets
    __shared__ unsigned s_localStart[kBins];         // digit start within the tile
    __shared__ unsigned s_globalBase[kBins];         // output position of the tile's first key of each digit
    __shared__ unsigned s_scanWarp[kWarps];
    // the tile staged in digit order; before that, each warp's match words (two rows of
    // kBins, in s_keys)
    __shared__ __align__(16) uint64_t s_keys[kTile];
    __shared__ uint32_t s_values[kTile];
    static_assert(2 * kWarps * kBins * sizeof(unsigned) <= sizeof(s_keys), "the match words fit");
    __shared__ int s_tile;

    start_dependents();
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(a.tileCounter, 1u);  // (cleared before the histogram)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned* match = reinterpret_cast<unsigned*>(s_keys) + warp * 2 * kBins;
    for (int b = lane; b < kBins; b += 32) {
        s_warpHist[warp][b] = 0u;
        match[b] = match[kBins + b] = 0u;
    }
    wait_predecessor();
    __syncthreads();
    const int tile = s_tile;
    const int tileBase = tile * kTile;
    const int warpBase = tileBase + warp * 32 * kItems;
    const unsigned mask = (1u << a.bits) - 1u;

    // load (striped per warp: item i of lane l is key warpBase + 32 i + l) and rank within the warp
    uint64_t key[kItems];
    uint32_t val[kItems];
    unsigned rank[kItems];
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const int idx = warpBase + 32 * i + lane;
        const bool valid = idx < a.n;
        key[i] = valid ? a.keysIn[idx] : 0ull;
        val[i] = valid ? (a.valuesIn ? a.valuesIn[idx] : (uint32_t)idx) : 0u;
    }
    auto digit = [&](uint64_t k) { return (unsigned)(k >> a.shift) & mask; };
    auto announce = [&](int i) {  // this lane's bit at its digit, in row i's match words
        if (warpBase + 32 * i + lane < a.n) atomicOr(&match[(i & 1) * kBins + digit(key[i])], 1u << lane);
    };
    const unsigned lowerLanes = (1u << lane) - 1u;
    announce(0);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        if (i + 1 < kItems) announce(i + 1);
        __syncwarp();  // row i's bits (and the counts of row i - 1) are in place
        const bool valid = warpBase + 32 * i + lane < a.n;
        const unsigned d = digit(key[i]);
        unsigned peers = 0u, base = 0u;
        if (valid) {
            peers = match[(i & 1) * kBins + d];
            base = s_warpHist[warp][d];
        }
        __syncwarp();  // read by every lane
        if (valid && (peers & lowerLanes) == 0u) {  // the digit's first lane
            s_warpHist[warp][d] = base + __popc(peers);
            match[(i & 1) * kBins + d] = 0u;  // for row i + 2
        }
        rank[i] = base + __popc(peers & lowerLanes);
        __syncwarp();
    }
    __syncthreads();

    // per digit: offsets of the warps, the tile's count, published at once
    const int b = threadIdx.x;  // kThreads == kBins
    unsigned count = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const unsigned c = s_warpHist[w][b];
        s_warpHist[w][b] = count;
        count += c;
    }
    unsigned* mine = a.lookback + (size_t)tile * kBins + b;
    st_relaxed(mine, (tile == 0 ? kFlagInclusive : kFlagAggregate) | count);

    // digit starts within the tile (block-wide exclusive scan of the counts)
    {
        unsigned incl = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_scanWarp[warp] = incl;
        __syncthreads();
        unsigned base = 0;
        for (int w = 0; w < warp; ++w) base += s_scanWarp[w];
        s_localStart[b] = base + incl - count;
    }
    __syncthreads();

    // stage the tile in digit order (the match words are not needed any more)
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        if (warpBase + 32 * i + lane < a.n) {
            const unsigned d = digit(key[i]);
            const unsigned pos = s_localStart[d] + s_warpHist[warp][d] + rank[i];
            s_keys[pos] = key[i];
            s_values[pos] = val[i];
        }
    }

    // look back over the predecessors' words, a window per round trip: add aggregates
    // until an inclusive prefix; re-poll from a word not yet published
    unsigned exclusive = 0;
    if (tile > 0) {
        int t = tile - 1;
        int spins = 0;
        bool done = false;
        while (!done && t >= 0) {
            unsigned w[kWindow];
#pragma unroll
            for (int q = 0; q < kWindow; ++q)
                w[q] = t - q >= 0 ? ld_relaxed(a.lookback + (size_t)(t - q) * kBins + b) : kFlagInclusive;
            int used = 0;
            bool open = true;
#pragma unroll
            for (int q = 0; q < kWindow; ++q) {
                open = open && (w[q] & ~kCountMask) != 0u;
                if (open) {
                    exclusive += w[q] & kCountMask;
                    ++used;
                    if (w[q] & kFlagInclusive) {
                        done = true;
                        open = false;
                    }
                }
            }
            if (done) break;
            t -= used;
            if (used < kWindow) {  // tile t has not published yet
                if (++spins > a.spinLimit || ld_relaxed(a.status) != 0u) {
                    atomicOr(a.status, 1u);
                    break;
                }
                __nanosleep(20);
            }
        }
        st_relaxed(mine, kFlagInclusive | ((exclusive + count) & kCountMask));
    }
    s_globalBase[b] = a.digitStart[b] + exclusive - s_localStart[b];
    __syncthreads();

    // write it out (runs of one digit are contiguous)
    const int tileCount = min(kTile, a.n - tileBase);
    for (int j = threadIdx.x; j < tileCount; j += kThreads) {
        const uint64_t k = s_keys[j];
        const unsigned dst = s_globalBase[digit(k)] + (unsigned)j;
        if (dst < (unsigned)a.n) {  // always, unless an earlier wait gave up (then status is set)
            a.keysOut[dst] = k;
            a.valuesOut[dst] = s_values[j];
        } else {
            atomicOr(a.status, 4u);
        }
    }
}

__global__ void k_iota(uint32_t* __restrict__ v, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = (uint32_t)i;
}

static int num_passes(int beginBit, int endBit) { return (endBit - beginBit + 7) / 8; }
static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct SortLayout {
    size_t hist, counters, lookback, keysAlt, valuesAlt, total, zeroBytes;
};

static SortLayout sort_layout(int n, int beginBit, int endBit) {
    const int passes = num_passes(beginBit, endBit);
    const size_t tiles = ((size_t)n + kTile - 1) / kTile;
    SortLayout l;
    size_t off = 0;
    l.hist = off;
    off = align256(off + sizeof(unsigned) * passes * kBins);
    l.counters = off;  // passes tile counters + status
    off = align256(off + sizeof(unsigned) * (passes + 1));
    l.lookback = off;
    off = align256(off + sizeof(unsigned) * passes * tiles * kBins);
    l.zeroBytes = off;
    l.keysAlt = off;
    off = align256(off + sizeof(uint64_t) * (size_t)n);
    l.valuesAlt = off;
    off = align256(off + sizeof(uint32_t) * (size_t)n);
    l.total = off;
    return l;
}

size_t sort_temp_bytes(int n, int beginBit, int endBit) {
    if (n < 0 || beginBit < 0 || endBit > 64 || beginBit > endBit) return 0;
    return sort_layout(n, beginBit, endBit).total;
}

int sort_launches(int n, int beginBit, int endBit) {
    if (n <= 0) return 0;
    const int passes = num_passes(beginBit, endBit);
    return passes == 0 ? 1 : 2 + passes;
}

cudaError_t radix_sort(void* temp, size_t tempBytes, const uint64_t* keysIn, uint64_t* keysOut,
                       const uint32_t* valuesIn, uint32_t* valuesOut, int n, int beginBit, int endBit,
                       cudaStream_t s, unsigned** statusOut) {
    if (n < 0 || beginBit < 0 || endBit > 64 || beginBit > endBit) return cudaErrorInvalidValue;
    const SortLayout l = sort_layout(n, beginBit, endBit);
    if (!temp || tempBytes < l.total) return cudaErrorInvalidValue;
    char* base = static_cast<char*>(temp);
    unsigned* hist = reinterpret_cast<unsigned*>(base + l.hist);
    unsigned* counters = reinterpret_cast<unsigned*>(base + l.counters);
    const int passes = num_passes(beginBit, endBit);
    unsigned* status = counters + passes;
    if (statusOut) *statusOut = status;
    cudaError_t e = cudaMemsetAsync(temp, 0, l.zeroBytes, s);
    if (e != cudaSuccess || n == 0) return e;
    if (passes == 0) {
        e = cudaMemcpyAsync(keysOut, keysIn, sizeof(uint64_t) * (size_t)n, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return e;
        if (valuesIn) return cudaMemcpyAsync(valuesOut, valuesIn, sizeof(uint32_t) * (size_t)n,
                                             cudaMemcpyDeviceToDevice, s);
        k_iota<<<blocks_for(n, 256), 256, 0, s>>>(valuesOut, n);
        return cudaGetLastError();
    }
    const int histBlocks = min(blocks_for(n, kThreads * kHistKeys), 4 * sm_count());
    k_histogram<<<histBlocks, kThreads, 0, s>>>(keysIn, n, beginBit, endBit, passes, hist);
    if ((e = launch_dependent(k_digit_starts, passes, kBins, s, hist)) != cudaSuccess) return e;
    const size_t tiles = ((size_t)n + kTile - 1) / kTile;
    uint64_t* keysAlt = reinterpret_cast<uint64_t*>(base + l.keysAlt);
    uint32_t* valuesAlt = reinterpret_cast<uint32_t*>(base + l.valuesAlt);
    const uint64_t* srcK = keysIn;
    const uint32_t* srcV = valuesIn;
    for (int p = 0; p < passes; ++p) {
        // the last pass writes the caller's output
        const bool toOut = ((passes - 1 - p) % 2) == 0;
        SweepArgs a;
        a.keysIn = srcK;
        a.valuesIn = srcV;
        a.keysOut = toOut ? keysOut : keysAlt;
        a.valuesOut = toOut ? valuesOut : valuesAlt;
        a.n = n;
        a.shift = beginBit + 8 * p;
        a.bits = min(8, endBit - a.shift);
        a.digitStart = hist + p * kBins;
        a.lookback = reinterpret_cast<unsigned*>(base + l.lookback) + (size_t)p * tiles * kBins;
        a.tileCounter = counters + p;
        a.status = status;
        a.spinLimit = g_sortSpinLimit > 0 ? g_sortSpinLimit : kSpinLimit;
        if ((e = launch_dependent(k_onesweep, (int)tiles, kThreads, s, a)) != cudaSuccess) return e;
        srcK = a.keysOut;
        srcV = a.valuesOut;
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// Karras radix tree (T. Karras, "Maximizing Parallelism in the Construction of
// BVHs, Octrees, and k-d Trees", HPG 2012) over the sorted keys, with the boxes of
// its nodes.  Equal keys are told apart by their positions (the prefix length of two
// equal keys is 64 + the common prefix of their positions).
//
// Built bottom-up (the pairing of C. Apetrei, "Fast and Simple Agglomerative LBVH
// Construction", CGVC 2014): a subtree over the positions [l, r] belongs with the
// neighbour whose key shares the longer prefix with its end, so its parent splits
// at gamma = r (it is the left child) or gamma = l - 1 (the right one).  The two
// children of a split meet at gamma: the first leaves its far end there and stops,
// the second joins both.  Karras numbers the node over [l, r] r if it is a left
// child and l if it is a right one (the root 0), so that the children of the split
// gamma are gamma and gamma + 1; node numbers, children and parents are the ones
// of his top-down construction.
//
// A CTA takes kRun consecutive positions and joins everything inside them in shared
// memory: in rounds over a queue of the subtrees that still climb (half of them end
// in each round; threads that climb on their own path keep a warp busy for its
// longest one), the last 64 each on its own path.  What reaches beyond the run is listed (a few dozen subtrees per CTA)
// and meets through global memory in a second kernel, with acquire/release
// exchanges: a chain of a few microseconds per level, which inside the first kernel
// kept whole CTAs waiting (720 us).  5.9 M leaves at D = 4: 356 + 69 us, in place of
// the binary searches of the top-down construction (715 warp instructions per 32
// nodes, 149 us) and of a refit that took a global acquire/release atomic and two
// box loads per node (its barriers were half of its stalls, 660 us).
// ---------------------------------------------------------------------------------

constexpr int kRun = 512;        // positions per CTA
constexpr int kRunThreads = 256;
constexpr int kMaxDepth = 128;   // > the deepest possible tree (64 key bits + 32 position bits)

__device__ __forceinline__ int key_prefix(uint64_t a, uint64_t b, int i, int j) {
    if (a == b) return 64 + __clz((unsigned)(i ^ j));
    return __clzll((long long)(a ^ b));
}

__device__ __forceinline__ int exchange_acq_rel(int* p, int v) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.exch.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// The box of child c (c < 0: the leaf at sorted position ~c).
// READONLY: the boxes are final (point location) and go through L1, a whole box in
// 16-byte loads (8-byte ones at odd D, whose boxes start at multiples of 8 bytes); while
// the tree is built another thread writes them, so they are read through L2.
template <int D, bool READONLY = false>
__device__ __forceinline__ void child_box(const MdasDeviceGrid& g, const uint32_t* __restrict__ order, const float* boxes,
                                          int c, float (&mn)[D], float (&mx)[D]) {
    if (c < 0) {
        float h[(4 + 2 * D + 3) / 4 * 4];  // the leaf record's node and box (the record extends past them)
        ld_head64<4 + 2 * D>(g.nb + (size_t)order[~c] * g.nbFloats, h);
#pragma unroll
        for (int j = 0; j < D; ++j) {
            mn[j] = h[4 + j];
            mx[j] = h[4 + D + j];
        }
    } else if constexpr (READONLY) {
        using V = typename std::conditional<D % 2 == 0, float4, float2>::type;
        constexpr int W = sizeof(V) / sizeof(float);
        const V* b = reinterpret_cast<const V*>(boxes + (size_t)c * 2 * D);
        float v[2 * D];
#pragma unroll
        for (int j = 0; j < 2 * D / W; ++j) {
            const V x = __ldg(b + j);
            v[W * j] = x.x;
            v[W * j + 1] = x.y;
            if constexpr (W == 4) {
                v[W * j + 2] = x.z;
                v[W * j + 3] = x.w;
            }
        }
#pragma unroll
        for (int j = 0; j < D; ++j) {
            mn[j] = v[j];
            mx[j] = v[D + j];
        }
    } else {
        const float* b = boxes + (size_t)c * 2 * D;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            mn[j] = __ldcg(b + j);
            mx[j] = __ldcg(b + D + j);
        }
    }
}

template <int D>
struct TreeArgs {
    MdasDeviceGrid g;
    const uint64_t* keys;
    const uint32_t* order;
    int n;
    int2* children;
    int* parents;
    float* boxes;
    int* ends;  // [n - 1], -1: the far end of the first child to reach a split
    // subtrees that climb beyond their run: ends l (bit 31: a left child) and r; their
    // number (0 at the start)
    uint2* pending;
    unsigned* pendingCount;
};

// The subtree over [l, r] with its box.
template <int D>
struct Subtree {
    int l, r;
    float mn[D], mx[D];
};

// The split of the parent of [l, r]: gamma = r (left child) or l - 1; -2 for the
// root.  key(i): the key at position i.
template <class Key>
__device__ __forceinline__ int parent_split(int l, int r, int n, Key key) {
    const int dl = l > 0 ? key_prefix(key(l - 1), key(l), l - 1, l) : -1;
    const int dr = r < n - 1 ? key_prefix(key(r), key(r + 1), r, r + 1) : -1;
    if (dl < 0 && dr < 0) return -2;
    return dr > dl ? r : l - 1;
}

// Joins t with its sibling across the split gamma, whose far end is `far` and whose
// box is (smn, smx): t becomes the parent.  Returns the split of the parent's own
// parent (-2: t is the root); id: the parent's number, cl and cr its children.
template <int D, class Key>
__device__ __forceinline__ int join(Subtree<D>& t, int gamma, int far, const float (&smn)[D], const float (&smx)[D],
                                    int n, int& id, int& cl, int& cr, Key key) {
    const bool left = t.r == gamma;  // t is the left child
    const int l = left ? t.l : far, r = left ? far : t.r;
#pragma unroll
    for (int j = 0; j < D; ++j) {
        t.mn[j] = left ? fminf(t.mn[j], smn[j]) : fminf(smn[j], t.mn[j]);
        t.mx[j] = left ? fmaxf(t.mx[j], smx[j]) : fmaxf(smx[j], t.mx[j]);
    }
    t.l = l;
    t.r = r;
    const int up = parent_split(l, r, n, key);
    id = up == -2 ? 0 : up == r ? r : l;
    cl = l == gamma ? ~gamma : gamma;
    cr = r == gamma + 1 ? ~(gamma + 1) : gamma + 1;
    return up;
}

// Writes node id (of the split gamma) with its box.
template <int D>
__device__ __forceinline__ void write_node(const TreeArgs<D>& a, const Subtree<D>& t, int gamma, int id, int cl, int cr,
                                           bool root) {
    a.children[id] = make_int2(cl, cr);
    a.parents[cl >= 0 ? cl : (a.n - 1) + gamma] = id;
    a.parents[cr >= 0 ? cr : (a.n - 1) + gamma + 1] = id;
    if (root) a.parents[0] = -1;
    float* b = a.boxes + (size_t)id * 2 * D;
    if constexpr (D % 2 == 0) {  // (8-byte aligned halves, 16-byte ones at D = 4)
        if constexpr (D == 4) {
            __stcg(reinterpret_cast<float4*>(b), make_float4(t.mn[0], t.mn[1], t.mn[2], t.mn[3]));
            __stcg(reinterpret_cast<float4*>(b) + 1, make_float4(t.mx[0], t.mx[1], t.mx[2], t.mx[3]));
        } else {
#pragma unroll
            for (int j = 0; j < D; j += 2) {
                __stcg(reinterpret_cast<float2*>(b + j), make_float2(t.mn[j], t.mn[j + 1]));
                __stcg(reinterpret_cast<float2*>(b + D + j), make_float2(t.mx[j], t.mx[j + 1]));
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < D; ++j) {
            __stcg(b + j, t.mn[j]);
            __stcg(b + D + j, t.mx[j]);
        }
    }
}

// Climbs from t (whose box is in global memory) through meetings in global memory.
template <int D>
__device__ __forceinline__ void climb_global(const TreeArgs<D>& a, Subtree<D>& t, int gamma) {
    auto key = [&](int i) { return a.keys[i]; };
    for (int depth = 0; gamma != -2 && depth < kMaxDepth; ++depth) {
        const bool left = t.r == gamma;
        // release: the box written last is visible to the second arrival; acquire: the
        // second arrival sees its sibling's box
        const int far = exchange_acq_rel(&a.ends[gamma], left ? t.l : t.r);
        if (far < 0) return;
        const int sib = left ? (far == gamma + 1 ? ~(gamma + 1) : gamma + 1) : (far == gamma ? ~gamma : gamma);
        float smn[D], smx[D];
        child_box<D>(a.g, a.order, a.boxes, sib, smn, smx);
        int id, cl, cr;
        const int at = gamma;
        gamma = join<D>(t, at, far, smn, smx, a.n, id, cl, cr, key);
        write_node<D>(a, t, at, id, cl, cr, gamma == -2);
    }
}

// A queued subtree of a run: its ends (positions in the run) and whether it is a
// left child (then it meets its sibling at the split after its right end, else
// before its left end).
__device__ __forceinline__ unsigned queue_pack(int l, int r, bool left) {
    return (unsigned)l | ((unsigned)r << 10) | ((unsigned)left << 20);
}

// Latency bounds it (a round is a chain of shared-memory steps and two barriers), so
// what counts is how many positions an SM holds: a subtree's box takes the slot of
// its node number, which is one of its ends (the boxes below it are not needed any
// more), and nodes go straight to global memory.
template <int D>
__global__ void __launch_bounds__(kRunThreads) k_tree(TreeArgs<D> a) {
    static_assert(kRun <= 1024, "positions in 10 bits");
    // position p of the run at p - c0: keys (from c0 - 1), the meeting points (the
    // split after position p; -1: nobody yet, >= 0: the first child's far end, -2:
    // both), boxes of the subtrees that climb, by coordinate
    __shared__ uint64_t s_keys[kRun + 2];
    __shared__ int s_ends[kRun];
    __shared__ unsigned s_queue[2][kRun], s_beyond[kRun];
    __shared__ int s_count[3];  // of the queues (by round), and of s_beyond
    __shared__ float s_box[2 * D * kRun];
    const int c0 = blockIdx.x * kRun;
    const int c1 = min(c0 + kRun, a.n);
    const int t0 = threadIdx.x;
    for (int i = t0; i < kRun + 2; i += kRunThreads) {
        const int p = c0 - 1 + i;
        s_keys[i] = p >= 0 && p < a.n ? a.keys[p] : 0ull;
    }
    auto load = [&](int i, float (&mn)[D], float (&mx)[D]) {
#pragma unroll
        for (int j = 0; j < D; ++j) {
            mn[j] = s_box[j * kRun + i];
            mx[j] = s_box[(D + j) * kRun + i];
        }
    };
    auto store = [&](int i, const float (&mn)[D], const float (&mx)[D]) {
#pragma unroll
        for (int j = 0; j < D; ++j) {
            s_box[j * kRun + i] = mn[j];
            s_box[(D + j) * kRun + i] = mx[j];
        }
    };
    for (int i = t0; i < kRun; i += kRunThreads) {
        s_ends[i] = -1;
        if (c0 + i < c1) {
            float mn[D], mx[D];
            child_box<D>(a.g, a.order, a.boxes, ~(c0 + i), mn, mx);
            store(i, mn, mx);
        }
    }
    if (t0 < 3) s_count[t0] = t0 == 0 ? c1 - c0 : 0;
    __syncthreads();
    auto key = [&](int i) { return s_keys[i - (c0 - 1)]; };
    // the leaves enter the queue; then rounds until nothing climbs
    for (int i = t0; c0 + i < c1; i += kRunThreads) {
        const int up = parent_split(c0 + i, c0 + i, a.n, key);
        s_queue[0][i] = queue_pack(i, i, up == c0 + i);
    }
    __syncthreads();
    // One step of a subtree up its run: whether it goes on as its parent (q).
    auto climb = [&](unsigned& q) {
        const bool left = (q >> 20) & 1u;
        Subtree<D> t;
        const int li = (int)(q & 1023u), ri = (int)((q >> 10) & 1023u);
        t.l = c0 + li;
        t.r = c0 + ri;
        const int gamma = left ? t.r : t.l - 1;
        if (gamma < c0 || gamma > c1 - 2) {  // the sibling lies beyond the run
            s_beyond[atomicAdd(&s_count[2], 1)] = q;
            return false;
        }
        const int far = atomicExch(&s_ends[gamma - c0], left ? t.l : t.r);
        if (far < 0) return false;  // first: the sibling goes on, or the sweep below
        __threadfence_block();
        s_ends[gamma - c0] = -2;
        load(left ? ri : li, t.mn, t.mx);
        float smn[D], smx[D];
        load((left ? gamma + 1 : gamma) - c0, smn, smx);
        int id, cl, cr;
        const int up = join<D>(t, gamma, far, smn, smx, a.n, id, cl, cr, key);
        store(id - c0, t.mn, t.mx);
        write_node<D>(a, t, gamma, id, cl, cr, up == -2);
        q = queue_pack(t.l - c0, t.r - c0, up == t.r);
        __threadfence_block();  // the box before the next meeting
        return up != -2;
    };
    int cur = 0;
    for (; s_count[cur] > 64; cur ^= 1) {
        const int count = s_count[cur];
        for (int i = t0; i < count; i += kRunThreads) {
            unsigned q = s_queue[cur][i];
            if (climb(q)) s_queue[cur ^ 1][atomicAdd(&s_count[cur ^ 1], 1)] = q;
        }
        __syncthreads();
        if (t0 == 0) s_count[cur] = 0;
        __syncthreads();
    }
    // the last ones, each on its own path
    if (t0 < s_count[cur]) {
        unsigned q = s_queue[cur][t0];
        for (int depth = 0; depth < kMaxDepth; ++depth)
            if (!climb(q)) break;
    }
    __syncthreads();
    // what climbs beyond the run, and the meetings that only one child reached inside
    // it (the other comes from beyond): into the list, in one piece per run
    for (int i = t0; i < (c1 - c0) - 1; i += kRunThreads) {
        const int far = s_ends[i];
        if (far < 0) continue;
        const bool left = far <= c0 + i;
        const int l = left ? far - c0 : i + 1, r = left ? i : far - c0;
        s_beyond[atomicAdd(&s_count[2], 1)] = queue_pack(l, r, left);
    }
    __syncthreads();
    if (t0 == 0) s_count[0] = (int)atomicAdd(a.pendingCount, (unsigned)s_count[2]);
    __syncthreads();
    for (int i = t0; i < s_count[2]; i += kRunThreads) {
        const unsigned q = s_beyond[i];
        a.pending[s_count[0] + i] = make_uint2((unsigned)(c0 + (int)(q & 1023u)) | ((q >> 20) << 31),
                                               (unsigned)(c0 + (int)((q >> 10) & 1023u)));
    }
}

// The subtrees that climb beyond their runs.
template <int D>
__global__ void __launch_bounds__(128) k_tree_top(TreeArgs<D> a) {
    const int count = (int)*a.pendingCount;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const uint2 q = a.pending[i];
        const bool left = q.x >> 31;
        Subtree<D> t;
        t.l = (int)(q.x & 0x7fffffffu);
        t.r = (int)q.y;
        const int gamma = left ? t.r : t.l - 1;
        if (gamma < 0 || gamma > a.n - 2) continue;  // (the root)
        const int id = left ? t.r : t.l;
        child_box<D>(a.g, a.order, a.boxes, t.l == t.r ? ~id : id, t.mn, t.mx);
        climb_global<D>(a, t, gamma);
    }
}

template <int D>
static cudaError_t launch_tree(const TreeArgs<D>& a, cudaStream_t s) {
    // (as many runs per SM as its shared memory holds)
    cudaError_t e = cudaFuncSetAttribute(k_tree<D>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    k_tree<D><<<(a.n + kRun - 1) / kRun, kRunThreads, 0, s>>>(a);
    k_tree_top<D><<<8 * sm_count(), 128, 0, s>>>(a);
    return cudaGetLastError();
}

size_t tree_scratch_bytes(int n) { return 256 + sizeof(uint2) * (size_t)(n > 0 ? n : 0); }

cudaError_t karras_tree(const MdasDeviceGrid& g, const uint64_t* sortedKeys, const uint32_t* order, int n,
                        int2* children, int* parents, unsigned* visits, void* scratch, float* boxes, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (n == 1) return cudaMemsetAsync(parents, 0xff, sizeof(int), s);  // the only leaf has no parent
    cudaError_t e = cudaMemsetAsync(visits, 0xff, sizeof(int) * (size_t)(n - 1), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(scratch, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    unsigned* count = static_cast<unsigned*>(scratch);
    uint2* pending = reinterpret_cast<uint2*>(static_cast<char*>(scratch) + 256);
    int* ends = reinterpret_cast<int*>(visits);
    ORDER_SWITCH_D(g.D, (e = launch_tree<DD>(TreeArgs<DD>{g, sortedKeys, order, n, children, parents, boxes, ends,
                                                          pending, count}, s)));
    return e;
}

// Point location: depth-first, left child first, pruning with closed boxes;
// a leaf holds p if mn <= p < mx in every dimension (p <= mx where the leaf's
// face is on the domain's upper face).  Left-first depth-first order visits
// leaves in key order, so the answer is the first holding leaf in key order.
constexpr int kStack = kMaxDepth;

// Bound by the chain of loads down the tree (L2, about 23 levels): at a node both
// children's boxes and both children's children are asked for together, so that a
// level costs one round trip where a pop of one node at a time costs its box, then its
// children, then often the other child's box.  That holds with whole boxes in wide loads
// and every dimension tested; one 4-byte load and branch per side made a level a chain of
// loads again and unsorted points slower than a pop at a time.  Whole calls, D = 4, pop of
// one / both by 4-byte loads / both by wide ones: 60,000 points in 188 K leaves
// 91 / 101 / 78 us, in 1.5 M leaves 99 / 104 / 91; 1 M points in 5.9 M leaves
// 348 / 327 / 304; D = 6, 1 M points in 373 K leaves 356 / 396 / 346.
// perm (may be null): the queries in the order the threads take them (points
// sorted by a coarse Morton key, so that a warp walks one region of the tree).
template <int D>
__global__ void k_locate(MdasDeviceGrid g, const uint32_t* __restrict__ order, int n, const int2* __restrict__ children,
                         const float* __restrict__ boxes, const float* __restrict__ points, int m,
                         const uint32_t* __restrict__ perm, int* __restrict__ leaves, unsigned* status) {
    float domMx[D];
    {
        float dmn[D];
        if (n == 1) child_box<D, true>(g, order, boxes, ~0, dmn, domMx);
        else child_box<D, true>(g, order, boxes, 0, dmn, domMx);
    }
    // whether node c's box holds p: closed for an internal node, the leaf's own rule else
    auto holds = [&](const float (&p)[D], int c) {
        float mn[D], mx[D];
        child_box<D, true>(g, order, boxes, c, mn, mx);
        bool in = true;
#pragma unroll
        for (int j = 0; j < D; ++j)
            in = in & (mn[j] <= p[j]) & ((p[j] < mx[j]) | ((p[j] == mx[j]) & ((c >= 0) | (mx[j] >= domMx[j]))));
        return in;
    };
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < m; t += gridDim.x * blockDim.x) {
        const int q = perm ? (int)perm[t] : t;
        if (q < 0 || q >= m) {  // a permutation from a sort that gave up
            atomicOr(status, 4u);
            continue;
        }
        float p[D];
#pragma unroll
        for (int j = 0; j < D; ++j) p[j] = points[(size_t)q * D + j];
        int stack[kStack];  // right children still to visit; their own test passed
        int sp = 0;
        int found = -1;
        const int root = n == 1 ? ~0 : 0;
        bool in = holds(p, root);
        int2 ch = make_int2(0, 0);
        if (root < 0) {
            if (in) found = (int)order[0];
            in = false;
        } else if (in) {
            ch = children[0];
        }
        while (in) {
            const int l = ch.x, r = ch.y;
            // (unused where the child is a leaf)
            const int2 ofL = children[l < 0 ? 0 : l], ofR = children[r < 0 ? 0 : r];
            const bool inL = holds(p, l), inR = holds(p, r);
            int next = l;
            if (inL) {
                if (inR && l >= 0) {
                    if (sp + 1 > kStack) {
                        atomicOr(status, 2u);
                        break;
                    }
                    stack[sp++] = r;
                }
                ch = ofL;
            } else if (inR) {
                next = r;
                ch = ofR;
            } else {
                if (sp == 0) break;
                next = stack[--sp];
                if (next >= 0) ch = children[next];
            }
            if (next < 0) {
                found = (int)order[~next];
                break;
            }
        }
        leaves[q] = found;
    }
}

cudaError_t locate(const MdasDeviceGrid& g, const uint32_t* order, int n, const int2* children, const float* boxes,
                   const float* points, int m, const uint32_t* perm, int* leaves, unsigned* status, cudaStream_t s) {
    if (m <= 0) return cudaSuccess;
    if (n <= 0) return cudaMemsetAsync(leaves, 0xff, sizeof(int) * (size_t)m, s);
    ORDER_SWITCH_D(g.D, (k_locate<DD><<<blocks_for(m, 128), 128, 0, s>>>(g, order, n, children, boxes, points, m,
                                                                         perm, leaves, status)));
    return cudaGetLastError();
}

int query_fine_bits(int D, int bitsPerDim, int extraImgBits) {
    const int base = D * bitsPerDim + 2 * extraImgBits;
    int fine = base >= 32 ? 0 : (32 - base) / D;
    if (fine > 31 - bitsPerDim - extraImgBits) fine = 31 - bitsPerDim - extraImgBits;
    return fine > 0 ? fine : 0;
}

void set_test_wait_limit(int polls) { g_sortSpinLimit = polls > 0 ? polls : 0; }

}  // namespace mdas_order
