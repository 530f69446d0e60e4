// Bucket lists without a sort per bucket, for renderers whose element g has the instances of a
// rectangle of buckets (binning.cuh) on a small bucket grid.
//
// A bucket's list is ordered by (depth key, element). Ordering the elements once, by a stable
// radix sort of the n depth keys (none at all when the renderer has no depth key), and then filling
// the buckets in that order gives the same lists as sorting every bucket's instances: an element
// has several instances, so n keys are far fewer than the keys of all buckets, and the fill is a
// counting pass:
//
//   1. chunk_count: chunks of consecutive ranks count their instances per bucket;
//   2. chunk_prefix: per bucket, the counts' exclusive prefix over the chunks and the bucket's total;
//   3. (caller) bucket starts: exclusive scan of the totals;
//   4. chunk_fill: every chunk marks its elements in one bitmap per bucket; a set bit's place in the
//      bucket is the chunk's prefix plus the number of set bits before it. Each bucket's entries of a
//      chunk are written side by side.
//
// Everything is exact and deterministic; no block waits on another. Bound by
// launches and latency on small calls, by the fill's writes on large ones. Binning time against scattering
// all instances and sorting every bucket (tile_sort_*): 200k elements without depth keys on 256 buckets 376 ->
// 24 us, on 2025 buckets 573 -> 103 us, 30k on 1024 buckets 67 -> 30 us, 5k on 256 buckets 24 -> 11 us; with
// depth keys 200k surfels on 256 buckets 385 -> 94 us, on 2025 buckets 704 -> 141 us, 1M Gaussians on 512
// rays (13M instances) 1716 -> 289 us.
#pragma once

#include "us3d_common.cuh"
#include "scan.cuh"
#include "binning.cuh"

namespace us3d {

// The bitmaps of a chunk (bits: buckets x elements) fit 64 KB; with more buckets than
// STABLE_MAX_BUCKETS a chunk would hold too few elements for its bitmap to be worth scanning.
constexpr int64_t STABLE_MAX_BUCKETS = 2048;
constexpr int STABLE_BITS = 512 * 1024;
constexpr int STABLE_MAX_CHUNK = 1024, STABLE_MIN_CHUNK = 128;  // 2048 buckets x 256 fit STABLE_BITS
constexpr int STABLE_THREADS = 512;

// Elements with a depth key take this path from STABLE_MIN_KEYED on: below, the radix sort's twelve
// launches cost more than sorting short buckets (20k surfels on 256 buckets 70 us against 44 us, 60k 60 us
// against 133 us; scanlines of 40k Gaussians with short lists 50 against 45 us, with long ones 50 against 123 us).
// GaussianPile draws its own line further up.
constexpr int64_t STABLE_MIN_KEYED = 32768;
static inline bool stable_bins(int64_t n, int64_t n_buckets, bool keyed) {
    return n_buckets <= STABLE_MAX_BUCKETS && (!keyed || n >= STABLE_MIN_KEYED);
}
// Elements per chunk: as many as the bitmaps hold, fewer on a small call so that every SM has two chunks.
static inline int stable_chunk(int64_t n, int64_t n_buckets) {
    int c = STABLE_MAX_CHUNK;
    while (c > STABLE_MIN_CHUNK && ((int64_t)c * n_buckets > STABLE_BITS || n < (int64_t)c * 296)) c >>= 1;
    return c;
}
static inline int64_t stable_chunks(int64_t n, int64_t n_buckets) {
    const int c = stable_chunk(n, n_buckets);
    return n > 0 ? (n + c - 1) / c : 1;
}

// ------------------------------------------------------------------------------------
// Stable radix sort of (32-bit key, element index), least significant digit first
// ------------------------------------------------------------------------------------
constexpr int RADIX_BINS = 256;
constexpr int RADIX_THREADS = 256;
// Elements per thread: few on a small call, whose blocks would otherwise leave most SMs idle (200k keys,
// all four passes 83 -> 45 us), many on a large one (fewer counts to scan).
constexpr int RADIX_ROUNDS_FEW = 4, RADIX_ROUNDS_MANY = 16;
constexpr int64_t RADIX_MANY = 148 * 4 * RADIX_THREADS * RADIX_ROUNDS_FEW;  // four blocks of few per SM
constexpr int RADIX_WARPS = RADIX_THREADS / 32;

static inline int64_t radix_blocks(int64_t n) {
    const int64_t tile = RADIX_THREADS * (n > RADIX_MANY ? RADIX_ROUNDS_MANY : RADIX_ROUNDS_FEW);
    return n > 0 ? (n + tile - 1) / tile : 1;
}

template <int ROUNDS>
static __global__ void __launch_bounds__(RADIX_THREADS)
radix_count_kernel(int64_t n, const uint32_t* __restrict__ keys, int shift, int nb, int* __restrict__ counts) {
    __shared__ int s_cnt[RADIX_BINS];
    s_cnt[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * (RADIX_THREADS * ROUNDS);
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int64_t i = base + r * RADIX_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&s_cnt[(keys[i] >> shift) & (RADIX_BINS - 1)], 1);
    }
    __syncthreads();
    counts[(int64_t)threadIdx.x * nb + blockIdx.x] = s_cnt[threadIdx.x];
}

// One warp per digit: the exclusive prefix of its counts over the blocks, in place, and its total.
static __global__ void __launch_bounds__(RADIX_THREADS)
radix_prefix_kernel(int nb, int* __restrict__ counts, int* __restrict__ totals) {
    const int d = (blockIdx.x * RADIX_THREADS + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (d >= RADIX_BINS) return;
    int* c = counts + (int64_t)d * nb;
    int carry = 0;
    for (int b0 = 0; b0 < nb; b0 += 32) {
        const int v = b0 + lane < nb ? c[b0 + lane] : 0;
        int inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (b0 + lane < nb) c[b0 + lane] = carry + inc - v;
        carry += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) totals[d] = carry;
}

// vals_in NULL: the elements' own indices (the first pass).
template <int ROUNDS>
static __global__ void __launch_bounds__(RADIX_THREADS)
radix_scatter_kernel(int64_t n, const uint32_t* __restrict__ keys_in, const int* __restrict__ vals_in, int shift, int nb,
                     const int* __restrict__ counts, const int* __restrict__ totals, uint32_t* __restrict__ keys_out,
                     int* __restrict__ vals_out) {
    __shared__ int s_hist[RADIX_WARPS][RADIX_BINS];
    __shared__ int s_warp[RADIX_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int w = 0; w < RADIX_WARPS; ++w) s_hist[w][threadIdx.x] = 0;
    __syncthreads();
    // a warp holds 32 ROUNDS consecutive elements, 32 of them per round
    const int64_t base = (int64_t)blockIdx.x * (RADIX_THREADS * ROUNDS) + (int64_t)warp * (32 * ROUNDS);
    uint32_t key[ROUNDS];
    int rank[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int64_t i = base + r * 32 + lane;
        key[r] = i < n ? keys_in[i] : 0u;
    }
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int64_t i = base + r * 32 + lane;
        const int d = i < n ? (int)((key[r] >> shift) & (RADIX_BINS - 1)) : RADIX_BINS;
        const unsigned same = __match_any_sync(0xffffffffu, d);
        const int before = __popc(same & ((1u << lane) - 1u));
        int seen = 0;
        if (d < RADIX_BINS) seen = s_hist[warp][d];
        __syncwarp();
        if (d < RADIX_BINS && before == 0) s_hist[warp][d] = seen + __popc(same);
        __syncwarp();
        rank[r] = seen + before;
    }
    __syncthreads();
    {  // thread d: digit d's first place for every warp of this block
        const int d = threadIdx.x;
        const int tot = totals[d];
        int inc = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        int place = inc - tot + counts[(int64_t)d * nb + blockIdx.x];
        for (int w = 0; w < warp; ++w) place += s_warp[w];
#pragma unroll
        for (int w = 0; w < RADIX_WARPS; ++w) {
            const int c = s_hist[w][d];
            s_hist[w][d] = place;
            place += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const int64_t i = base + r * 32 + lane;
        if (i >= n) continue;
        const int p = s_hist[warp][(key[r] >> shift) & (RADIX_BINS - 1)] + rank[r];
        keys_out[p] = key[r];
        vals_out[p] = vals_in ? vals_in[i] : (int)i;
    }
}

// Scratch of the ordering and the bucket fill.
struct StableScratch {
    int* chunk_count;        // chunks x buckets
    uint32_t *key_a, *key_b; // n each (keyed only)
    int *order_a, *order_b;  // n each (keyed only)
    int* digit_count;        // RADIX_BINS x radix blocks (keyed only)
    int* digit_total;        // RADIX_BINS (keyed only)
};

static inline StableScratch stable_carve(Carver& c, int64_t n, int64_t n_buckets, bool keyed) {
    StableScratch s = {};
    s.chunk_count = c.take<int>((size_t)(stable_chunks(n, n_buckets) * n_buckets));
    if (keyed) {
        s.order_a = c.take<int>((size_t)n);
        s.order_b = c.take<int>((size_t)n);
        s.key_a = c.take<uint32_t>((size_t)n);
        s.key_b = c.take<uint32_t>((size_t)n);
        s.digit_count = c.take<int>((size_t)(RADIX_BINS * radix_blocks(n)));
        s.digit_total = c.take<int>(RADIX_BINS);
    }
    return s;
}

// Elements in (key, index) order; *order receives the array that holds it.
static inline cudaError_t launch_order(int64_t n, const uint32_t* keys, const StableScratch& s, const int** order,
                                       cudaStream_t stream) {
    *order = s.order_a;
    if (n <= 0) return cudaSuccess;
    const int nb = (int)radix_blocks(n);
    const uint32_t* kin = keys;
    const int* vin = nullptr;
    for (int pass = 0; pass < 4; ++pass) {
        uint32_t* kout = pass & 1 ? s.key_b : s.key_a;
        int* vout = pass & 1 ? s.order_a : s.order_b;  // the last pass writes order_a
        const bool many = n > RADIX_MANY;
        const auto count = many ? radix_count_kernel<RADIX_ROUNDS_MANY> : radix_count_kernel<RADIX_ROUNDS_FEW>;
        const auto scatter = many ? radix_scatter_kernel<RADIX_ROUNDS_MANY> : radix_scatter_kernel<RADIX_ROUNDS_FEW>;
        count<<<nb, RADIX_THREADS, 0, stream>>>(n, kin, 8 * pass, nb, s.digit_count);
        radix_prefix_kernel<<<RADIX_BINS / RADIX_WARPS, RADIX_THREADS, 0, stream>>>(nb, s.digit_count, s.digit_total);
        scatter<<<nb, RADIX_THREADS, 0, stream>>>(n, kin, vin, 8 * pass, nb, s.digit_count, s.digit_total, kout, vout);
        kin = kout;
        vin = vout;
    }
    return cudaGetLastError();
}
static inline int order_launches(int64_t n) { return n > 0 ? 12 : 0; }

// ------------------------------------------------------------------------------------
// Bucket fill in the elements' order (NULL: their own)
// ------------------------------------------------------------------------------------

template <class Rect>
static __global__ void __launch_bounds__(STABLE_THREADS)
chunk_count_kernel(int64_t n, int gx, int n_buckets, int chunk, Rect rect, const int* __restrict__ order,
                   int* __restrict__ counts) {
    extern __shared__ int s_cnt[];
    for (int i = threadIdx.x; i < n_buckets; i += blockDim.x) s_cnt[i] = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < chunk; e += blockDim.x) {
        const int64_t i = (int64_t)blockIdx.x * chunk + e;
        if (i >= n) break;
        const int4 r = rect(order ? order[i] : i);
        for (int y = r.y; y < r.w; ++y)
            for (int x = r.x; x < r.z; ++x) atomicAdd(&s_cnt[y * gx + x], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_buckets; i += blockDim.x) counts[(int64_t)blockIdx.x * n_buckets + i] = s_cnt[i];
}

// Block (32 buckets x 32 runs of chunks): counts become their exclusive prefix over the chunks.
static __global__ void __launch_bounds__(1024)
chunk_prefix_kernel(int chunks, int n_buckets, int* __restrict__ counts, int* __restrict__ total) {
    __shared__ int s_run[32][33];
    const int t = blockIdx.x * 32 + threadIdx.x, run = threadIdx.y;
    const int per = (chunks + 31) / 32, c0 = min(chunks, run * per), c1 = min(chunks, c0 + per);
    int sum = 0;
    if (t < n_buckets)
        for (int c = c0; c < c1; ++c) sum += counts[(int64_t)c * n_buckets + t];
    s_run[run][threadIdx.x] = sum;
    __syncthreads();
    int before = 0;
    for (int r = 0; r < run; ++r) before += s_run[r][threadIdx.x];
    if (t >= n_buckets) return;
    for (int c = c0; c < c1; ++c) {
        const int64_t i = (int64_t)c * n_buckets + t;
        const int v = counts[i];
        counts[i] = before;
        before += v;
    }
    if (run == 31) total[t] = before;
}

// Dynamic shared memory: the bitmaps, n_buckets rows of chunk / 32 words (rows padded by one word, so
// that the elements of one word of different buckets lie in different banks).
template <class Rect>
static __global__ void __launch_bounds__(STABLE_THREADS)
chunk_fill_kernel(int64_t n, int gx, int n_buckets, int chunk, Rect rect, const int* __restrict__ order,
                  const int* __restrict__ inst_offset, const int* __restrict__ prefix, const int* __restrict__ start,
                  const long long* __restrict__ header, int* __restrict__ sorted_gid, int* __restrict__ sorted_inst) {
    extern __shared__ unsigned s_bits[];
    __shared__ int4 s_rect[STABLE_MAX_CHUNK];
    __shared__ int s_gid[STABLE_MAX_CHUNK], s_first[STABLE_MAX_CHUNK];
    if (header[H_FLAGS] != 0) return;
    const int words = chunk >> 5, pitch = words + 1;
    for (int i = threadIdx.x; i < n_buckets * pitch; i += blockDim.x) s_bits[i] = 0u;
    __syncthreads();
    for (int e = threadIdx.x; e < chunk; e += blockDim.x) {
        const int64_t i = (int64_t)blockIdx.x * chunk + e;
        if (i >= n) break;
        const int g = order ? order[i] : (int)i;
        const int4 r = rect(g);
        s_rect[e] = r;
        s_gid[e] = g;
        s_first[e] = inst_offset[g];
        for (int y = r.y; y < r.w; ++y)
            for (int x = r.x; x < r.z; ++x) atomicOr(&s_bits[(y * gx + x) * pitch + (e >> 5)], 1u << (e & 31));
    }
    __syncthreads();
    // a warp takes 32 / words buckets at a time, one bitmap word per lane
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = 32 / words, sub = lane / words, wl = lane - sub * words;
    const int* pre = prefix + (int64_t)blockIdx.x * n_buckets;
    for (int t0 = warp * per; t0 < n_buckets; t0 += (STABLE_THREADS / 32) * per) {
        const int t = t0 + sub;
        unsigned bits = t < n_buckets ? s_bits[t * pitch + wl] : 0u;
        const int c = __popc(bits);
        int inc = c;
        for (int o = 1; o < words; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc, o, words);
            if (wl >= o) inc += u;
        }
        if (bits == 0u) continue;
        int pos = start[t] + pre[t] + inc - c;
        const int ty = t / gx, tx = t - ty * gx;
        for (; bits != 0u; bits &= bits - 1u, ++pos) {
            const int e = wl * 32 + __ffs(bits) - 1;
            const int4 r = s_rect[e];
            sorted_gid[pos] = s_gid[e];
            sorted_inst[pos] = s_first[e] + (ty - r.y) * (r.z - r.x) + (tx - r.x);
        }
    }
}

static inline size_t stable_fill_smem(int64_t n, int64_t n_buckets) {
    return (size_t)n_buckets * (stable_chunk(n, n_buckets) / 32 + 1) * sizeof(unsigned);
}

template <class Rect>
static inline cudaError_t launch_chunk_count(int64_t n, int gx, int64_t n_buckets, Rect rect, const int* order,
                                             const StableScratch& s, int* bucket_count, cudaStream_t stream) {
    const int chunk = stable_chunk(n, n_buckets);
    const unsigned chunks = (unsigned)stable_chunks(n, n_buckets);
    chunk_count_kernel<Rect><<<chunks, STABLE_THREADS, (size_t)n_buckets * sizeof(int), stream>>>(
        n, gx, (int)n_buckets, chunk, rect, order, s.chunk_count);
    chunk_prefix_kernel<<<(unsigned)((n_buckets + 31) / 32), dim3(32, 32), 0, stream>>>((int)chunks, (int)n_buckets,
                                                                                        s.chunk_count, bucket_count);
    return cudaGetLastError();
}

// attr_done: per device, whether the kernel's shared-memory limit was raised (one array per
// translation unit and Rect, 128 devices).
template <class Rect>
static inline cudaError_t launch_chunk_fill(int64_t n, int gx, int64_t n_buckets, Rect rect, const int* order,
                                            const StableScratch& s, const int* inst_offset, const int* start,
                                            const long long* header, int* sorted_gid, int* sorted_inst, bool* attr_done,
                                            cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (!(dev >= 0 && dev < 128 && attr_done[dev])) {
        const size_t most = (STABLE_BITS / 32 + STABLE_MAX_BUCKETS) * sizeof(unsigned);
        e = cudaFuncSetAttribute(chunk_fill_kernel<Rect>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 128) attr_done[dev] = true;
    }
    chunk_fill_kernel<Rect><<<(unsigned)stable_chunks(n, n_buckets), STABLE_THREADS, stable_fill_smem(n, n_buckets),
                              stream>>>(n, gx, (int)n_buckets, stable_chunk(n, n_buckets), rect, order, inst_offset,
                                        s.chunk_count, start, header, sorted_gid, sorted_inst);
    return cudaGetLastError();
}

// After the scan of the bucket counts: its total must be that of the elements' instances (FLAG_TABLE
// otherwise) and fit the capacity (FLAG_OVERFLOW).
struct BinsEnd {
    long long* header;
    int64_t cap;
    __device__ __forceinline__ void operator()(long long tt) const {
        const long long tg = header[H_SCAN_G];
        long long flags = header[H_FLAGS];
        if (tg != tt) flags |= FLAG_TABLE;
        if (tg > cap || tg > 0x7fffffffLL) flags |= FLAG_OVERFLOW;
        header[H_TOTAL] = tg;
        header[H_FLAGS] = flags;
    }
};

// Per-device flags of raised shared-memory limits (one object per translation unit).
struct BinAttr {
    bool sort[128], fill[128];
};

// Bucket starts, instance offsets and every bucket's elements and instance ids in (depth key, element)
// order (dkey NULL: element order): by the stable fill when there are no instance keys (keys NULL, the caller's
// choice by stable_bins), else by scattering every instance and sorting each bucket. count[] must be zero on entry.
template <class Rect>
static inline cudaError_t launch_bins(int64_t n, int gx, int64_t n_buckets, Rect rect, const uint32_t* dkey,
                                      const int* touched, const StableScratch& stable, int* count, int* start,
                                      int* cursor, int* inst_offset, long long* bs_g, long long* bs_t, long long* header,
                                      int64_t cap, unsigned long long* keys, int* slot_inst, int* sorted_gid,
                                      int* sorted_inst, BinAttr& attr, cudaStream_t stream) {
    cudaError_t e = exclusive_scan(touched, n, inst_offset, bs_g, header + H_SCAN_G, stream);
    if (e != cudaSuccess) return e;
    const bool fill = keys == nullptr;
    const int* order = nullptr;
    if (fill) {
        if (dkey) e = launch_order(n, dkey, stable, &order, stream);
        if (e == cudaSuccess) e = launch_chunk_count(n, gx, n_buckets, rect, order, stable, count, stream);
    } else {
        e = launch_rect_count(n, gx, n_buckets, rect, count, stream);
    }
    if (e != cudaSuccess) return e;
    e = exclusive_scan(count, n_buckets, start, bs_t, header + H_SCAN_T, stream, ScanLen{n_buckets},
                       BinsEnd{header, cap});
    if (e != cudaSuccess) return e;
    if (fill)
        return launch_chunk_fill(n, gx, n_buckets, rect, order, stable, inst_offset, start, header, sorted_gid,
                                 sorted_inst, attr.fill, stream);
    e = launch_rect_scatter(n, gx, n_buckets, rect, dkey, inst_offset, start, cursor, header, keys, slot_inst, stream);
    if (e != cudaSuccess) return e;
    return launch_tile_sort(n_buckets, n, start, header, keys, slot_inst, sorted_gid, sorted_inst, attr.sort, stream);
}

// Kernel launches launch_bins makes.
static inline int bins_launches(int64_t n, int64_t n_buckets, bool fill, bool keyed) {
    const int scans = scan_launches(n) + scan_launches(n_buckets);
    if (fill) return scans + (keyed ? order_launches(n) : 0) + 2 + (n > 0);
    return scans + 2 * (n > 0) + tile_sort_launches(n);
}

}  // namespace us3d
