// Device-wide exclusive prefix sum of int32 counts (no spin-waits), in as few launches as the length
// allows:
//
//   up to 16,384 counts   one block scans them (one launch; three launches of tiny grids cost 6 us);
//   up to 4 M             scan_reduce: each 4096-element block sums its counts to an int64;
//                         scan_downsweep: each block sums the blocks before it, scans its counts again
//                         and adds that prefix;
//   more                  the block sums are scanned by a launch of their own in between.
//
// out[i] = sum(in[0..i)) for i in [0, n], out[n] = total (int32, valid while the total
// fits; the int64 total is also stored for overflow checks by the caller).
//
// The length may be a device value (Len; counts past it are not read and out past it is not written),
// and End runs once, in one thread, with the total: what follows a scan (overflow flags) needs no
// launch of its own.
#pragma once

#include "us3d_common.cuh"

namespace us3d {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_CHUNKS = SCAN_ITEMS / 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
constexpr int SCAN_ONE_THREADS = 1024;
constexpr int64_t SCAN_ONE = SCAN_ONE_THREADS * SCAN_ITEMS;  // counts one block scans
constexpr int SCAN_DIRECT_BLOCKS = 1024;                     // blocks whose sums each block adds up itself

static inline int scan_num_blocks(int64_t n) { return (int)((n + SCAN_TILE - 1) / SCAN_TILE); }

struct ScanLen {  // a length known to the host
    int64_t n;
    __device__ __forceinline__ int64_t operator()() const { return n; }
};
struct ScanEnd {  // nothing to do with the total
    __device__ __forceinline__ void operator()(long long) const {}
};

// Inclusive warp scan of a 64-bit value.
static __device__ __forceinline__ long long warp_inclusive_scan(long long v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan (blockDim.x == THREADS); returns the block total in *total.
template <int THREADS>
static __device__ __forceinline__ long long block_exclusive_scan(long long v, long long* total) {
    __shared__ long long warp_sums[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long inc = warp_inclusive_scan(v);
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        long long s = (lane < THREADS / 32) ? warp_sums[lane] : 0;
        long long si = warp_inclusive_scan(s);
        if (lane < THREADS / 32) warp_sums[lane] = si - s;
    }
    __syncthreads();
    long long excl = inc - v + warp_sums[warp];
    // Total = exclusive prefix of the last thread + its value.
    __shared__ long long s_total;
    if (threadIdx.x == THREADS - 1) s_total = excl + v;
    __syncthreads();
    *total = s_total;
    return excl;
}

static __device__ __forceinline__ int scan_clamp(long long t) { return t > 0x7fffffffLL ? 0x7fffffff : (int)t; }

// The counts of one block, THREADS * SCAN_ITEMS of them from `base` on: SCAN_CHUNKS times a chunk of four
// neighbours per thread, so that a warp reads and writes 512 bytes in a row (with a thread's 16 counts in
// a row one block took 11 us for 16,384 counts; 4 us so, and the two launches over 1M counts 6 instead of 10).
template <int THREADS>
struct ScanBlock {
    static constexpr int WARPS = THREADS / 32;
    int x[SCAN_CHUNKS][4];
    long long run[SCAN_CHUNKS];  // sum of the block's counts before each chunk's four

    static __device__ __forceinline__ int64_t at(int64_t base, int c) {
        return base + ((int64_t)c * THREADS + threadIdx.x) * 4;
    }
    __device__ __forceinline__ void load(const int* __restrict__ in, int64_t n, int64_t base) {
        const bool vec = (reinterpret_cast<uintptr_t>(in) & 15) == 0;  // base: a multiple of 4
#pragma unroll
        for (int c = 0; c < SCAN_CHUNKS; ++c) {
            const int64_t i = at(base, c);
            if (vec && i + 4 <= n) {
                const int4 v = *reinterpret_cast<const int4*>(in + i);
                x[c][0] = v.x; x[c][1] = v.y; x[c][2] = v.z; x[c][3] = v.w;
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) x[c][k] = i + k < n ? in[i + k] : 0;
            }
        }
    }
    // Returns the block's total; `run` only when asked for.
    template <bool PREFIX>
    __device__ __forceinline__ long long scan() {
        __shared__ long long sums[SCAN_CHUNKS * WARPS];
        __shared__ long long s_total;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int c = 0; c < SCAN_CHUNKS; ++c) {
            const long long v = (long long)x[c][0] + x[c][1] + x[c][2] + x[c][3];
            const long long inc = warp_inclusive_scan(v);
            run[c] = inc - v;
            if (lane == 31) sums[c * WARPS + warp] = inc;
        }
        __syncthreads();
        if (warp == 0) {
            constexpr int PER = SCAN_CHUNKS * WARPS / 32;
            long long mine[PER], v = 0;
#pragma unroll
            for (int k = 0; k < PER; ++k) v += mine[k] = sums[lane * PER + k];
            const long long inc = warp_inclusive_scan(v);
            if (lane == 31) s_total = inc;
            long long before = inc - v;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                sums[lane * PER + k] = before;
                before += mine[k];
            }
        }
        __syncthreads();
        if (PREFIX) {
#pragma unroll
            for (int c = 0; c < SCAN_CHUNKS; ++c) run[c] += sums[c * WARPS + warp];
        }
        return s_total;
    }
    __device__ __forceinline__ void store(int* __restrict__ out, int64_t n, int64_t base, long long before) const {
        const bool vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
#pragma unroll
        for (int c = 0; c < SCAN_CHUNKS; ++c) {
            const int64_t i = at(base, c);
            long long r = before + run[c];
            int o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                o[k] = (int)r;
                r += x[c][k];
            }
            if (vec && i + 4 <= n) {
                *reinterpret_cast<int4*>(out + i) = make_int4(o[0], o[1], o[2], o[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (i + k < n) out[i + k] = o[k];
            }
        }
    }
};

template <class Len, class End>
static __global__ void __launch_bounds__(SCAN_ONE_THREADS)
scan_one_kernel(const int* __restrict__ in, Len len, int* __restrict__ out, long long* __restrict__ total_out, End end) {
    const int64_t n = len();
    ScanBlock<SCAN_ONE_THREADS> b;
    b.load(in, n, 0);
    const long long total = b.scan<true>();
    b.store(out, n, 0, 0);
    if (threadIdx.x == 0) {
        out[n] = scan_clamp(total);
        *total_out = total;
        end(total);
    }
}

template <class Len>
static __global__ void __launch_bounds__(SCAN_THREADS)
scan_reduce_kernel(const int* __restrict__ in, Len len, long long* __restrict__ block_sums) {
    const int64_t n = len();
    if ((int64_t)blockIdx.x * SCAN_TILE >= n && blockIdx.x > 0) return;
    ScanBlock<SCAN_THREADS> b;
    b.load(in, n, (int64_t)blockIdx.x * SCAN_TILE);
    const long long total = b.scan<false>();
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

template <class Len>
static __global__ void __launch_bounds__(SCAN_THREADS)
scan_blocksums_kernel(long long* __restrict__ block_sums, Len len) {
    const int64_t n = len();
    const int nb = n > 0 ? (int)((n + SCAN_TILE - 1) / SCAN_TILE) : 1;
    long long carry = 0;
    for (int base = 0; base < nb; base += SCAN_THREADS) {
        const int i = base + threadIdx.x;
        long long v = (i < nb) ? block_sums[i] : 0;
        long long tot;
        long long ex = block_exclusive_scan<SCAN_THREADS>(v, &tot);
        if (i < nb) block_sums[i] = carry + ex;
        carry += tot;
        __syncthreads();
    }
}

// DIRECT: block_sums holds the blocks' sums, which every block adds up to its own prefix; otherwise
// their prefixes.
template <bool DIRECT, class Len, class End>
static __global__ void __launch_bounds__(SCAN_THREADS)
scan_downsweep_kernel(const int* __restrict__ in, Len len, const long long* __restrict__ block_sums,
                      int* __restrict__ out, long long* __restrict__ total_out, End end) {
    const int64_t n = len();
    if ((int64_t)blockIdx.x * SCAN_TILE >= n && blockIdx.x > 0) return;
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
    ScanBlock<SCAN_THREADS> b;
    b.load(in, n, base);
    long long before = 0;
    if (DIRECT) {
        long long mine = 0;
        for (int k = threadIdx.x; k < (int)blockIdx.x; k += SCAN_THREADS) mine += block_sums[k];
        block_exclusive_scan<SCAN_THREADS>(mine, &before);
    } else {
        before = block_sums[blockIdx.x];
    }
    const long long btot = b.scan<true>();
    b.store(out, n, base, before);
    if ((int64_t)(blockIdx.x + 1) * SCAN_TILE >= n && threadIdx.x == 0) {  // the last block with counts
        const long long total = before + btot;
        out[n] = scan_clamp(total);
        *total_out = total;
        end(total);
    }
}

// Scans in[0, n) (n: the most counts there can be, when len gives fewer). block_sums must hold
// scan_num_blocks(n) entries (>= 1).
template <class Len = ScanLen, class End = ScanEnd>
static inline cudaError_t exclusive_scan(const int* in, int64_t n, int* out, long long* block_sums, long long* total,
                                         cudaStream_t stream, Len len, End end) {
    if (n <= SCAN_ONE) {
        scan_one_kernel<<<1, SCAN_ONE_THREADS, 0, stream>>>(in, len, out, total, end);
        return cudaGetLastError();
    }
    const int nb = scan_num_blocks(n);
    scan_reduce_kernel<<<nb, SCAN_THREADS, 0, stream>>>(in, len, block_sums);
    if (nb <= SCAN_DIRECT_BLOCKS) {
        scan_downsweep_kernel<true><<<nb, SCAN_THREADS, 0, stream>>>(in, len, block_sums, out, total, end);
    } else {
        scan_blocksums_kernel<<<1, SCAN_THREADS, 0, stream>>>(block_sums, len);
        scan_downsweep_kernel<false><<<nb, SCAN_THREADS, 0, stream>>>(in, len, block_sums, out, total, end);
    }
    return cudaGetLastError();
}
static inline cudaError_t exclusive_scan(const int* in, int64_t n, int* out, long long* block_sums, long long* total,
                                         cudaStream_t stream) {
    return exclusive_scan(in, n, out, block_sums, total, stream, ScanLen{n}, ScanEnd{});
}
// Kernel launches exclusive_scan makes.
static inline int scan_launches(int64_t n) {
    return n <= SCAN_ONE ? 1 : (scan_num_blocks(n) <= SCAN_DIRECT_BLOCKS ? 2 : 3);
}

}  // namespace us3d
