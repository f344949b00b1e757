// radix.cuh -- hand-written stable LSD radix sort of uint64 keys with an
// optional value array, 8-bit digits, one pass over the data per digit.
// Replaces the cub::DeviceRadixSort calls of src/rbsc/rbsc.cu:386-390 and 409
// where this implementation still sorts: the exact collision check, the
// sort-based relabel mode, the lumping with double weights, the quotient of
// the edge-batch mode and the R-MAT generator's duplicate removal.
//
// k_rs_hist reads the keys once and counts every digit of the sort; one block
// per digit turns the counts into the digits' starts (k_rs_starts).  A
// digit's pass (k_rs_pass) reads each tile of 4096 keys once, ranks them,
// publishes the tile's digit counts, adds up the counts of the tiles before it
// by looking back over their published words (a word is a count and a state
// in one 64-bit store: the tile's own count first, then the running count up
// to it, which ends the look-back), and writes the keys, staged in shared
// memory in digit order, to their places (coalesced runs).  The scheme is the
// published single-pass radix sort with decoupled look-back (Merrill and
// Garland 2016, Adinets and Merrill 2022).  Tiles are taken by a ticket, so
// every tile that a block waits for is running or done; the wait is bounded
// all the same, and a block whose wait runs out counts the digits of the keys
// that it did not wait for itself, so every pass ends with its output written.
//
// What bounds it: the latency of the ranking chain and the look-back, hidden
// by four blocks per SM (16 M keys with 8-byte values: 182 us a digit, 2.9
// TB/s; three blocks 256 us, five 188, ranks by __match_any_sync with three
// 231-306).  The form before, with a histogram kernel, a scan over a digit x
// tile table and two more reads of the keys, took 342 us a digit.
//
// Stability inside a tile: warp w owns keys [w*512, (w+1)*512) of the tile,
// walks them 32 at a time in memory order, and ranks equal digits by ballots
// over the digit's bits.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "common.cuh"
#include "scan.cuh"

namespace rbsc {

constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsIters = 16;                                  // keys per lane
constexpr uint64_t kRsTile = (uint64_t)kRsThreads * kRsIters;  // 4096
constexpr int kRsBins = 256;
constexpr int kRsMaxDigits = 8;
constexpr uint32_t kRsSpins = 1u << 16;  // polls of one predecessor: tens of milliseconds

// Temporary memory: digit counts and one ticket per digit, then a look-back
// word per (tile, digit value).
struct RsTemp {
    uint32_t hist[kRsMaxDigits][kRsBins];
    uint32_t ticket[kRsMaxDigits];
    uint32_t pad[56];
};
static_assert(sizeof(RsTemp) % 256 == 0, "the look-back words follow it");

__device__ __forceinline__ uint32_t rs_digit(unsigned long long k, int shift, uint32_t mask) { return (uint32_t)(k >> shift) & mask; }

// Counts of all digits.  Keys that agree over a warp (the high digits of keys
// that are nearly in order) count with one shared-memory atomic.
static __global__ void __launch_bounds__(kRsThreads) k_rs_hist(const unsigned long long* __restrict__ keys, uint64_t n, int begin_bit,
                                                               int end_bit, RsTemp* __restrict__ t)
{
    __shared__ uint32_t s_hist[kRsMaxDigits][kRsBins];
    const int digits = (end_bit - begin_bit + 7) / 8;
    for (int i = threadIdx.x; i < digits * kRsBins; i += kRsThreads) (&s_hist[0][0])[i] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * kRsThreads;
    constexpr int U = 4;
    for (uint64_t base = (uint64_t)blockIdx.x * kRsThreads + (threadIdx.x & ~31u); base < n; base += stride * U) {
        unsigned long long k[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const uint64_t i = base + stride * q + (threadIdx.x & 31u);
            k[q] = i < n ? keys[i] : 0ull;
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const uint64_t i0 = base + stride * q;
            if (i0 >= n) break;
            const bool valid = i0 + (threadIdx.x & 31u) < n;
            const bool full = i0 + 32u <= n;
            const unsigned long long k0 = __shfl_sync(0xffffffffu, k[q], 0);
            for (int d = 0; d < digits; ++d) {
                const int sh = begin_bit + 8 * d;
                const uint32_t mask = end_bit - sh >= 8 ? 0xffu : (1u << (end_bit - sh)) - 1u;
                const uint32_t v = rs_digit(k[q], sh, mask);
                if (full && __all_sync(0xffffffffu, v == rs_digit(k0, sh, mask))) {
                    if ((threadIdx.x & 31u) == 0) atomicAdd(&s_hist[d][v], 32u);
                } else if (valid) {
                    atomicAdd(&s_hist[d][v], 1u);
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < digits * kRsBins; i += kRsThreads) {
        const uint32_t c = (&s_hist[0][0])[i];
        if (c) atomicAdd(&(&t->hist[0][0])[i], c);
    }
}

// counts of digit blockIdx.x -> exclusive prefix
static __global__ void __launch_bounds__(kRsThreads) k_rs_starts(RsTemp* __restrict__ t)
{
    __shared__ uint32_t total;
    uint32_t* h = t->hist[blockIdx.x];
    const uint32_t c = h[threadIdx.x];
    h[threadIdx.x] = block_excl_scan<uint32_t>(c, &total);
}

// A look-back word: count in the low half; high half: digit number * 4 +
// state (1 = the tile's own count, 2 = the count up to and with the tile).
__device__ __forceinline__ unsigned long long rs_word(int digit, uint32_t state, uint32_t count)
{
    return ((unsigned long long)((uint32_t)(digit + 1) * 4u + state) << 32) | count;
}

template <typename V, bool HAS_V>
static __global__ void __launch_bounds__(kRsThreads, 4) k_rs_pass(const unsigned long long* __restrict__ keys_in,
                                                                  const V* __restrict__ vals_in,
                                                                  unsigned long long* __restrict__ keys_out, V* __restrict__ vals_out,
                                                                  uint64_t n, int digit, int shift, uint32_t mask,
                                                                  RsTemp* __restrict__ t, unsigned long long* __restrict__ words,
                                                                  uint32_t max_spins)
{
    __shared__ uint32_t s_cnt[kRsWarps][kRsBins];
    __shared__ uint32_t s_start[kRsBins];  // tile-local start of each digit's run
    __shared__ uint32_t s_base[kRsBins];   // its place in the output, minus the start
    __shared__ uint32_t s_left[kRsBins];   // tiles before this one whose counts it did not wait for
    __shared__ unsigned long long s_stage[kRsTile];
    __shared__ uint32_t s_tile, s_late, s_total;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        s_tile = atomicAdd(&t->ticket[digit], 1u);
        s_late = 0u;
    }
    for (int i = threadIdx.x; i < kRsWarps * kRsBins; i += kRsThreads) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint64_t tbase = (uint64_t)tile * kRsTile;
    const uint32_t cnt = (uint32_t)(n - tbase < kRsTile ? n - tbase : kRsTile);
    const uint32_t at0 = (uint32_t)warp * (kRsIters * 32) + lane;  // the thread's first key in the tile
    unsigned long long key[kRsIters];
#pragma unroll
    for (int it = 0; it < kRsIters; ++it) {
        const uint32_t i = at0 + it * 32;
        key[it] = i < cnt ? __ldcs(keys_in + tbase + i) : 0ull;
    }
    // rank among the warp's equal digits, then tile-local position; two 16-bit
    // values per register
    uint32_t pos2[kRsIters / 2];
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int it = 0; it < kRsIters; ++it) {
        const bool valid = at0 + it * 32 < cnt;
        const uint32_t d = rs_digit(key[it], shift, mask);
        unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < 8; ++b) {  // (bits past the digit's are 0 in every lane)
            const unsigned one = __ballot_sync(0xffffffffu, (d & (1u << b)) != 0u);
            peers &= one ^ (((d >> b) & 1u) - 1u);
        }
        // rank among equal digits of this warp so far; their first lane moves the count
        const uint32_t before = s_cnt[warp][d];
        const uint32_t rank = before + __popc(peers & lt);
        pos2[it / 2] = it & 1 ? pos2[it / 2] | rank << 16 : rank;
        __syncwarp();
        if (valid && !(peers & lt)) s_cnt[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        const int d = threadIdx.x;  // kRsThreads == kRsBins
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kRsWarps; ++w) {
            const uint32_t c = s_cnt[w][d];
            s_cnt[w][d] = run;
            run += c;
        }
        volatile unsigned long long* const mine = words + (size_t)tile * kRsBins + d;
        uint32_t prev = 0;
        if (tile == 0) {
            *mine = rs_word(digit, 2, run);
        } else {
            *mine = rs_word(digit, 1, run);
        }
        const uint32_t start = block_excl_scan<uint32_t>(run, &s_total);
        s_start[d] = start;
        if (tile != 0) {
            const uint32_t own = (uint32_t)(digit + 1);
            uint32_t spins = 0, p = tile;
            while (p > 0) {
                const unsigned long long w = *(volatile unsigned long long*)(words + (size_t)(p - 1u) * kRsBins + d);
                if ((uint32_t)(w >> 34) == own) {  // published in this digit's pass
                    prev += (uint32_t)w;
                    spins = 0;
                    --p;
                    if ((uint32_t)(w >> 32) & 2u) p = 0;
                } else if (++spins > max_spins) {
                    s_late = 1u;
                    break;
                }
            }
            s_left[d] = p;
            if (p == 0) *mine = rs_word(digit, 2, prev + run);
        }
        s_base[d] = t->hist[digit][d] + prev - start;
    }
    __syncthreads();
    if (s_late) {  // count them here (later tiles make do with this one's own count)
        uint32_t c = 0;
        const unsigned long long* k = keys_in;
#pragma unroll 1
        for (uint32_t j = s_left[threadIdx.x] * (uint32_t)kRsTile; j > 0; --j) c += rs_digit(*k++, shift, mask) == threadIdx.x ? 1u : 0u;
        s_base[threadIdx.x] += c;
        __syncthreads();
    }
#pragma unroll
    for (int it = 0; it < kRsIters; ++it) {
        if (at0 + it * 32 < cnt) {
            const uint32_t d = rs_digit(key[it], shift, mask);
            const uint32_t at = (pos2[it / 2] >> (16 * (it & 1)) & 0xffffu) + s_start[d] + s_cnt[warp][d];
            pos2[it / 2] = it & 1 ? (pos2[it / 2] & 0xffffu) | at << 16 : (pos2[it / 2] & 0xffff0000u) | at;
            s_stage[at] = key[it];
        }
    }
    __syncthreads();
    uint32_t dst[kRsIters];
#pragma unroll
    for (int q = 0; q < kRsIters; ++q) {
        const uint32_t j = (uint32_t)q * kRsThreads + threadIdx.x;
        if (j < cnt) {
            const unsigned long long k = s_stage[j];
            dst[q] = s_base[rs_digit(k, shift, mask)] + j;
            keys_out[dst[q]] = k;
        }
    }
    if (HAS_V) {
        V* s_val = reinterpret_cast<V*>(s_stage);
        __syncthreads();
#pragma unroll
        for (int it = 0; it < kRsIters; ++it) {
            const uint32_t i = at0 + it * 32;
            if (i < cnt) s_val[pos2[it / 2] >> (16 * (it & 1)) & 0xffffu] = __ldcs(vals_in + tbase + i);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kRsIters; ++q) {
            const uint32_t j = (uint32_t)q * kRsThreads + threadIdx.x;
            if (j < cnt) vals_out[dst[q]] = s_val[j];
        }
    }
}

inline size_t radix_temp_bytes(uint64_t n)
{
    return sizeof(RsTemp) + ceil_div<uint64_t>(n ? n : 1, kRsTile) * kRsBins * sizeof(unsigned long long);
}

// Sorts keys[0..n) on bits [begin_bit, end_bit) (stable), carrying vals when
// non-null.  Ping-pongs between (keys, vals) and (keys_alt, vals_alt); returns
// true when the sorted result ended in the *_alt buffers.  n < 2^32.  Launches
// only (capturable); temp holds radix_temp_bytes(n).  max_spins: see kRsSpins.
template <typename V>
inline cudaError_t radix_sort(unsigned long long* keys, unsigned long long* keys_alt, V* vals, V* vals_alt, uint64_t n, int begin_bit, int end_bit,
                              void* temp, cudaStream_t s, bool* in_alt, uint32_t max_spins = kRsSpins)
{
    *in_alt = false;
    if (n <= 1 || end_bit <= begin_bit) return cudaSuccess;
    const uint32_t tiles = (uint32_t)ceil_div<uint64_t>(n, kRsTile);
    RsTemp* t = static_cast<RsTemp*>(temp);
    unsigned long long* words = reinterpret_cast<unsigned long long*>(t + 1);
    const int digits = (end_bit - begin_bit + 7) / 8;
    cudaError_t e = cudaMemsetAsync(temp, 0, radix_temp_bytes(n), s);
    if (e != cudaSuccess) return e;
    rbsc::launch_counter() += 2;
    k_rs_hist<<<(unsigned)(tiles < 148u * 8u ? tiles : 148u * 8u), kRsThreads, 0, s>>>(keys, n, begin_bit, end_bit, t);
    k_rs_starts<<<digits, kRsThreads, 0, s>>>(t);
    unsigned long long *ki = keys, *ko = keys_alt;
    V *vi = vals, *vo = vals_alt;
    for (int d = 0; d < digits; ++d) {
        const int shift = begin_bit + 8 * d, bits = end_bit - shift < 8 ? end_bit - shift : 8;
        const uint32_t mask = (1u << bits) - 1u;
        ++rbsc::launch_counter();
        if (vals) k_rs_pass<V, true><<<tiles, kRsThreads, 0, s>>>(ki, vi, ko, vo, n, d, shift, mask, t, words, max_spins);
        else k_rs_pass<V, false><<<tiles, kRsThreads, 0, s>>>(ki, vi, ko, vo, n, d, shift, mask, t, words, max_spins);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        unsigned long long* tk = ki; ki = ko; ko = tk;
        V* tv = vi; vi = vo; vo = tv;
        *in_alt = !*in_alt;
    }
    return cudaSuccess;
}

}  // namespace rbsc
