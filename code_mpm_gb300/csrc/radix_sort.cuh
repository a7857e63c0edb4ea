// Stable LSD radix sort of (32-bit key, 32-bit value) pairs, DB-bit digits
// (8 to 10; the caller picks the fewest passes that cover the key bits).
//
// Used to order particles by cell key.  Stability within a digit
// pass comes from ranking every key against the keys before it in its tile
// (warp match + per-warp digit counters, then a prefix over the warps), so
// equal keys keep their input order; with values 0..n-1 as input the output
// is the particle order of a stable CPU sort by key (std::stable_sort).
//
// Per pass: k_rs_hist (per-tile digit histogram, digit-major layout),
// k_rs_scan (a block per digit scans that digit's tiles and leaves the digit's
// total), k_rs_scatter (whose blocks scan the totals themselves).  All three
// are latency at the sizes they see (700,000 keys in 171 tiles), so the scan
// is spread over the digits, the tiles are small enough for every SM to have
// several, and the kernels follow each other by dependent launch.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace mpm {

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
// Keys per thread (the kernels' ITEMS): 4 where the keys are few (the order of
// 700,000 particles took 43 us with 4, 50 with 8, 67 with 16; 192 before, with
// 16 and a one-block scan), 8 above (1M: 55, 53, 71).
constexpr int RS_ITEMS = 8, RS_FEW_ITEMS = 4;
constexpr long long RS_FEW = 3 << 18;  // up to so many keys
constexpr int RS_TILE = RS_THREADS * RS_ITEMS, RS_FEW_TILE = RS_THREADS * RS_FEW_ITEMS;

template <int DB, int ITEMS>
static __global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const unsigned* keys, long long n, int shift,
                                                         unsigned* counts, int nblocks) {
    constexpr unsigned NB = 1u << DB, MASK = NB - 1u;
    __shared__ unsigned h[NB];
    for (int i = threadIdx.x; i < (int)NB; i += RS_THREADS) h[i] = 0;
    step_enter<true>();
    __syncthreads();
    long long base = (long long)blockIdx.x * (RS_THREADS * ITEMS);
#pragma unroll 4
    for (int j = 0; j < ITEMS; ++j) {
        long long idx = base + (long long)j * RS_THREADS + threadIdx.x;
        if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & MASK], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < (int)NB; i += RS_THREADS) counts[(size_t)i * nblocks + blockIdx.x] = h[i];
}

// Block d: exclusive scan over the tiles of digit d's counts, in place; the
// digit's total goes to counts[gridDim.x * nblocks + d].
constexpr int RS_SCAN_THREADS = 256;
constexpr int RS_SCAN_ITEMS = 4;

static __global__ void __launch_bounds__(RS_SCAN_THREADS) k_rs_scan(unsigned* counts, int nblocks) {
    __shared__ unsigned wsum[2][RS_SCAN_THREADS / 32];
    step_enter<true>();
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    unsigned* row = counts + (size_t)blockIdx.x * nblocks;
    unsigned before = 0;
    int side = 0;
    for (int at = 0; at < nblocks; at += RS_SCAN_THREADS * RS_SCAN_ITEMS, side ^= 1) {
        const int i0 = at + t * RS_SCAN_ITEMS;
        unsigned v[RS_SCAN_ITEMS], s = 0;
#pragma unroll
        for (int j = 0; j < RS_SCAN_ITEMS; ++j) {
            v[j] = i0 + j < nblocks ? row[i0 + j] : 0u;
            s += v[j];
        }
        unsigned inc = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(FULL_MASK, inc, d);
            if (lane >= d) inc += o;
        }
        if (lane == 31) wsum[side][w] = inc;
        __syncthreads();  // (the other side's sums are still being read by slower warps)
        unsigned run = before + inc - s, all = 0;
#pragma unroll
        for (int k = 0; k < RS_SCAN_THREADS / 32; ++k) {
            const unsigned x = wsum[side][k];
            if (k < w) run += x;
            all += x;
        }
#pragma unroll
        for (int j = 0; j < RS_SCAN_ITEMS; ++j) {
            if (i0 + j < nblocks) row[i0 + j] = run;
            run += v[j];
        }
        before += all;
    }
    if (t == 0) counts[(size_t)gridDim.x * nblocks + blockIdx.x] = before;
}

template <int DB, int ITEMS>
static __global__ void __launch_bounds__(RS_THREADS) k_rs_scatter(const unsigned* kin, const unsigned* vin,
                                                            unsigned* __restrict__ kout, unsigned* __restrict__ vout,
                                                            long long n, int shift, const unsigned* offs,
                                                            int nblocks) {
    constexpr unsigned NB = 1u << DB, MASK = NB - 1u;
    __shared__ unsigned wcnt[RS_WARPS][NB];
    __shared__ unsigned gofs[NB];
    __shared__ unsigned wtot[RS_WARPS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < RS_WARPS * (int)NB; i += RS_THREADS) (&wcnt[0][0])[i] = 0;
    step_enter<true>();
    {  // where each digit's keys of this tile go: the digits before it, then its keys in earlier tiles
        constexpr int PER = (int)NB / RS_THREADS;
        unsigned v[PER], s = 0;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            v[j] = offs[(size_t)NB * nblocks + threadIdx.x * PER + j];
            s += v[j];
        }
        unsigned inc = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(FULL_MASK, inc, d);
            if (lane >= d) inc += o;
        }
        if (lane == 31) wtot[w] = inc;
        __syncthreads();
        unsigned run = inc - s;
#pragma unroll
        for (int k = 0; k < RS_WARPS; ++k)
            if (k < w) run += wtot[k];
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int d = threadIdx.x * PER + j;
            gofs[d] = run + offs[(size_t)d * nblocks + blockIdx.x];
            run += v[j];
        }
    }
    __syncthreads();
    const long long base = (long long)blockIdx.x * (RS_THREADS * ITEMS) + (long long)w * (32 * ITEMS);
    const unsigned lt = (1u << lane) - 1u;
    unsigned k[ITEMS], v[ITEMS], r[ITEMS];
#pragma unroll
    for (int c = 0; c < ITEMS; ++c) {
        long long idx = base + c * 32 + lane;
        bool ok = idx < n;
        unsigned key = ok ? kin[idx] : 0u;
        unsigned val = ok ? (vin ? vin[idx] : (unsigned)idx) : 0u;  // no input values: the identity
        unsigned d = ok ? ((key >> shift) & MASK) : (NB + lane);  // invalid lanes never match a digit
        unsigned peers = __match_any_sync(0xffffffffu, d);
        unsigned rank = 0;
        if (ok) rank = wcnt[w][d] + __popc(peers & lt);
        __syncwarp();
        if (ok && lane == __ffs(peers) - 1) wcnt[w][d] += __popc(peers);
        __syncwarp();
        k[c] = key;
        v[c] = val;
        r[c] = rank;
    }
    __syncthreads();
    for (int d = threadIdx.x; d < (int)NB; d += RS_THREADS) {
        unsigned run = 0;
        for (int ww = 0; ww < RS_WARPS; ++ww) {
            unsigned t = wcnt[ww][d];
            wcnt[ww][d] = run;
            run += t;
        }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < ITEMS; ++c) {
        long long idx = base + c * 32 + lane;
        if (idx < n) {
            unsigned d = (k[c] >> shift) & MASK;
            unsigned dst = gofs[d] + wcnt[w][d] + r[c];
            if (kout) kout[dst] = k[c];  // (the last pass of a caller that wants the order alone)
            vout[dst] = v[c];
        }
    }
}

}  // namespace mpm
