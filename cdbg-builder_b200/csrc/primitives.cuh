// Device-wide primitives written for this project: exclusive scan and a
// stable LSD radix sort of (key, value) pairs, u32 or u64 keys.
//
// Radix sort: one fused histogram pass computes the digit histograms of every
// requested pass in a single read of the keys; passes of large sorts whose digit
// is constant over all keys are skipped.  Each executed pass is ONE kernel (k_rs_onesweep):
// tiles rank their keys stably with warp match-any, find their global digit
// offsets by a decoupled look-back per digit, stage the tile in shared memory
// in digit order and write each digit's run contiguously.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>
#include <vector>

#include "arena.cuh"
#include "common.cuh"
#include "run_sums.hpp"

namespace cdbg {
namespace prim {
// Internal linkage: every translation unit that sorts gets its own copy.
namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <typename U>
__device__ __forceinline__ U warp_inclusive_scan(U v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        U t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive block scan of one value per thread; returns the block total in *total.
template <typename U, int THREADS>
__device__ __forceinline__ U block_exclusive_scan(U v, U* smem_warp, U& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NW = THREADS / 32;
    U inc = warp_inclusive_scan(v);
    if (lane == 31) smem_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        U w = lane < NW ? smem_warp[lane] : U(0);
        U wi = warp_inclusive_scan(w);
        if (lane < NW) smem_warp[lane] = wi - w;
        if (lane == NW - 1) smem_warp[NW] = wi;
    }
    __syncthreads();
    U r = smem_warp[warp] + inc - v;
    total = smem_warp[NW];
    __syncthreads();
    return r;
}

// ------------------------------------------------------------ ordered output
// Decoupled look-back for tiles that take their indices in launch order from
// an atomic counter.  One warp of the tile calls it (all 32 lanes, the same
// arguments): lane 0 publishes the tile's count `tot` in status[tile]; the
// warp reads its predecessors' status 32 at a time (lane l the l-th nearest),
// adds their counts back to the nearest published inclusive prefix, lane 0
// publishes the tile's own inclusive prefix, and every lane gets the
// exclusive one in `excl`.  status[] is zeroed before the launch.  A
// predecessor took its index earlier, so it is running or done; every wait is
// still bounded, and on a timeout the tile publishes what it has (so its
// successors never wait on it) and returns false.
constexpr unsigned long long LB_AGG = 1ull << LOOKBACK_SUM_BITS, LB_INC = 2ull << LOOKBACK_SUM_BITS,
                             LB_VAL = (1ull << LOOKBACK_SUM_BITS) - 1;
static_assert(LOOKBACK_SUM_BITS == 62, "two flag bits above the sum");
__device__ __forceinline__ bool lookback_exclusive(unsigned long long* status, uint64_t tile, uint64_t tot,
                                                   uint64_t& excl) {
    const int lane = threadIdx.x & 31;
    excl = 0;
    if (tile == 0) {
        if (lane == 0) atomicExch(&status[0], LB_INC | tot);
        return true;
    }
    if (lane == 0) atomicExch(&status[tile], LB_AGG | tot);
    bool ok = true;
    uint64_t sum = 0;
    for (uint64_t end = tile;;) {  // window: tiles end - 1 - lane
        unsigned long long v = LB_INC;  // before tile 0: an inclusive prefix of 0
        if (end >= (uint64_t)lane + 1) {
            const uint64_t j = end - 1 - lane;
            for (uint32_t spin = 0; spin < (1u << 24); ++spin) {
                v = *(volatile unsigned long long*)&status[j];
                if (v >> 62) break;
            }
        }
        if (!__all_sync(0xffffffffu, (v >> 62) != 0)) {
            ok = false;
            break;
        }
        const uint32_t inc = __ballot_sync(0xffffffffu, (v >> 62) == 2);
        const int stop = inc ? __ffs(inc) - 1 : 31;  // nearest inclusive lane
        uint64_t x = lane <= stop ? (v & LB_VAL) : 0;
#pragma unroll
        for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        sum += x;
        if (inc) break;
        end -= 32;
    }
    if (lane == 0) atomicExch(&status[tile], LB_INC | ((sum + tot) & LB_VAL));
    excl = sum;
    return ok;
}

// Positions of the selected elements of a tile of SEL_TILE = 8 rounds x 256
// threads among all selected ones, in element order: element tile * SEL_TILE +
// round * 256 + thread.  Every thread of the 256 calls select_tile, select_put
// and (after a barrier, one warp select_scan, and another barrier) select_pos; a
// kernel with two selections gives each its own warp, so their look-backs wait
// side by side.
constexpr int SEL_ROUNDS = 8;
constexpr int SEL_TILE = SEL_ROUNDS * 256;
struct ordered_select {
    uint32_t bal[SEL_ROUNDS * 8];  // selected lanes of (round, warp)
    uint32_t cnt[SEL_ROUNDS * 8];  // selected before (round, warp) in the tile
    uint64_t tile, base;
};
__device__ __forceinline__ uint64_t select_tile(ordered_select& s, uint32_t* tile_counter) {
    if (threadIdx.x == 0) s.tile = atomicAdd(tile_counter, 1u);
    __syncthreads();
    return s.tile;
}
// Bit r of `sel`: this thread's element of round r is selected.
__device__ __forceinline__ void select_put(ordered_select& s, uint32_t sel) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int r = 0; r < SEL_ROUNDS; ++r) {
        const uint32_t b = __ballot_sync(0xffffffffu, (sel >> r) & 1u);
        if (lane == 0) s.bal[r * 8 + warp] = b;
    }
}
// By one whole warp; the last tile stores the total.
__device__ __forceinline__ void select_scan(ordered_select& s, uint64_t tile, uint64_t ntiles,
                                            unsigned long long* status, unsigned long long* total, uint32_t* err) {
    static_assert(SEL_ROUNDS * 8 == 64, "two counts per lane");
    const int lane = threadIdx.x & 31;
    const uint32_t c0 = __popc(s.bal[2 * lane]), c1 = __popc(s.bal[2 * lane + 1]);
    const uint32_t x = warp_inclusive_scan(c0 + c1);
    const uint32_t tot = __shfl_sync(0xffffffffu, x, 31);
    s.cnt[2 * lane] = x - c0 - c1;
    s.cnt[2 * lane + 1] = x - c1;
    uint64_t excl = 0;
    const bool ok = lookback_exclusive(status, tile, tot, excl);
    if (lane == 0) {
        if (!ok) set_error(err, ERR_CHAIN_LIMIT);
        s.base = excl;
        if (tile == ntiles - 1) *total = excl + tot;
    }
}
// All of it for a kernel with one selection.
__device__ __forceinline__ void select_rank(ordered_select& s, uint32_t sel, uint64_t tile, uint64_t ntiles,
                                            unsigned long long* status, unsigned long long* total, uint32_t* err) {
    select_put(s, sel);
    __syncthreads();
    if (threadIdx.x < 32) select_scan(s, tile, ntiles, status, total, err);
    __syncthreads();
}
// Selected elements before this thread's element of round r.
__device__ __forceinline__ uint64_t select_pos(ordered_select const& s, int r) {
    const int i = r * 8 + (int)(threadIdx.x >> 5);
    return s.base + s.cnt[i] + __popc(s.bal[i] & lanemask_lt());
}

// ------------------------------------------------------------------ scan
// Shared-memory index of tile element j, padded so that a thread reading its
// consecutive elements meets no bank conflict (4- and 8-byte types).
template <typename V>
__device__ __forceinline__ uint32_t scan_pad(uint32_t j) {
    return j + (j >> (sizeof(V) == 8 ? 4 : 5));
}

// One tile of the scan, [base, base + THREADS * ITEMS) of n: coalesced loads and
// stores through shared memory, each thread scanning ITEMS consecutive elements.
// `before(tot)` turns the tile's total into the sum of everything before it
// (called by the whole block); returns the inclusive sum of the tile's end to
// the last thread.
template <typename T, typename U, int THREADS, int ITEMS, typename Before>
__device__ __forceinline__ U scan_tile(T const* __restrict__ in, uint64_t n, uint64_t base, U* __restrict__ out,
                                       U* buf, U* sw, Before const& before) {
    // the inputs go through the same buffer as the outputs (a T is no wider)
    static_assert(sizeof(T) <= sizeof(U), "inputs are staged in the output buffer");
    T* sin = reinterpret_cast<T*>(buf);
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t j = (uint32_t)i * THREADS + threadIdx.x;
        sin[scan_pad<T>(j)] = (base + j < n) ? in[base + j] : T(0);
    }
    __syncthreads();
    T v[ITEMS];
    U s = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        v[i] = sin[scan_pad<T>(threadIdx.x * ITEMS + i)];
        s += (U)v[i];
    }
    U tot;
    U p = block_exclusive_scan<U, THREADS>(s, sw, tot);  // (its barriers separate the reads from the writes below)
    p += before(tot);
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        buf[scan_pad<U>(threadIdx.x * ITEMS + i)] = p;
        p += (U)v[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t j = (uint32_t)i * THREADS + threadIdx.x;
        if (base + j < n) out[base + j] = buf[scan_pad<U>(j)];
    }
    return p;
}

// n <= SCAN_ONE elements by one block, in one launch.
constexpr int SCAN_ONE_THREADS = 512;
constexpr int SCAN_ONE_ITEMS = 8;
constexpr uint64_t SCAN_ONE = SCAN_ONE_THREADS * SCAN_ONE_ITEMS;
template <typename T, typename U>
__global__ void __launch_bounds__(SCAN_ONE_THREADS) k_scan_one(T const* __restrict__ in, uint64_t n,
                                                               U* __restrict__ out, U* total_out) {
    __shared__ U sw[SCAN_ONE_THREADS / 32 + 1];
    __shared__ U buf[SCAN_ONE + SCAN_ONE / 16];
    const U p = scan_tile<T, U, SCAN_ONE_THREADS, SCAN_ONE_ITEMS>(in, n, 0, out, buf, sw, [](U) { return U(0); });
    if (total_out && threadIdx.x == SCAN_ONE_THREADS - 1) *total_out = p;
}

// More in one pass over the data: tiles take their indices in launch order and
// find the sum before them by decoupled look-back.
// Bound: HBM (one read and one write; tile sums, their scan and the tiles again
// read the input twice: 3.5 -> 2.9 ms of a 200-genome build, three launches
// where this takes one and a memset).
template <typename T, typename U>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan(T const* __restrict__ in, uint64_t n, U* __restrict__ out,
                                                       uint32_t* tile_counter, unsigned long long* status,
                                                       U* total_out, uint32_t* err) {
    __shared__ U sw[SCAN_THREADS / 32 + 1];
    __shared__ U buf[SCAN_TILE + SCAN_TILE / 16];
    __shared__ uint64_t s_tile, s_excl;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const uint64_t tile = s_tile;
    const U p = scan_tile<T, U, SCAN_THREADS, SCAN_ITEMS>(in, n, tile * SCAN_TILE, out, buf, sw, [&](U tot) {
        if (threadIdx.x < 32) {
            uint64_t excl = 0;
            const bool ok = lookback_exclusive(status, tile, (uint64_t)tot, excl);
            if (threadIdx.x == 0) {
                if (!ok) set_error(err, ERR_CHAIN_LIMIT);
                s_excl = excl;
            }
        }
        __syncthreads();
        return (U)s_excl;
    });
    if (total_out && tile == gridDim.x - 1 && threadIdx.x == SCAN_THREADS - 1) *total_out = p;
}

// out[i] = sum(in[0..i)), in place allowed (out == in when T == U).  When
// total_dev is given the grand total is written there (device memory).  Sums
// stay below 2^62.
template <typename T, typename U>
void exclusive_scan(T const* in, U* out, uint64_t n, dev_arena& A, cudaStream_t st,
                    U* total_dev = nullptr) {
    if (n == 0) {
        if (total_dev) CDBG_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(U), st));
        return;
    }
    if (n <= SCAN_ONE) {
        {
            CDBG_PROF("k_scan_one", st);
            k_scan_one<T, U><<<1, SCAN_ONE_THREADS, 0, st>>>(in, n, out, total_dev);
        }
        CDBG_CHECK_LAUNCH();
        return;
    }
    const uint64_t tiles = ceil_div(n, SCAN_TILE);
    auto m = A.mark();
    unsigned long long* status = A.alloc<unsigned long long>(tiles + 1);  // and the tile counter
    CDBG_CUDA(cudaMemsetAsync(status, 0, 8 * (tiles + 1), st));
    {
        CDBG_PROF_BYTES("k_scan", st, n * (sizeof(T) + sizeof(U)));
        k_scan<T, U><<<(unsigned)tiles, SCAN_THREADS, 0, st>>>(in, n, out, reinterpret_cast<uint32_t*>(status + tiles),
                                                               status, total_dev, g_dev_err);
    }
    CDBG_CHECK_LAUNCH();
    A.release(m);
}

// ------------------------------------------------------------------ radix sort
constexpr int RS_THREADS = 256;
constexpr int RS_BITS = 8;
constexpr int RS_BINS = 1 << RS_BITS;
constexpr int RS_WARPS = RS_THREADS / 32;

// One pass of the LSD sort in a single kernel (decoupled look-back per
// digit).  Tiles take their indices in launch order from *tile_counter, so
// every predecessor of a tile is running or done.  A tile ranks its keys
// stably (warp w owns positions [w*ITEMS*32, (w+1)*ITEMS*32), processed in
// rounds of 32 matched by ballots), publishes its per-digit counts in
// status[tile][d], walks back over its predecessors' entries of the same digit
// until an inclusive prefix (one thread per digit), publishes its own
// inclusive prefix, stages the tile in shared memory in digit order and writes
// each digit's run contiguously at digit_start[d] + prefix.  Status words are
// [flag:2 | epoch:4 | count:58]; the epoch is the pass number, so one zeroing
// per sort serves every pass.  Waits are bounded: a tile that gives up sets
// *err and publishes what it has, so no successor waits on it, and its
// successors' positions can only come out smaller than the true ones, which
// keeps every write inside the output.
// Bound: the ranking's instructions and their latency (52% issue, 59% of the ALU
// pipe at 24 warps per SM).  A 200-genome build's passes: 9.8 ms; all matches
// before the counter updates and values after the keys through the same buffer
// 9.3; matches by ballots instead of match.any 9.05; no bounds checks between the
// loads and the stores (positions past the end rank last), one lookup per key for
// its place 8.5; digits kept instead of destinations, for 4 blocks per SM, 8.2.
// 12 or 20 keys per thread 8.8 and 8.9, a look-back over four predecessors at a
// time 0.7 slower.
constexpr unsigned long long RS_AGG = 1ull << 62, RS_INC = 2ull << 62, RS_VALMASK = (1ull << 58) - 1;

template <int BITS, int ITEMS, typename K, typename V>
struct rs_smem {
    static constexpr int BINS = 1 << BITS;
    static constexpr int TILE = RS_THREADS * ITEMS;
    static_assert(sizeof(V) <= sizeof(K), "keys and values share the buffer");
    K sk[TILE];                     // keys in digit order, then values
    uint32_t wcnt[RS_WARPS][BINS];  // per-warp digit counts, then tile-local starts
    uint32_t goff[BINS];            // a digit's output position less its tile-local one
    uint64_t sw[RS_WARPS + 1];
    uint32_t tile;
};

// The lanes of the warp with this lane's low BITS bits of `d`.
template <int BITS>
__device__ __forceinline__ uint32_t match_digit(uint32_t d) {
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < BITS; ++b) {
        const bool one = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, one);
        peers &= one ? m : ~m;
    }
    return peers;
}

template <int BITS, int ITEMS, typename K, typename V>
__global__ void __launch_bounds__(RS_THREADS, 4) k_rs_onesweep(K const* __restrict__ keys_in,
                                                            V const* __restrict__ vals_in,
                                                            K* __restrict__ keys_out, V* __restrict__ vals_out,
                                                            uint64_t n, int shift, uint32_t* tile_counter,
                                                            unsigned long long* status,
                                                            unsigned long long const* __restrict__ hist,
                                                            uint32_t epoch, uint32_t* err) {
    using S = rs_smem<BITS, ITEMS, K, V>;
    constexpr int BINS = S::BINS, TILE = S::TILE, DPT = (BINS + RS_THREADS - 1) / RS_THREADS;
    extern __shared__ __align__(16) unsigned char rs_raw[];
    S& sm = *reinterpret_cast<S*>(rs_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < RS_WARPS * BINS; i += RS_THREADS) (&sm.wcnt[0][0])[i] = 0;
    if (threadIdx.x == 0) sm.tile = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const uint64_t tile = sm.tile;
    const uint64_t base = tile * TILE;
    const uint32_t tile_n = (uint32_t)((n - base) < (uint64_t)TILE ? (n - base) : TILE);
    K k[ITEMS];
    uint32_t rk[ITEMS];
    const uint32_t p0 = (uint32_t)warp * (ITEMS * 32) + lane;  // round r: position p0 + 32 r
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) k[r] = p0 + 32u * r < tile_n ? keys_in[base + p0 + 32u * r] : ~K(0);
    auto digit = [&](K key) { return (uint32_t)(key >> shift) & (BINS - 1); };
    // the lanes of each round with the same digit: all rounds' matches first,
    // they do not depend on each other; then the warp's counters round by round.
    // Positions past the end hold the largest key: they rank after every pair,
    // and their digit's count leaves them out.
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) rk[r] = match_digit<BITS>((uint32_t)(k[r] >> shift));
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t peers = rk[r];
        const uint32_t below = __popc(peers & lanemask_lt());
        uint32_t old = 0;
        if (below == 0) {
            const uint32_t d = digit(k[r]);
            old = sm.wcnt[warp][d];
            sm.wcnt[warp][d] = old + __popc(peers);
        }
        __syncwarp();  // the next round's reader of a counter may be another lane
        rk[r] = __shfl_sync(0xffffffffu, old, __ffs(peers) - 1) + below;
    }
    __syncthreads();
    // per digit: exclusive prefix over warps and the tile's count
    uint32_t cnt[DPT];
#pragma unroll
    for (int j = 0; j < DPT; ++j) {
        const int d = threadIdx.x + j * RS_THREADS;
        uint32_t run = 0;
        if (d < BINS) {
#pragma unroll
            for (int w = 0; w < RS_WARPS; ++w) {
                const uint32_t c = sm.wcnt[w][d];
                sm.wcnt[w][d] = run;
                run += c;
            }
            if ((uint32_t)d == digit(~K(0))) run -= TILE - tile_n;
            const unsigned long long ep = (unsigned long long)epoch << 58;
            *(volatile unsigned long long*)&status[tile * BINS + d] = (tile == 0 ? RS_INC : RS_AGG) | ep | run;
        }
        cnt[j] = run;
    }
    // look-back, one thread per digit
    uint32_t before[DPT];
#pragma unroll
    for (int j = 0; j < DPT; ++j) {
        const int d = threadIdx.x + j * RS_THREADS;
        before[j] = 0;
        if (d >= BINS) continue;
        uint64_t excl = 0;
        if (tile > 0) {
            bool ok = true;
            for (uint64_t t = tile - 1;; --t) {
                unsigned long long w = 0;
                uint32_t spin = 0;
                for (; spin < (1u << 24); ++spin) {
                    w = *(volatile unsigned long long*)&status[t * BINS + d];
                    if ((w >> 62) != 0 && ((w >> 58) & 15u) == epoch) break;
                }
                if (spin == (1u << 24)) {
                    ok = false;
                    break;
                }
                excl += w & RS_VALMASK;
                if ((w >> 62) == 2 || t == 0) break;
            }
            if (!ok) set_error(err, ERR_CHAIN_LIMIT);
            const unsigned long long ep = (unsigned long long)epoch << 58;
            *(volatile unsigned long long*)&status[tile * BINS + d] = RS_INC | ep | ((excl + cnt[j]) & RS_VALMASK);
        }
        before[j] = (uint32_t)excl;
    }
    // digit starts (exclusive scans over digits): tile-local ones of the counts,
    // global ones of the pass's histogram
    {
        // thread t owns digits t, t + RS_THREADS, ...: one block scan per
        // column keeps the starts in digit order.  Both scans at once: a tile's
        // counts add up to at most TILE, the histogram to n < 2^48.
        uint64_t carry = 0;
#pragma unroll
        for (int j = 0; j < DPT; ++j) {
            const int d = threadIdx.x + j * RS_THREADS;
            const uint64_t both = d < BINS ? ((uint64_t)__ldg(hist + d) << 16) | cnt[j] : 0;
            uint64_t tot;
            const uint64_t ex = carry + block_exclusive_scan<uint64_t, RS_THREADS>(both, sm.sw, tot);
            if (d < BINS) {
                const uint32_t ds = (uint32_t)(ex & 0xffffu);
#pragma unroll
                for (int w = 0; w < RS_WARPS; ++w) sm.wcnt[w][d] += ds;
                sm.goff[d] = (uint32_t)(ex >> 16) + before[j] - ds;
            }
            carry += tot;
        }
    }
    __syncthreads();
    // keys, then values, through the same buffer in digit order
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        rk[r] += sm.wcnt[warp][digit(k[r])];
        sm.sk[rk[r]] = k[r];
    }
    V v[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t p = p0 + 32u * r;
        v[r] = p >= tile_n ? V(0) : vals_in ? vals_in[base + p] : (V)(base + p);
    }
    __syncthreads();
    // (the digits of the positions written are kept, packed, for the values)
    constexpr int PACK = BITS <= 8 ? 4 : 2;
    uint32_t dg[(ITEMS + PACK - 1) / PACK] = {};
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t p = threadIdx.x + i * RS_THREADS;
        const K key = sm.sk[p];
        const uint32_t d = digit(key), o = sm.goff[d] + p;  // (n < 2^32)
        dg[i / PACK] |= d << (32 / PACK * (i % PACK));
        if (p < tile_n && o < n) keys_out[o] = key;
    }
    __syncthreads();
    V* sv = reinterpret_cast<V*>(sm.sk);
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) sv[rk[r]] = v[r];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t p = threadIdx.x + i * RS_THREADS;
        const uint32_t o = sm.goff[(dg[i / PACK] >> (32 / PACK * (i % PACK))) & (BINS - 1)] + p;
        if (p < tile_n && o < n) vals_out[o] = sv[p];
    }
}

// Up to RS_SMALL pairs: the whole LSD sort by one block in shared memory, in one
// launch, 8-bit digits whatever the tuning says.  Ranks as k_rs_onesweep's; a
// pass whose digit is the same in every key is skipped.
// Bound: latency, about 2 us a pass; a memset, a histogram and one launch per
// pass take about 5 us each at these sizes.
constexpr int RSS_THREADS = 1024;
constexpr int RSS_ITEMS = 8;
constexpr int RSS_WARPS = RSS_THREADS / 32;
constexpr uint32_t RS_SMALL = RSS_THREADS * RSS_ITEMS;
template <typename K, typename V>
struct rss_smem {
    K sk[RS_SMALL];
    V sv[RS_SMALL];
    uint16_t wcnt[RSS_WARPS][RS_BINS];  // per-warp digit counts, then prefixes
    uint32_t dstart[RS_BINS];
    uint32_t sw[RSS_WARPS + 1];
};
template <typename K, typename V>
__global__ void __launch_bounds__(RSS_THREADS) k_rs_small(K* __restrict__ keys, V* __restrict__ vals, uint32_t n,
                                                          int begin_bit, int end_bit, bool iota) {
    extern __shared__ __align__(16) unsigned char rs_raw[];
    rss_smem<K, V>& sm = *reinterpret_cast<rss_smem<K, V>*>(rs_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t p0 = (uint32_t)warp * (RSS_ITEMS * 32) + lane;
    K k[RSS_ITEMS];
    V v[RSS_ITEMS];
#pragma unroll
    for (int r = 0; r < RSS_ITEMS; ++r) {
        const uint32_t p = p0 + 32u * r;
        k[r] = p < n ? keys[p] : ~K(0);
        v[r] = p >= n ? V(0) : iota ? (V)p : vals[p];
    }
    for (int shift = begin_bit; shift < end_bit; shift += RS_BITS) {
        const uint32_t mask = end_bit - shift < RS_BITS ? (1u << (end_bit - shift)) - 1u : RS_BINS - 1u;
        for (int i = threadIdx.x; i < RSS_WARPS * RS_BINS / 2; i += RSS_THREADS)
            reinterpret_cast<uint32_t*>(&sm.wcnt[0][0])[i] = 0;
        __syncthreads();
        uint32_t rk[RSS_ITEMS];
#pragma unroll
        for (int r = 0; r < RSS_ITEMS; ++r) {
            const bool ok = p0 + 32u * r < n;
            const uint32_t d = ok ? (uint32_t)(k[r] >> shift) & mask : (uint32_t)RS_BINS;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            const int leader = __ffs(peers) - 1;
            uint32_t old = 0;
            if (ok && lane == leader) {
                old = sm.wcnt[warp][d];
                sm.wcnt[warp][d] = (uint16_t)(old + __popc(peers));
            }
            __syncwarp();  // (as in k_rs_onesweep)
            rk[r] = __shfl_sync(0xffffffffu, old, leader) + __popc(peers & lanemask_lt());
        }
        __syncthreads();
        uint32_t cnt = 0;
        if (threadIdx.x < RS_BINS) {
#pragma unroll 8
            for (int w = 0; w < RSS_WARPS; ++w) {
                const uint32_t c = sm.wcnt[w][threadIdx.x];
                sm.wcnt[w][threadIdx.x] = (uint16_t)cnt;
                cnt += c;
            }
        }
        uint32_t tot;
        const uint32_t ex = block_exclusive_scan<uint32_t, RSS_THREADS>(cnt, sm.sw, tot);
        if (threadIdx.x < RS_BINS) sm.dstart[threadIdx.x] = ex;
        if (__syncthreads_or(cnt == n)) continue;  // one digit for all
#pragma unroll
        for (int r = 0; r < RSS_ITEMS; ++r) {
            if (p0 + 32u * r < n) {
                const uint32_t d = (uint32_t)(k[r] >> shift) & mask;
                const uint32_t at = sm.dstart[d] + sm.wcnt[warp][d] + rk[r];
                sm.sk[at] = k[r];
                sm.sv[at] = v[r];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < RSS_ITEMS; ++r) {
            const uint32_t p = p0 + 32u * r;
            if (p < n) {
                k[r] = sm.sk[p];
                v[r] = sm.sv[p];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RSS_ITEMS; ++r) {
        const uint32_t p = p0 + 32u * r;
        if (p < n) {
            keys[p] = k[r];
            vals[p] = v[r];
        }
    }
}
template <typename V, typename K>
void radix_sort_small(K* keys, V* vals, uint64_t n, int begin_bit, int end_bit, cudaStream_t st, bool iota) {
    CDBG_CUDA(cudaFuncSetAttribute(k_rs_small<K, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(rss_smem<K, V>)));
    {
        CDBG_PROF("k_rs_small", st);
        k_rs_small<K, V><<<1, RSS_THREADS, sizeof(rss_smem<K, V>), st>>>(keys, vals, (uint32_t)n, begin_bit, end_bit,
                                                                          iota);
    }
    CDBG_CHECK_LAUNCH();
}

// Histograms of all passes with BITS-bit digits, in one read.  hist is
// npasses x 2^BITS u64, zeroed by the caller.
template <int BITS, typename K>
__global__ void __launch_bounds__(RS_THREADS) k_rs_histograms_w(K const* __restrict__ keys, uint64_t n,
                                                                int begin_bit, int npasses,
                                                                unsigned long long* hist) {
    constexpr int BINS = 1 << BITS;
    extern __shared__ uint32_t hw[];  // npasses x BINS
    for (int i = threadIdx.x; i < npasses * BINS; i += RS_THREADS) hw[i] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * RS_THREADS;
    for (uint64_t i = (uint64_t)blockIdx.x * RS_THREADS + threadIdx.x; i < n; i += stride) {
        const K k = keys[i];
        for (int p = 0; p < npasses; ++p) atomicAdd(&hw[p * BINS + ((k >> (begin_bit + p * BITS)) & (BINS - 1))], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < npasses * BINS; i += RS_THREADS) {
        const uint32_t v = hw[i];
        if (v) atomicAdd(&hist[i], (unsigned long long)v);
    }
}

constexpr uint64_t RS_HOST_CHECK = 1ull << 20;
template <typename V>
__global__ void k_iota(V* __restrict__ vals, uint64_t n) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) vals[i] = (V)i;
}
template <int BITS, typename V, typename K>
int radix_sort_pairs_w(K* keys, V* vals, uint64_t n, int begin_bit, int end_bit, dev_arena& A,
                       cudaStream_t st, uint32_t* err, bool iota) {
    constexpr int BINS = 1 << BITS;
    constexpr int ITEMS = 16;
    using S = rs_smem<BITS, ITEMS, K, V>;
    constexpr int TILE = S::TILE;
    static_assert(TILE < (1 << 16), "a tile's counts are scanned in 16 bits");
    const int npasses = (end_bit - begin_bit + BITS - 1) / BITS;
    if (npasses > 15) throw std::runtime_error("radix sort: too many passes");
    auto m = A.mark();
    const uint64_t ntiles = ceil_div(n, (uint64_t)TILE);
    K* k2 = A.alloc<K>(n);
    V* v2 = A.alloc<V>(n);
    // zeroed together: look-back status, histograms, tile counters
    const size_t words = ntiles * BINS + (size_t)npasses * BINS + (npasses + 1) / 2;
    unsigned long long* status = A.alloc<unsigned long long>(words);
    unsigned long long* hist = status + ntiles * BINS;
    uint32_t* counters = reinterpret_cast<uint32_t*>(hist + (size_t)npasses * BINS);
    CDBG_CUDA(cudaMemsetAsync(status, 0, 8 * words, st));
    {
        uint64_t blocks = ceil_div(n, (uint64_t)RS_THREADS * 16);
        if (blocks > 148 * 8) blocks = 148 * 8;
        const size_t hs = sizeof(uint32_t) * npasses * BINS;
        if (hs > 48 * 1024)
            CDBG_CUDA(cudaFuncSetAttribute(k_rs_histograms_w<BITS, K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)hs));
        {
            CDBG_PROF("k_rs_histograms", st);
            k_rs_histograms_w<BITS, K><<<(unsigned)blocks, RS_THREADS, hs, st>>>(keys, n, begin_bit, npasses, hist);
        }
        CDBG_CHECK_LAUNCH();
    }
    // A pass whose digit is the same in every key is skipped, which needs the
    // histograms on the host.  Below RS_HOST_CHECK pairs a pass costs no more
    // than that wait (about 10 us), and every pass runs.
    std::vector<unsigned long long> h;
    if (n >= RS_HOST_CHECK) {
        h.resize((size_t)npasses * BINS);
        read_small(h.data(), hist, h.size() * 8, st);
    }
    CDBG_CUDA(cudaFuncSetAttribute(k_rs_onesweep<BITS, ITEMS, K, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(S)));
    K *kin = keys, *kout = k2;
    V *vin = vals, *vout = v2;
    int ran = 0;
    for (int p = 0; p < npasses; ++p) {
        bool trivial = false;
        for (int d = 0; d < BINS && !h.empty(); ++d)
            if (h[(size_t)p * BINS + d] == n) trivial = true;
        if (trivial) continue;
        const int shift = begin_bit + p * BITS;
        {
            // one read and one write of every (key, value) pair
            CDBG_PROF_BYTES("k_rs_onesweep", st, 2.0 * n * (sizeof(K) + sizeof(V)));
            k_rs_onesweep<BITS, ITEMS, K, V><<<(unsigned)ntiles, RS_THREADS, sizeof(S), st>>>(
                kin, iota && ran == 0 ? nullptr : vin, kout, vout, n, shift, counters + p, status, hist + (size_t)p * BINS, (uint32_t)(p + 1),
                err);
        }
        CDBG_CHECK_LAUNCH();
        std::swap(kin, kout);
        std::swap(vin, vout);
        ++ran;
    }
    if (iota && ran == 0) {
        k_iota<V><<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(vals, n);
        CDBG_CHECK_LAUNCH();
    }
    if (kin != keys) {
        CDBG_CUDA(cudaMemcpyAsync(keys, kin, n * sizeof(K), cudaMemcpyDeviceToDevice, st));
        CDBG_CUDA(cudaMemcpyAsync(vals, vin, n * sizeof(V), cudaMemcpyDeviceToDevice, st));
    }
    A.release(m);
    return ran;
}

// Stable sort of (keys, vals) by key bits [begin_bit, end_bit) with 8-bit or
// 11-bit digits (g_radix_bits: the engine's tuning; 11 bits take 3 passes
// where 8 bits take 4, with 8x the counters and look-back state per tile).
// Results end in (keys, vals); the arena provides the ping-pong buffers.
// With `iota`, the values on entry are 0, 1, .. n - 1 whatever `vals` holds.
// Returns the number of passes run.  A look-back that gives up sets *err.
template <typename V, typename K = uint64_t>
int radix_sort_pairs(K* keys, V* vals, uint64_t n, int begin_bit, int end_bit, dev_arena& A, cudaStream_t st,
                     uint32_t* err, bool iota = false) {
    static_assert(sizeof(K) == 4 || sizeof(K) == 8, "u32 or u64 keys");
    if (end_bit > 8 * (int)sizeof(K)) end_bit = 8 * (int)sizeof(K);
    if (!iota && (n <= 1 || end_bit <= begin_bit)) return 0;
    if (n <= RS_SMALL) {
        radix_sort_small<V, K>(keys, vals, n, begin_bit, end_bit, st, iota);
        return 1;
    }
    if (g_radix_bits == 11) return radix_sort_pairs_w<11, V, K>(keys, vals, n, begin_bit, end_bit, A, st, err, iota);
    return radix_sort_pairs_w<RS_BITS, V, K>(keys, vals, n, begin_bit, end_bit, A, st, err, iota);
}

// ----------------------------------------- exact 64-bit order, 32-bit passes
// Keys whose top 32 bits tie but whose full keys differ, after a stable sort
// on the top 32 bits: positions i with hi(i) == hi(i - 1), key(i) != key(i - 1)
// appended to `list` (count in *cnt, at most `cap` stored).
__global__ void k_hi_mismatch(uint64_t const* __restrict__ keys, uint64_t n, uint32_t* __restrict__ list,
                              unsigned long long* cnt, uint64_t cap) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool m = false;
    if (i > 0 && i < n) {
        const uint64_t a = keys[i - 1], b = keys[i];
        m = (a >> 32) == (b >> 32) && a != b;
    }
    const uint32_t bal = __ballot_sync(0xffffffffu, m);
    if (!bal) return;
    const int lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == __ffs(bal) - 1) base = atomicAdd(cnt, (unsigned long long)__popc(bal));
    base = __shfl_sync(0xffffffffu, base, __ffs(bal) - 1);
    if (m) {
        const uint64_t o = base + __popc(bal & lanemask_lt());
        if (o < cap) list[o] = (uint32_t)i;
    }
}

__device__ __forceinline__ uint64_t hi_lower_bound(uint64_t const* keys, uint64_t lo, uint64_t hi, uint32_t h) {
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if ((uint32_t)(keys[mid] >> 32) < h)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// For each (sorted) mismatch position: the run of its top 32 bits [s, e),
// and whether it is the run's first mismatch (the run's representative).
__global__ void k_hi_runs(uint64_t const* __restrict__ keys, uint64_t n, uint32_t const* __restrict__ list,
                          uint64_t nm, uint64_t* __restrict__ rs, uint64_t* __restrict__ len) {
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nm) return;
    const uint64_t i = list[j];
    const uint32_t h = (uint32_t)(keys[i] >> 32);
    const uint64_t s = hi_lower_bound(keys, 0, i, h);
    const uint64_t e = h == 0xffffffffu ? n : hi_lower_bound(keys, i, n, h + 1);
    const bool rep = j == 0 || list[j - 1] < s;
    rs[j] = s;
    len[j] = rep ? e - s : 0;
}

__device__ __forceinline__ uint64_t upper_bound_off(uint64_t const* a, uint64_t n, uint64_t x) {
    uint64_t lo = 0, hi = n;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (a[mid] <= x)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Compact element j of the mixed runs: run r (by its compact offset) and its
// position in the full array.
__device__ __forceinline__ uint64_t hi_pos(uint64_t const* off, uint64_t const* rs, uint64_t nm, uint64_t j,
                                           uint64_t& r) {
    // the last entry starting at or before j; entries that are not their
    // run's representative have length 0 and follow it, so they start after j
    r = upper_bound_off(off, nm + 1, j) - 1;
    return rs[r] + (j - off[r]);
}

__global__ void k_hi_gather_keys(uint64_t const* __restrict__ keys, uint64_t const* __restrict__ off,
                                 uint64_t const* __restrict__ rs, uint64_t nm, uint64_t M,
                                 uint64_t* __restrict__ ckey, uint32_t* __restrict__ cpos) {
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= M) return;
    uint64_t r;
    const uint64_t q = hi_pos(off, rs, nm, j, r);
    ckey[j] = ((uint64_t)r << 32) | (uint32_t)keys[q];
    cpos[j] = (uint32_t)q;
}

template <typename V>
__global__ void k_hi_permute(uint64_t const* __restrict__ keys, V const* __restrict__ vals,
                             uint32_t const* __restrict__ cpos, uint64_t M, uint64_t* __restrict__ tk,
                             V* __restrict__ tv) {
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= M) return;
    tk[j] = keys[cpos[j]];
    tv[j] = vals[cpos[j]];
}

template <typename V>
__global__ void k_hi_scatter(uint64_t* __restrict__ keys, V* __restrict__ vals, uint64_t const* __restrict__ off,
                             uint64_t const* __restrict__ rs, uint64_t nm, uint64_t M,
                             uint64_t const* __restrict__ tk, V const* __restrict__ tv) {
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= M) return;
    uint64_t r;
    const uint64_t q = hi_pos(off, rs, nm, j, r);
    keys[q] = tk[j];
    vals[q] = tv[j];
}

// Stable sort of (u64 keys, vals) by all 64 key bits -- the same order as an
// 8-pass LSD sort -- in 4 passes over the top 32 bits: keys that tie on those
// bits but differ below them (rare when the top bits are a hash) are found
// afterwards, and only their runs are sorted again on (run, low 32 bits).
// n < 2^32; `iota` as in radix_sort_pairs.
template <typename V>
void sort_pairs_u64_exact(uint64_t* keys, V* vals, uint64_t n, dev_arena& A, cudaStream_t st, uint32_t* err,
                          bool iota = false) {
    if (n == 0 || (n == 1 && !iota)) return;
    if (n >= (1ull << 32)) throw std::runtime_error("sort_pairs_u64_exact: n >= 2^32");
    if (n <= RS_SMALL) {  // all 64 bits in the one launch
        radix_sort_small<V, uint64_t>(keys, vals, n, 0, 64, st, iota);
        return;
    }
    radix_sort_pairs<V, uint64_t>(keys, vals, n, 32, 64, A, st, err, iota);
    auto m = A.mark();
    const uint64_t cap = n / 8 + 1024;
    uint32_t* list = A.alloc<uint32_t>(cap);
    unsigned long long* cnt = A.alloc<unsigned long long>(1);
    CDBG_CUDA(cudaMemsetAsync(cnt, 0, 8, st));
    {
        CDBG_PROF("k_hi_mismatch", st);
        k_hi_mismatch<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(keys, n, list, cnt, cap);
    }
    CDBG_CHECK_LAUNCH();
    unsigned long long nm = 0;
    read_small(&nm, cnt, 8, st);
    if (nm > cap) {
        // far from a hash: the full stable sort of the (already top-sorted)
        // pairs gives the same order as sorting the input
        A.release(m);
        radix_sort_pairs<V, uint64_t>(keys, vals, n, 0, 64, A, st, err);
        return;
    }
    if (nm == 0) {
        A.release(m);
        return;
    }
    uint32_t* dummy = A.alloc<uint32_t>(nm);
    radix_sort_pairs<uint32_t, uint32_t>(list, dummy, nm, 0, 32, A, st, err);
    uint64_t* rs = A.alloc<uint64_t>(nm);
    uint64_t* len = A.alloc<uint64_t>(nm);
    uint64_t* off = A.alloc<uint64_t>(nm + 1);
    k_hi_runs<<<(unsigned)ceil_div(nm, 256), 256, 0, st>>>(keys, n, list, nm, rs, len);
    CDBG_CHECK_LAUNCH();
    exclusive_scan<uint64_t, uint64_t>(len, off, nm, A, st, off + nm);
    uint64_t M = 0;
    read_small(&M, off + nm, 8, st);
    uint64_t* ckey = A.alloc<uint64_t>(M);
    uint32_t* cpos = A.alloc<uint32_t>(M);
    k_hi_gather_keys<<<(unsigned)ceil_div(M, 256), 256, 0, st>>>(keys, off, rs, nm, M, ckey, cpos);
    CDBG_CHECK_LAUNCH();
    int rb = 1;
    while ((1ull << rb) < nm) ++rb;
    radix_sort_pairs<uint32_t, uint64_t>(ckey, cpos, M, 0, 32 + rb, A, st, err);
    uint64_t* tk = A.alloc<uint64_t>(M);
    V* tv = A.alloc<V>(M);
    k_hi_permute<V><<<(unsigned)ceil_div(M, 256), 256, 0, st>>>(keys, vals, cpos, M, tk, tv);
    CDBG_CHECK_LAUNCH();
    k_hi_scatter<V><<<(unsigned)ceil_div(M, 256), 256, 0, st>>>(keys, vals, off, rs, nm, M, tk, tv);
    CDBG_CHECK_LAUNCH();
    A.release(m);
}

}  // namespace
}  // namespace prim
}  // namespace cdbg
