// What one ACGT run adds to the run table's sums, and the widths those sums
// need.  Plain C++: also compiled on the host.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define CDBG_HD __host__ __device__ __forceinline__
#else
#define CDBG_HD inline
#endif

namespace cdbg {

// A look-back status word holds a sum of this many bits beside its 2-bit flag.
constexpr int LOOKBACK_SUM_BITS = 62;

// Runs of one input: their indices are 32-bit, the largest value is "none".
constexpr uint64_t MAX_RAW_RUNS = 0xfffffffeull;
// Bases of one run.
constexpr uint64_t MAX_RUN_BASES = 0xfffffffeull;

struct run_sums {
    uint64_t runs, words, tiles;
};
// A run of l bases: itself, its words of 32 bases and its minimizer tiles of tt
// (k-1)-mers when it has at least k bases, nothing otherwise.
CDBG_HD run_sums run_adds(uint64_t l, uint32_t k, uint32_t tt) {
    if (l < k) return run_sums{0, 0, 0};
    return run_sums{1, (l + 31) / 32, (l - k + 2 + tt - 1) / tt};
}

}  // namespace cdbg
