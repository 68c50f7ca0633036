// Which form of the extension-mask pass a bucket takes, and in how many blocks.
// Plain C++: also compiled on the host alone.
#pragma once

#include <stdint.h>

#include <algorithm>

namespace cdbg {

// The three forms: a filter of the bucket's keys in shared memory, a wide filter
// (128-bit k-mers), no filter (flat).
enum : int { EXT_FILTER = 0, EXT_WIDE = 1, EXT_FLAT = 2 };

struct ext_plan {
    // A filter pays up to these many occurrences: its keys fill it beyond.  us per
    // million k-mers by distinct k-mers per bucket, filter / flat: k = 31: 63 K 28.8
    // / 50, 111 K 36 / 50, 189 K (about 2^18 occurrences) 54 / 50, 473 K 133 / 50; k
    // = 63: 77 K 52 / 92, 139 K 66 / 93, 348 K 148 / 94.  The wide filter of 128-bit
    // k-mers takes twice the shared memory in one block of twice the threads per SM
    // (the same warps): wide / flat at 272 K occurrences per bucket 68 / 96, 340 K 77 /
    // 96, 504 K 109 / 100; 64-bit ones would lose half their warps: 480 K 52 / 51.
    static constexpr uint64_t FILTER_OCC = 1u << 18;
    static constexpr uint64_t SMS = 148;

    uint64_t wide_occ;   // most occurrences of a bucket with any filter
    uint64_t spread;     // see cut()
    uint64_t block_occ;  // what a filter block costs beside its keys
    uint64_t flat_max;   // occurrences of a flat block where the SMs are busy
    uint64_t share;      // of the batch's occurrences, about four per resident block

    // Flat blocks: four or two rounds of their threads; fewer leave threads idle,
    // more put the tables of too many buckets in flight for L2 (k = 31: 57 / 54 / 50 /
    // 56 / 88 us per million k-mers at 256 / 512 / 1024 / 2048 / 4096; k = 63: 98 / 93 /
    // 98 / 120 / 156).
    ext_plan(bool wide_keys, uint64_t batch_occ)
        : wide_occ(wide_keys ? 7u << 16 : FILTER_OCC),
          spread(wide_keys ? 6 : 8),
          block_occ(wide_keys ? 220 : 350),
          flat_max(wide_keys ? 512 : 1024),
          share(std::max<uint64_t>(16384, batch_occ / (SMS * 8))) {}

    // Blocks of a filter form for a bucket of n occurrences: each reads all the
    // bucket's keys, for its part of them.
    uint64_t parts(uint64_t n) const { return n > share + share / 2 ? (n + share - 1) / share : 1; }

    // Buckets of a group (occurrences off[i + 1] - off[i], nb of them) of at least
    // this many occurrences go flat.  Where a group's buckets are few, a filter's
    // blocks leave most SMs idle and the longest, which reads its bucket's keys and
    // looks its part up, is the time; where they are small, a block's launch and its
    // filter are.  A flat pass spreads over the chip whatever the buckets are.  In
    // occurrences at the flat rate, plus launches:
    //   filter  max(half of them + block_occ a block, (n + n / parts(n)) * 2 SMS / spread) + 100 K
    //   flat    their number + 600 K
    // and the cut by powers of two that costs least.  Masks and links, us per million
    // k-mers with the filter wherever the keys fit / by this rule / eight probes for
    // all: k = 63, 8e6 bases, 100 K occurrences a bucket 107 / 107 / 135, 400 K 237 /
    // 134 / 137; twenty similar genomes of 0.4e6 bases in 7 buckets 307 / 136 / 125; k =
    // 31, a genome of 8e6, 110 K 55 / 54 / 90, 230 K 91 / 72 / 90.
    uint64_t cut(uint64_t const* off, uint64_t nb) const {
        uint64_t sum[65] = {}, most[65] = {}, blk[65] = {};  // by the size's bits; [64]: too large for a filter
        uint64_t flat = 0, filter = 0, blocks = 0, best = ~0ull, at = 0;
        for (uint64_t b = 0; b < nb; ++b) {
            const uint64_t n = off[b + 1] - off[b];
            const int c = n > wide_occ ? 64 : n ? 64 - __builtin_clzll(n) : 0;
            sum[c] += n;
            most[c] = std::max(most[c], n);
            blk[c] += parts(n);
            flat += n;
        }
        for (int c = 0; c < 64; ++c) {  // buckets below 2^c by a filter
            if (c && !sum[c]) continue;
            if (c) blocks += blk[c];
            filter += sum[c];
            flat -= sum[c];
            const uint64_t n = most[c];
            uint64_t cost = flat ? flat + 600000 : 0;
            if (filter)
                cost += 100000 + std::max(filter / 2 + block_occ * blocks, (n + n / parts(n)) * 2 * SMS / spread);
            if (cost <= best) {
                best = cost;
                at = 1ull << c;
            }
        }
        return at;
    }
    int form(uint64_t n, uint64_t cut) const { return n >= cut || n > wide_occ ? EXT_FLAT : n > FILTER_OCC ? EXT_WIDE : EXT_FILTER; }
    // Occurrences of a flat block of a group of tn: one round of its threads where
    // more would leave SMs idle.
    uint32_t flat_occ(uint64_t tn) const {
        return (uint32_t)std::min(flat_max, (tn / (SMS * 8) / 256 + 1) * 256);
    }
    // Flat blocks over several buckets at a time, for `count` buckets of `sum`
    // occurrences together: below four blocks' worth each.  us per million k-mers of
    // masks and links, a block per bucket at least / packed / eight probes for all: k
    // = 31, 8e6 bases in buckets of 30 543 / 57 / 56, of 125 179 / 66 / 65; in buckets
    // of 300 K 66 / 70 / 87 (the search of each k-mer's bucket).
    bool packed(uint64_t sum, uint64_t count, uint64_t tn) const { return sum < 4 * count * flat_occ(tn); }
};

}  // namespace cdbg
