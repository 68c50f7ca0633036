// Phase 2 (bucket-process) kernels for sm_100a.
//
// Restates phase2_bucket_process/bucket_walker.hpp:166-779 on the device.
// Buckets are processed in batches (consecutive buckets whose k-mer
// occurrences fit a budget); every batch runs the same stages:
//
//  load     one thread per k-mer occurrence rolls its canonical k-mer straight
//           from the 2-bit record stream and aggregates it into its bucket's
//           open-addressing table (load_bucket, bucket_walker.hpp:166-255):
//           boundary side bits and `primary` OR-ed, the first owning record
//           plus a second-owner bit, and the first-insertion rank (the
//           occurrence index, in (record, index) order) by atomicMin.
//  nodes    distinct k-mers are numbered in first-insertion order -- the
//           iteration order of the reference's insertion-ordered map, which is
//           its seed and class order -- by one scan over the batch's
//           occurrences: an occurrence is its k-mer's first when the slot says so.
//  resolve  a primary k-mer owned by one record has that record's color set;
//           one owned by several records gets the union of their sets
//           (bucket_walker.hpp:360-428), built once per run of k-mers with the
//           same owning records in a per-warp shared-memory bitmap.  Sets are
//           hashed (order-independent 64-bit set hash) and
//           interned in a global device dictionary with full list equality;
//           new classes get global ids in order of first appearance (bucket,
//           then insertion rank), which is the id order of the reference's
//           streaming_color_set_dict when buckets are merged in order
//           (bucket_walker.hpp:713-757, streaming_color_set_dict.hpp:148-182).
//           New classes are hybrid-encoded (hybrid_color_sets.hpp:48-95) into
//           the .color_sets bit vector.
//  walk     8-neighbour extension masks (local_ext_mask, :260-271) and the
//           clean-step links of walk_step (:317-336).  Clean links pair the
//           ports of k-mers into disjoint chains (paths and cycles); one thread
//           per chain replays the reference's sequential seed loop restricted
//           to that chain (emit_from_seed, :451-566): seeds in insertion order,
//           a shared visited set, contig-break stops and the seed shortcuts.
//           Chains never interact, so this equals the whole-bucket loop.
//  emit     fragments in seed order, serialized in the frag_unitig_writer
//           record layout (unitig_spill.hpp:491-522) with global class ids.

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "device_kmer.cuh"
#include "ext_plan.hpp"
#include "phase2.cuh"
#include "primitives.cuh"

namespace cdbg {

namespace {

constexpr uint32_t NONE32 = 0xffffffffu;
constexpr uint32_t MULTI_TAG = 0x80000000u;
constexpr uint32_t M_LEFT = 1, M_RIGHT = 2, M_PRIMARY = 4;
constexpr uint32_t M_MULTI = 8;  // table only: owned by two or more records
constexpr uint32_t SK_BEGIN = 1, SK_END = 2, SK_OWNS_FIRST = 4, SK_OWNS_LAST = 8;
constexpr uint64_t HASH_EMPTY = ~0ull;

inline unsigned grid(uint64_t n, unsigned t) { return (unsigned)ceil_div(n, t); }

template <typename T>
T read_dev(T const* p, cudaStream_t st) {
    T v;
    read_small(&v, p, sizeof(T), st);
    return v;
}

__device__ __forceinline__ uint32_t upper_bound_u64(uint64_t const* a, uint64_t n, uint64_t x) {
    uint64_t lo = 0, hi = n;
    while (lo < hi) {
        uint64_t mid = (lo + hi) >> 1;
        if (a[mid] <= x)
            lo = mid + 1;
        else
            hi = mid;
    }
    return (uint32_t)lo;
}

// upper_bound(off, n1, x) - 1 (the bucket of x, `off` ascending) for the
// active lanes of a warp whose x ascend with the lane (consecutive records or
// occurrences, so nearly always one bucket): the first active lane searches,
// the others take its bucket when x lies in its range and search otherwise.
// Every lane of the warp calls it.
__device__ __forceinline__ uint32_t warp_bucket_of(uint64_t const* off, uint64_t n1, uint64_t x, bool active) {
    const uint32_t am = __ballot_sync(0xffffffffu, active);
    if (!am) return 0;
    const int leader = __ffs(am) - 1;
    const uint64_t xl = __shfl_sync(0xffffffffu, x, leader);
    uint32_t b = 0;
    if ((int)(threadIdx.x & 31) == leader) b = upper_bound_u64(off, n1, xl) - 1;
    b = __shfl_sync(0xffffffffu, b, leader);
    if (active && !(off[b] <= x && x < off[b + 1])) b = upper_bound_u64(off, n1, x) - 1;
    return b;
}

// ------------------------------------------------------------------ set hash
// Order-independent hash of a color set: the sum, over the 32-color words
// that hold at least one color, of a mix of (word index, word bits), then
// mixed with the set size.  A list and a bitmap of the same set hash alike;
// one mix per nonzero word instead of one per color.
__host__ __device__ __forceinline__ uint64_t word_mix(uint32_t w, uint32_t bits) {
    return mix64((((uint64_t)w << 32) | bits) * 0x9E3779B97F4A7C15ULL + 0x632BE59BD9B4E019ULL);
}
// Sum of word_mix over an ascending color list.
__host__ __device__ __forceinline__ uint64_t list_word_sum(uint32_t const* c, uint64_t n) {
    uint64_t acc = 0;
    uint32_t cw = 0xffffffffu, bits = 0;
    for (uint64_t i = 0; i < n; ++i) {
        const uint32_t v = c[i], w = v >> 5;
        if (w != cw) {
            if (bits) acc += word_mix(cw, bits);
            cw = w;
            bits = 0;
        }
        bits |= 1u << (v & 31);
    }
    if (bits) acc += word_mix(cw, bits);
    return acc;
}
__host__ __device__ __forceinline__ uint64_t set_hash_final(uint64_t acc, uint64_t n) {
    uint64_t h = mix64(acc ^ (n * 0xD6E8FEB86659FD93ULL));
    return h == HASH_EMPTY ? HASH_EMPTY - 1 : h;
}

// ------------------------------------------------------------------ tables
__device__ __forceinline__ u128 key_cas(u128* a, u128 cmp, u128 val) {
    uint64_t olo, ohi;
    const uint64_t clo = (uint64_t)cmp, chi = (uint64_t)(cmp >> 64);
    const uint64_t vlo = (uint64_t)val, vhi = (uint64_t)(val >> 64);
    asm volatile(
        "{\n\t.reg .b128 d, c, v;\n\t"
        "mov.b128 c, {%2, %3};\n\t"
        "mov.b128 v, {%4, %5};\n\t"
        "atom.global.cas.b128 d, [%6], c, v;\n\t"
        "mov.b128 {%0, %1}, d;\n\t}"
        : "=l"(olo), "=l"(ohi)
        : "l"(clo), "l"(chi), "l"(vlo), "l"(vhi), "l"(a)
        : "memory");
    return ((u128)ohi << 64) | (u128)olo;
}

// One table slot: everything the load stage aggregates for a k-mer in 16
// bytes (32 for 128-bit k-mers), two slots per 32-byte sector.
//   rank  first insertion: the batch's lowest occurrence index of the k-mer
//         (occurrences are in (record, index) order)
//   om    bits 0-3: side bits, primary, M_MULTI; bits 4-31: the first owning
//         record (relative to the batch) + 1, 0 when none
template <typename K>
struct slot_t;
template <>
struct alignas(16) slot_t<uint64_t> {
    uint64_t key;
    uint32_t rank;
    uint32_t om;
};
template <>
struct alignas(16) slot_t<u128> {
    u128 key;
    uint32_t rank;
    uint32_t om;
    uint64_t pad;
};
static_assert(sizeof(slot_t<uint64_t>) == 16, "slot layout");
static_assert(sizeof(slot_t<u128>) == 32, "slot layout");
constexpr uint64_t MAX_BATCH_RECORDS = (1ull << 28) - 2;  // owner field of `om`

// Probing is linear.  64-bit-key slots go by pairs of neighbours (a sector): from
// pair slot_home(x, cap / 2) on, both slots read by one 32-byte load and taken in
// order, until x or an empty slot.  A probe is a dependent read, and a warp waits
// for its longest: at the load of a 200-genome build (1/3) single slots take 1.24
// steps found / 1.58 absent and 3.6 for the slowest of 32, pairs 1.04 / 1.1 and 2
// (k_insert of that build 10.0 -> 9.6 ms).  128-bit-key slots fill a sector each
// and go one by one from slot_home(x, cap): pairs read two sectors where one
// mostly decides (neighbour lookups 86 -> 100 us per million k-mers).
// The hash: the key folded to 64 bits, an odd-constant multiply, and its top 32
// bits scaled to the number of homes (< 2^32).  Table positions decide no output
// (nodes are numbered by first occurrence, not by slot), only probe lengths.
__device__ __forceinline__ uint32_t slot_hash(uint64_t x) {
    return (uint32_t)(((x ^ (x >> 31)) * 0x9e3779b97f4a7c15ULL) >> 32);
}
__device__ __forceinline__ uint32_t slot_hash(u128 x) {
    return slot_hash((uint64_t)((uint64_t)x ^ ((uint64_t)(x >> 64) * 0xc2b2ae3d27d4eb4fULL)));
}
template <typename K>
__device__ __forceinline__ uint32_t slot_home(K x, uint32_t homes) {
    return __umulhi(slot_hash(x), homes);
}

// Keys and (rank | om << 32) of a pair of 64-bit-key slots in one 32-byte load
// past L1.
__device__ __forceinline__ void pair_load(slot_t<uint64_t> const* e, uint64_t& k0, uint64_t& v0, uint64_t& k1,
                                          uint64_t& v1) {
    asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(k0), "=l"(v0), "=l"(k1), "=l"(v1)
                 : "l"(e)
                 : "memory");
}
// A 128-bit key, whole.
__device__ __forceinline__ u128 key_load(u128 const* e) {
    uint64_t lo, hi;
    asm volatile("{\n\t.reg .b128 d;\n\tld.relaxed.gpu.global.b128 d, [%2];\n\tmov.b128 {%0, %1}, d;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(e)
                 : "memory");
    return ((u128)hi << 64) | (u128)lo;
}

// Insert-or-find of x by the occurrence whose payload is `payload` (rank | om <<
// 32, what the slot of a new k-mer gets); returns the slot (absolute) or ~0 when
// the region is full.  `claimed` tells whether this call stored the payload;
// otherwise `ro` receives the slot's (rank | om << 32) as read while probing: a
// value the slot held, so possibly older than the current one (rank only falls
// and om only gains bits, which the caller's updates rely on).  `slots` holds
// the slots from absolute index off0 on (the tables of the bucket group being
// processed); returned indices are absolute.
// A 64-bit key is claimed together with its payload in one 128-bit
// compare-and-swap of the whole slot.
__device__ __forceinline__ uint64_t table_claim(slot_t<uint64_t>* slots, uint64_t off0, uint64_t off, uint64_t cap,
                                                uint64_t x, uint64_t payload, uint64_t& ro, bool& claimed) {
    const uint64_t EMPTY = kmer_ops<uint64_t>::empty();
    const uint32_t pairs = (uint32_t)(cap / 2);
    uint32_t p = slot_home(x, pairs);
    claimed = false;
    for (uint32_t i = 0; i < pairs; ++i) {
        slot_t<uint64_t>* e = &slots[off + 2 * (uint64_t)p - off0];
        uint64_t key[2], v[2];
        pair_load(e, key[0], v[0], key[1], v[1]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if (key[j] == EMPTY) {
                const u128 old = key_cas(reinterpret_cast<u128*>(e + j), ((u128)v[j] << 64) | (u128)EMPTY,
                                         ((u128)payload << 64) | (u128)x);
                key[j] = (uint64_t)old;
                if (key[j] == EMPTY && (uint64_t)(old >> 64) == v[j]) {
                    claimed = true;
                    return off + 2 * (uint64_t)p + j;
                }
                v[j] = (uint64_t)(old >> 64);
            }
            if (key[j] == x) {
                ro = v[j];
                return off + 2 * (uint64_t)p + j;
            }
        }
        p = p + 1 == pairs ? 0u : p + 1;
    }
    return ~0ull;
}
// A 128-bit key is claimed first and its payload stored by a second
// compare-and-swap of (rank, om), which fails only against another occurrence
// of the same k-mer.
__device__ __forceinline__ uint64_t table_claim(slot_t<u128>* slots, uint64_t off0, uint64_t off, uint64_t cap,
                                                u128 x, uint64_t payload, uint64_t& ro, bool& claimed) {
    const u128 EMPTY = kmer_ops<u128>::empty();
    const uint32_t cap32 = (uint32_t)cap;
    uint32_t p = slot_home(x, cap32);
    claimed = false;
    for (uint32_t i = 0; i < cap32; ++i) {
        slot_t<u128>* e = &slots[off + p - off0];
        u128 key = key_load(&e->key);
        if (key == EMPTY) {
            key = key_cas(&e->key, EMPTY, x);
            if (key == EMPTY) {
                const unsigned long long was = (unsigned long long)NONE32;
                ro = atomicCAS(reinterpret_cast<unsigned long long*>(&e->rank), was, payload);
                claimed = ro == was;
                return off + p;
            }
        }
        if (key == x) {
            ro = *(volatile uint64_t const*)&e->rank;
            return off + p;
        }
        p = p + 1 == cap32 ? 0u : p + 1;
    }
    return ~0ull;
}

struct rec_view {
    uint64_t const* start;
    uint32_t const* len;
    uint32_t const* flags;
    uint64_t const* col_off;
    uint32_t const* colors;
    uint32_t const* bucket;   // per record
    uint64_t const* occ;      // n + 1 exclusive prefix of k-mers per record
    uint64_t const* words;
};

// The k-mer tables of buckets b0, b0 + 1, ...: bucket b0 + i's table is
// the tab_cap[i] slots from absolute slot tab_off[i]; `slots` holds the slots
// from absolute index off0 on (one bucket group's tables at a time).
template <typename K>
struct tables {
    slot_t<K>* slots;
    uint64_t const* tab_off;
    uint64_t const* tab_cap;
    uint32_t b0;
    uint64_t off0;
};

// Occurrence o of the batch -> (record, index, canonical k-mer, contrib, owned).
template <typename K>
struct occ_info {
    uint32_t r;
    uint32_t idx;
    K can;
    uint32_t contrib;
    bool owned;
};

// Records of a tile of WORDS x 32 consecutive occurrences (a multiple of
// OCC_BLOCK, starting on one): the records that start in the tile mark their
// first occurrence in a bitmap, and an occurrence's record is the one of the
// nearest mark at or before it, or the tile's first record (r0).  One read of
// the tile's record prefix instead of a search per occurrence; records without
// k-mers mark nothing.
constexpr int OCC_BLOCK = 256;
template <int WORDS>
struct tile_records {
    uint32_t bits[WORDS];
    uint32_t at[WORDS * 32];  // record of each mark, from r0
};
// blk_rec[b] = the record holding occurrence O0 + b * OCC_BLOCK, the first
// occurrence of block b of the occurrence kernels (thread per record; a
// record spans at most a few block starts).
__global__ void k_block_records(uint64_t const* __restrict__ occ, uint64_t R0, uint64_t nrec, uint64_t O0,
                                uint64_t nblocks, uint32_t* __restrict__ blk_rec) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrec) return;
    const uint64_t a = occ[R0 + i] - O0, e = occ[R0 + i + 1] - O0;
    for (uint64_t b = (a + OCC_BLOCK - 1) / OCC_BLOCK; b * OCC_BLOCK < e && b < nblocks; ++b)
        blk_rec[b] = (uint32_t)(R0 + i);
}

// Whole block; blk = the tile's first occurrence block.
template <int WORDS>
__device__ __forceinline__ uint32_t load_tile_records(tile_records<WORDS>& w, uint64_t const* __restrict__ occ,
                                                      uint64_t R0, uint64_t nrec, uint64_t O0, uint64_t nblk,
                                                      uint32_t const* __restrict__ blk_rec, uint64_t blk) {
    static_assert(WORDS * 32 % OCC_BLOCK == 0, "whole occurrence blocks");
    const uint64_t nb = blk + WORDS * 32 / OCC_BLOCK;
    const uint32_t r0 = blk_rec[blk];
    const uint32_t r1 = nb < nblk ? blk_rec[nb] : (uint32_t)(R0 + nrec - 1);
    const uint64_t o0 = O0 + blk * OCC_BLOCK;
    for (uint32_t i = threadIdx.x; i < (uint32_t)WORDS; i += blockDim.x) w.bits[i] = 0;
    __syncthreads();
    for (uint32_t r = r0 + 1 + threadIdx.x; r <= r1; r += blockDim.x) {
        const uint64_t x = occ[r] - o0;
        if (x < (uint64_t)WORDS * 32 && occ[r + 1] - o0 > x) {
            atomicOr(&w.bits[x >> 5], 1u << (x & 31));
            w.at[x] = r - r0;
        }
    }
    __syncthreads();
    return r0;
}
// Record of occurrence `bit` of the tile's word `i`.
template <int WORDS>
__device__ __forceinline__ uint32_t tile_record(tile_records<WORDS> const& w, uint32_t r0, int i, uint32_t bit) {
    uint32_t x = w.bits[i] & (0xffffffffu >> (31 - bit));
    while (x == 0 && i > 0) x = w.bits[--i];
    return x ? r0 + w.at[i * 32 + 31 - __clz(x)] : r0;
}

template <typename K>
__device__ __forceinline__ occ_info<K> decode_occ_r(rec_view const& R, uint64_t r, uint64_t o, uint32_t k) {
    occ_info<K> oi;
    oi.r = (uint32_t)r;
    oi.idx = (uint32_t)(o - R.occ[r]);
    const uint32_t nk = R.len[r] - k + 1;
    const uint32_t f = R.flags[r];
    K fwd, rc;
    kmer_ops<K>::load(R.words, R.start[r] + oi.idx, k, fwd, rc);
    const bool isf = fwd <= rc;
    oi.can = isf ? fwd : rc;
    uint32_t contrib = 0;
    if (!(f & SK_BEGIN) && oi.idx == 0) contrib |= isf ? M_LEFT : M_RIGHT;
    if (!(f & SK_END) && oi.idx == nk - 1) contrib |= isf ? M_RIGHT : M_LEFT;
    oi.contrib = contrib;
    oi.owned = !((oi.idx == 0 && !(f & SK_OWNS_FIRST)) || (oi.idx == nk - 1 && !(f & SK_OWNS_LAST)));
    return oi;
}

// ------------------------------------------------------------------ kernels
__global__ void k_rec_prep(uint64_t n, uint32_t const* __restrict__ len, uint32_t k,
                           uint64_t const* __restrict__ bstart, uint32_t B,
                           uint64_t* __restrict__ nk, uint32_t* __restrict__ rbucket,
                           uint64_t const* __restrict__ col_off, uint32_t const* __restrict__ colors,
                           uint64_t* __restrict__ rhash) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t b = warp_bucket_of(bstart, (uint64_t)B + 1, r, r < n);
    if (r >= n) return;
    const uint32_t l = len[r];
    nk[r] = l >= k ? (uint64_t)(l - k + 1) : 0;
    rbucket[r] = b;
    const uint64_t c0 = col_off[r], c1 = col_off[r + 1];
    rhash[r] = set_hash_final(list_word_sum(colors + c0, c1 - c0), c1 - c0);
}

__global__ void k_gather_u64(uint64_t n, uint64_t const* __restrict__ src,
                             uint64_t const* __restrict__ idx, uint64_t* __restrict__ out) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = src[idx[i]];
}

template <typename K>
__global__ void k_init_tables(uint64_t T, slot_t<K>* slots) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T) return;
    slot_t<K> e;
    e.key = kmer_ops<K>::empty();
    e.rank = NONE32;
    e.om = 0;
    if constexpr (sizeof(K) == 16) e.pad = 0;
    slots[i] = e;
}

// Occurrences t0 .. t1 - 1 of the batch (one bucket group's), one per thread
// and one OCC_BLOCK per block.
template <typename K>
__global__ void __launch_bounds__(OCC_BLOCK, 8) k_insert(rec_view R, tables<K> T, uint64_t R0, uint64_t nrec,
                                                uint64_t O0, uint64_t t0, uint64_t t1, uint32_t k,
                                                uint64_t nblk, uint32_t const* __restrict__ blk_rec,
                                                uint32_t* __restrict__ occ_slot, uint32_t* err) {
    __shared__ tile_records<OCC_BLOCK / 32> win;
    const uint64_t blk = t0 / OCC_BLOCK + blockIdx.x;
    const uint32_t r0 = load_tile_records(win, R.occ, R0, nrec, O0, nblk, blk_rec, blk);
    const uint64_t t = blk * OCC_BLOCK + threadIdx.x;
    if (t < t0 || t >= t1) return;
    const uint64_t rec = tile_record(win, r0, threadIdx.x >> 5, threadIdx.x & 31);
    const occ_info<K> oi = decode_occ_r<K>(R, rec, O0 + t, k);
    const uint32_t tb = R.bucket[oi.r] - T.b0;
    const uint32_t mo = oi.contrib | (oi.owned ? M_PRIMARY : 0u);
    const uint32_t own = (uint32_t)(oi.r - R0 + 1) << 4;
    uint64_t ro = 0;
    bool claimed = false;
    // a new k-mer's slot: rank t, and om as the updates below would leave it
    const uint32_t om0 = oi.owned ? (own | mo) : mo;
    const uint64_t s = table_claim(T.slots, T.off0, T.tab_off[tb], T.tab_cap[tb], oi.can,
                                   (uint64_t)(uint32_t)t | ((uint64_t)om0 << 32), ro, claimed);
    if (s == ~0ull) {
        set_error(err, ERR_TABLE_FULL);
        occ_slot[t] = NONE32;
        return;
    }
    // slot of this occurrence, bit 31 = owned (read by k_number)
    occ_slot[t] = (uint32_t)s | (oi.owned ? 0x80000000u : 0u);
    if (claimed) return;
    // rank and om as read while probing (never newer than the slot): the
    // reduction and the updates below stay correct, and a k-mer whose slot
    // already holds everything this occurrence adds costs no further access
    slot_t<K>& e = T.slots[s - T.off0];
    if ((uint32_t)t < (uint32_t)ro) atomicMin(&e.rank, (uint32_t)t);
    uint32_t old = (uint32_t)(ro >> 32);
    if (!oi.owned) {
        if (mo && (old & mo) != mo) atomicOr(&e.om, mo);
        return;
    }
    // owner: the first owning record, M_MULTI once a second one appears.
    // `om` only gains bits, so the loop ends after a few changes by others.
    for (int it = 0;; ++it) {
        const uint32_t cur = old & ~0xfu;
        const uint32_t want = (cur == own || (old & M_MULTI)) ? (old | mo)
                              : (cur == 0)                   ? (old | own | mo)
                                                             : (old | M_MULTI | mo);
        if (want == old) break;
        const uint32_t prev = atomicCAS(&e.om, old, want);
        if (prev == old) break;
        old = prev;
        if (it == 64) {
            set_error(err, ERR_CAPACITY);
            break;
        }
    }
}

// Occurrence words: for the 32 occurrences 32 i .. 32 i + 31 of the batch, x =
// which of them are the first of their k-mer, y = the node index of the first
// such one (the number of first occurrences before the word).  A k-mer's slot
// keeps its first occurrence q (`rank`), so its node index is node_of(fw, q).
__device__ __forceinline__ uint32_t node_of(uint2 const* __restrict__ fw, uint32_t q) {
    const uint2 w = __ldg(fw + (q >> 5));
    return w.y + __popc(w.x & ((1u << (q & 31)) - 1u));
}

__device__ __forceinline__ void slot_read(slot_t<uint64_t> const* e, uint64_t& key, uint32_t& rank, uint32_t& om) {
    const ulonglong2 v = __ldg(reinterpret_cast<ulonglong2 const*>(e));
    key = v.x;
    rank = (uint32_t)v.y;
    om = (uint32_t)(v.y >> 32);
}
__device__ __forceinline__ void slot_read(slot_t<u128> const* e, u128& key, uint32_t& rank, uint32_t& om) {
    const ulonglong2 v = __ldg(reinterpret_cast<ulonglong2 const*>(e));
    const uint2 ro = __ldg(reinterpret_cast<uint2 const*>(&e->rank));
    key = ((u128)v.y << 64) | (u128)v.x;
    rank = ro.x;
    om = ro.y;
}

// Node numbering and multi-record pairs of one bucket group, in one pass over
// its occurrences t0 .. t1 - 1 (one slot read each):
//   - occurrence t is the first of its k-mer iff the slot's rank is t; its node
//     index is base[0] plus the number of first occurrences before it in the
//     group (insertion order), and it writes the k-mer's node arrays;
//   - an owned occurrence of a multi-record k-mer (M_PRIMARY and M_MULTI)
//     emits the pair (first occurrence of the k-mer, record), in occurrence
//     order from pair base[1] on: records ascend within a k-mer, so a stable
//     sort by k-mer alone orders the pairs.
// Tiles of NB_ROUNDS x 256 occurrences from ta (t0's occurrence block) take
// indices in launch order and find both offsets by one decoupled look-back
// (nodes in the low 31 bits, pairs above: a batch has fewer than 2^31
// occurrences); the last tile stores both totals in next[].
// Bound: random 16-byte slot reads (L2 sectors), all of a thread's in flight
// together.  A scan of the table for first occurrences, node numbering that
// stored the index back into the slot, and a separate pair pass took 14.5 ms of
// a 200-genome k = 31 build (3.8e8 occurrences), this pass and the pair
// conversion 5.2; 9.8 and 3.8 ms of a 60-genome k = 63 build.
constexpr int NB_ROUNDS = 8;
template <typename K>
__global__ void __launch_bounds__(256) k_number(uint64_t ta, uint64_t t0, uint64_t t1,
                                                uint32_t const* __restrict__ occ_slot, tables<K> TB,
                                                uint64_t const* __restrict__ occ, uint64_t R0, uint64_t nrec,
                                                uint64_t O0, uint64_t nblk, uint32_t const* __restrict__ blk_rec,
                                                unsigned long long const* base, unsigned long long* next,
                                                uint32_t* tile_counter, unsigned long long* status,
                                                uint2* __restrict__ fw, K* __restrict__ n_key,
                                                uint8_t* __restrict__ n_meta, uint32_t* __restrict__ n_rec,
                                                uint32_t* __restrict__ pnode, uint32_t* __restrict__ prec,
                                                uint32_t* err) {
    constexpr int NW = 256 / 32;
    constexpr int WORDS = NB_ROUNDS * NW;  // 32-occurrence words of a tile
    static_assert(WORDS == 64, "warp 0 scans two counts per lane");
    __shared__ uint64_t s_tile;
    __shared__ uint32_t wfirst[WORDS], wmulti[WORDS], wcnt[WORDS];
    __shared__ uint64_t s_node, s_pair;
    __shared__ tile_records<WORDS> win;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const uint64_t tile = s_tile;
    const uint64_t ntiles = (t1 - ta + WORDS * 32 - 1) / (WORDS * 32);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t tt = ta + tile * (WORDS * 32) + threadIdx.x;  // round rr: tt + 256 rr
    uint32_t sl[NB_ROUNDS];
#pragma unroll
    for (int rr = 0; rr < NB_ROUNDS; ++rr) {
        const uint64_t t = tt + 256u * rr;
        sl[rr] = t >= t0 && t < t1 ? __ldg(occ_slot + t) : NONE32;
    }
    K key[NB_ROUNDS];
    uint32_t rank[NB_ROUNDS], om[NB_ROUNDS];
#pragma unroll
    for (int rr = 0; rr < NB_ROUNDS; ++rr) {
        rank[rr] = NONE32;
        om[rr] = 0;
        if (sl[rr] != NONE32) slot_read(TB.slots + ((sl[rr] & 0x7fffffffu) - TB.off0), key[rr], rank[rr], om[rr]);
    }
    const uint32_t r0 = load_tile_records(win, occ, R0, nrec, O0, nblk, blk_rec,
                                          (ta + tile * (WORDS * 32)) / OCC_BLOCK);
    uint32_t first = 0, multi = 0;
#pragma unroll
    for (int rr = 0; rr < NB_ROUNDS; ++rr) {
        const bool f = rank[rr] == (uint32_t)(tt + 256u * rr);
        const bool m = (sl[rr] >> 31) && sl[rr] != NONE32 && (om[rr] & (M_PRIMARY | M_MULTI)) == (M_PRIMARY | M_MULTI);
        const uint32_t bf = __ballot_sync(0xffffffffu, f), bm = __ballot_sync(0xffffffffu, m);
        if (f) first |= 1u << rr;
        if (m) multi |= 1u << rr;
        if (lane == 0) {
            wfirst[rr * NW + warp] = bf;
            wmulti[rr * NW + warp] = bm;
            wcnt[rr * NW + warp] = __popc(bf) | (__popc(bm) << 16);
        }
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t c0 = wcnt[2 * lane], c1 = wcnt[2 * lane + 1];
        uint32_t x = c0 + c1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        const uint32_t tot = __shfl_sync(0xffffffffu, x, 31);
        const uint32_t ex = x - c0 - c1;
        wcnt[2 * lane] = ex;
        wcnt[2 * lane + 1] = ex + c0;
        uint64_t excl = 0;
        const uint64_t both = (uint64_t)(tot & 0xffffu) | ((uint64_t)(tot >> 16) << 31);
        const bool ok = prim::lookback_exclusive(status, tile, both, excl);
        if (lane == 0) {
            if (!ok) set_error(err, ERR_CHAIN_LIMIT);
            s_node = base[0] + (excl & 0x7fffffffu);
            s_pair = base[1] + (excl >> 31);
            if (tile == ntiles - 1) {
                next[0] = s_node + (tot & 0xffffu);
                next[1] = s_pair + (tot >> 16);
            }
        }
    }
    __syncthreads();
    const uint64_t node0 = s_node, pair0 = s_pair;
    if (threadIdx.x < WORDS) {
        const uint64_t w = ((ta + tile * (WORDS * 32)) >> 5) + threadIdx.x;
        if (w * 32 < t1) fw[w] = make_uint2(wfirst[threadIdx.x], (uint32_t)node0 + (wcnt[threadIdx.x] & 0xffffu));
    }
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int rr = 0; rr < NB_ROUNDS; ++rr) {
        const uint32_t i = rr * NW + warp;
        const bool f = (first >> rr) & 1u, m = (multi >> rr) & 1u;
        if (f) {
            const uint64_t n = node0 + (wcnt[i] & 0xffffu) + __popc(wfirst[i] & lt);
            n_key[n] = key[rr];
            n_meta[n] = (uint8_t)(om[rr] & 7u);
            uint32_t rec = NONE32;
            if (om[rr] & M_PRIMARY) rec = (om[rr] & M_MULTI) ? MULTI_TAG : (uint32_t)(R0 + (om[rr] >> 4) - 1);
            n_rec[n] = rec;
        }
        if (m) {
            const uint64_t at = pair0 + (wcnt[i] >> 16) + __popc(wmulti[i] & lt);
            pnode[at] = rank[rr];
            prec[at] = tile_record(win, r0, (int)i, (uint32_t)lane);
        }
    }
}

// Pairs [*pb, *pe) of one bucket group: first occurrences -> node indices.
__global__ void k_pair_nodes(unsigned long long const* pb, unsigned long long const* pe,
                             uint2 const* __restrict__ fw, uint32_t* __restrict__ pnode) {
    const uint64_t e = *pe;
    for (uint64_t i = *pb + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < e;
         i += (uint64_t)gridDim.x * blockDim.x)
        pnode[i] = node_of(fw, pnode[i]);
}

// Block-wide reservation of `want` consecutive entries of *cnt per thread,
// one atomic per block (a counter shared by millions of warps serializes
// their atomics).  Every thread of the block must call it.
template <int THREADS>
__device__ __forceinline__ unsigned long long block_reserve(uint32_t want, unsigned long long* cnt) {
    __shared__ unsigned long long s_warp[THREADS / 32];
    __shared__ unsigned long long s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long incl = want;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long run = 0;
        for (int w = 0; w < THREADS / 32; ++w) {
            const unsigned long long v = s_warp[w];
            s_warp[w] = run;
            run += v;
        }
        s_base = run ? atomicAdd(cnt, run) : 0ull;
    }
    __syncthreads();
    const unsigned long long r = s_base + s_warp[warp] + incl - want;
    __syncthreads();  // the shared words may be reused by the next call
    return r;
}

// Look-back state of one ordered selection (prim::ordered_select), zeroed.
struct select_ws {
    unsigned long long* status;
    unsigned long long* total;
    uint32_t* counter;
    uint64_t ntiles;
};

// Multi-record nodes from the (node, record) pairs in node order, in one pass:
// each pair once (a record may own a k-mer at two positions: equal pairs are
// neighbours) into urec, and the m-th node with its record range [moff[m],
// moff[m + 1]).
// Bound: latency of the pairs' loads, so every warp the SM holds (32 registers):
// 0.64 ms for the pairs of 200 genomes, 0.78 at 48 registers and 5 blocks per SM.
__global__ void __launch_bounds__(256, 8) k_multi_index(uint64_t n, uint32_t const* __restrict__ pn,
                                                     uint32_t const* __restrict__ pr, select_ws wk, select_ws wh,
                                                     uint32_t* __restrict__ urec, uint32_t* __restrict__ mnode,
                                                     uint64_t* __restrict__ moff, uint32_t* __restrict__ n_rec,
                                                     uint32_t* err) {
    __shared__ prim::ordered_select keep, head;
    const uint64_t tile = prim::select_tile(keep, wk.counter);
    uint32_t node[prim::SEL_ROUNDS], rec[prim::SEL_ROUNDS], sk = 0, sh = 0;
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t i = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        if (i >= n) continue;
        node[r] = pn[i];
        rec[r] = pr[i];
        const bool h = i == 0 || pn[i - 1] != node[r];
        if (h) sh |= 1u << r;
        if (h || pr[i - 1] != rec[r]) sk |= 1u << r;
    }
    prim::select_put(keep, sk);
    prim::select_put(head, sh);
    __syncthreads();
    if (threadIdx.x < 32)
        prim::select_scan(keep, tile, wk.ntiles, wk.status, wk.total, err);
    else if (threadIdx.x < 64)
        prim::select_scan(head, tile, wk.ntiles, wh.status, wh.total, err);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t i = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        const uint64_t o = prim::select_pos(keep, r), m = prim::select_pos(head, r);
        if ((sk >> r) & 1u) urec[o] = rec[r];
        if ((sh >> r) & 1u) {
            mnode[m] = node[r];
            moff[m] = o;
            n_rec[node[r]] = MULTI_TAG | (uint32_t)m;
        }
        if (i == n - 1) moff[m + ((sh >> r) & 1u)] = o + ((sk >> r) & 1u);
    }
}

// Multi-record nodes in node order whose owning-record list equals the
// previous one's (the k-mers of a stretch shared by the same records) share
// one union.  Bit m % 32 of same[m / 32]: node m's list is node m - 1's.  A lane
// compares lists of up to SHORT_LIST records itself, the warp the longer ones.
// A pass of its own, without order: repeats have stretches of k-mers in thousands
// of records, and a tile of those would hold up every later tile's look-back (300
// genomes with shared and tandem repeats, k = 63: 7.8 ms with the comparison inside
// k_multi_groups, 1.4 for the two).
constexpr uint64_t SHORT_LIST = 8;
__global__ void __launch_bounds__(256) k_multi_same(uint64_t M, uint64_t const* __restrict__ moff,
                                                    uint32_t const* __restrict__ urec, uint32_t* __restrict__ same) {
    const uint64_t m = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    const int lane = threadIdx.x & 31;
    if (m - lane >= M) return;
    uint64_t a0 = 0, a1 = 0;
    bool eq = false;
    if (m > 0 && m < M) {
        a0 = moff[m - 1];
        a1 = moff[m];
        eq = a1 - a0 == moff[m + 1] - a1;
    }
    const uint64_t n = a1 - a0;
    uint32_t todo = __ballot_sync(0xffffffffu, eq && n > SHORT_LIST);
    if (eq && n <= SHORT_LIST)
        for (uint64_t i = 0; i < n && eq; ++i) eq = urec[a0 + i] == urec[a1 + i];
    __syncwarp();
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const uint64_t x = __shfl_sync(0xffffffffu, a0, src), y = __shfl_sync(0xffffffffu, a1, src);
        bool bad = false;
        for (uint64_t base = 0; base < y - x && !bad; base += 128) {  // (the same trips for all lanes)
            bool b = false;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint64_t i = base + 32 * q + lane;
                b |= i < y - x && urec[x + i] != urec[y + i];
            }
            bad = __any_sync(0xffffffffu, b);
        }
        if (lane == src) eq = !bad;
    }
    const uint32_t w = __ballot_sync(0xffffffffu, eq);
    if (lane == 0) same[m >> 5] = w;
}

// Group g of the nodes above has its first node and its record range, every multi
// node its group.
__global__ void __launch_bounds__(256) k_multi_groups(uint64_t M, uint32_t const* __restrict__ same,
                                                      uint64_t const* __restrict__ moff,
                                                      uint32_t const* __restrict__ mnode, select_ws ws,
                                                      uint32_t* __restrict__ gnode, uint64_t* __restrict__ gbeg,
                                                      uint64_t* __restrict__ gend, uint32_t* __restrict__ mgrp,
                                                      uint32_t* err) {
    __shared__ prim::ordered_select head;
    const uint64_t tile = prim::select_tile(head, ws.counter);
    uint32_t sel = 0;
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t m = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        if (m < M && !((same[m >> 5] >> (m & 31)) & 1u)) sel |= 1u << r;
    }
    prim::select_rank(head, sel, tile, ws.ntiles, ws.status, ws.total, err);
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t m = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        if (m >= M) continue;
        const bool h = (sel >> r) & 1u;
        const uint64_t g = prim::select_pos(head, r) + (h ? 1 : 0) - 1;
        mgrp[m] = (uint32_t)g;
        if (h) {
            gnode[g] = mnode[m];
            gbeg[g] = moff[m];
            gend[g] = moff[m + 1];
        }
    }
}

// Warp-level helpers over a per-warp shared-memory bitmap of C bits.
__device__ __forceinline__ uint64_t warp_sum64(uint64_t v) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ uint32_t warp_excl_scan32(uint32_t v, uint32_t& total) {
    const int lane = threadIdx.x & 31;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    total = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
}

// OR the ascending list [c0, c1) of `list` into the shared bitmap `bm` of
// `nw` words (all 32 lanes call it).  A dense list (at least one element per
// 4 bit positions: 8 or more lanes per word) has the lanes holding the same
// word (consecutive lanes) combine their bits first, the first of them alone
// touching shared memory; a sparser one ORs lane by lane.  An unsorted list
// is ORed correctly either way.
__device__ __forceinline__ void warp_or_list(uint32_t* bm, uint32_t const* __restrict__ list, uint64_t c0,
                                             uint64_t c1, uint32_t nw, int lane) {
    if ((c1 - c0) * 4 < (uint64_t)nw * 32) {
        for (uint64_t c = c0 + lane; c < c1; c += 32) {
            const uint32_t v = list[c];
            atomicOr(&bm[v >> 5], 1u << (v & 31));
        }
        return;
    }
    for (uint64_t base = c0; base < c1; base += 32) {
        const bool in = base + lane < c1;
        const uint32_t v = in ? list[base + lane] : NONE32;
        const uint32_t w = v >> 5;
        uint32_t b = in ? 1u << (v & 31) : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t ob = __shfl_down_sync(0xffffffffu, b, o);
            const uint32_t ow = __shfl_down_sync(0xffffffffu, w, o);
            if (lane + o < 32 && ow == w) b |= ob;
        }
        const uint32_t pw = __shfl_up_sync(0xffffffffu, w, 1);
        if (in && (lane == 0 || pw != w)) atomicOr(&bm[w], b);
    }
}

// Union of the color lists of a multi-record node.  Pass 0: size and hash;
// pass 1: write the ascending list at pool[poff[m]].
template <bool WRITE>
__global__ void k_union(uint64_t M, uint64_t const* __restrict__ mbeg, uint64_t const* __restrict__ mend,
                        uint32_t const* __restrict__ urec,
                        uint64_t const* __restrict__ col_off, uint32_t const* __restrict__ colors,
                        uint32_t C, uint32_t* __restrict__ msize, uint64_t* __restrict__ mhash,
                        uint64_t const* __restrict__ poff, uint32_t* __restrict__ pool) {
    extern __shared__ uint32_t smem_bm[];
    const uint32_t nw = (C + 31) / 32;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    uint32_t* bm = smem_bm + (size_t)wib * nw;
    const uint64_t m = (uint64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    if (m >= M) return;
    for (uint32_t w = lane; w < nw; w += 32) bm[w] = 0;
    __syncwarp();
    for (uint64_t p = mbeg[m]; p < mend[m]; ++p) {
        const uint32_t r = urec[p];
        warp_or_list(bm, colors, col_off[r], col_off[r + 1], nw, lane);
    }
    __syncwarp();
    const uint32_t per = (nw + 31) / 32;
    const uint32_t w0 = lane * per, w1 = min(w0 + per, nw);
    uint32_t cnt = 0;
    uint64_t acc = 0;
    for (uint32_t w = w0; w < w1; ++w) {
        uint32_t x = bm[w];
        cnt += __popc(x);
        if (!WRITE && x) acc += word_mix(w, x);
    }
    uint32_t total;
    const uint32_t ex = warp_excl_scan32(cnt, total);
    if (!WRITE) {
        acc = warp_sum64(acc);
        if (lane == 0) {
            msize[m] = total;
            mhash[m] = set_hash_final(acc, total);
        }
    } else {
        uint32_t* out = pool + poff[m] + ex;
        for (uint32_t w = w0; w < w1; ++w) {
            uint32_t x = bm[w];
            while (x) {
                const uint32_t b = __ffs(x) - 1;
                x &= x - 1;
                *out++ = w * 32 + b;
            }
        }
    }
}

// ---- multi-record unions as bitmaps -----------------------------------------
// Records with at least `heavy` colors get a bitmap.
__global__ void k_heavy_flags(uint64_t nu, uint32_t const* __restrict__ urec, uint64_t const* __restrict__ col_off,
                              uint32_t R0, uint32_t heavy, uint32_t* __restrict__ flag) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nu) return;
    const uint32_t r = urec[i];
    if (col_off[r + 1] - col_off[r] >= heavy) flag[r - R0] = 1u;
}

// Heavy records' colors as bitmaps in rbits[hpos[r - R0] * nw].
__global__ void k_heavy_bitmaps(uint64_t nrec, uint32_t const* __restrict__ flag, uint64_t const* __restrict__ hpos,
                                uint32_t R0, uint64_t const* __restrict__ col_off, uint32_t const* __restrict__ colors,
                                uint32_t nw, uint32_t* __restrict__ rbits) {
    extern __shared__ uint32_t smem_bm[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    uint32_t* bm = smem_bm + (size_t)wib * nw;
    // 32 records per warp: the lanes read the flags at once (few records are
    // heavy), then the warp builds each heavy record's bitmap
    const uint64_t i0 = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + wib) * 32;
    if (i0 >= nrec) return;
    uint32_t fm = __ballot_sync(0xffffffffu, i0 + lane < nrec && flag[i0 + lane]);
    while (fm) {
        const uint64_t i = i0 + (uint32_t)(__ffs(fm) - 1);
        fm &= fm - 1;
        for (uint32_t w = lane; w < nw; w += 32) bm[w] = 0;
        __syncwarp();
        warp_or_list(bm, colors, col_off[R0 + i], col_off[R0 + i + 1], nw, lane);
        __syncwarp();
        uint32_t* out = rbits + hpos[i] * (uint64_t)nw;
        for (uint32_t w = lane; w < nw; w += 32) out[w] = bm[w];
        __syncwarp();
    }
}

// A group of GW lanes per union: OR of its records' color sets (bitmap words for
// heavy records, per-color bits for the rest) -> mbits, size, set hash.
// The records' metadata is fetched GW at a time, one record per lane; heavy
// records' bitmap words are ORed into registers (lane owns words lane + GW u,
// u < WPL), four records' lines in flight at a time; the rest have their
// colors spread over the lanes and set bits in the group's shared bitmap.
// Groups of a warp go through the loops together, and a union of more than
// 4 GW records has its remaining ones spread over the whole warp (90 genomes
// in skewed buckets: 3.1 ms, 4.3 with a group alone on its union).
// Bound: issue, at 32 registers so that all warps fit (40: 1.5 ms).  200
// genomes, 7 words, a handful of records per union: whole warps 2.9 ms, groups
// of 16 2.3, of 8 1.25.
template <int WPL, int GW>
__global__ void __launch_bounds__(256, WPL == 1 ? 8 : 1) k_union_bm(
    uint64_t M, uint64_t const* __restrict__ mbeg, uint64_t const* __restrict__ mend,
    uint32_t const* __restrict__ urec, uint64_t const* __restrict__ col_off, uint32_t const* __restrict__ colors,
    uint32_t R0, uint32_t const* __restrict__ hflag, uint64_t const* __restrict__ hpos,
    uint32_t const* __restrict__ rbits, uint32_t nw, uint32_t* __restrict__ mbits, uint32_t* __restrict__ msize,
    uint64_t* __restrict__ mhash) {
    extern __shared__ uint32_t smem_bm[];
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr uint32_t GMASK = GW == 32 ? FULL : (1u << (GW & 31)) - 1u;
    const int lane = threadIdx.x & 31, gl = lane & (GW - 1), gs = lane & ~(GW - 1);
    const uint32_t grp = threadIdx.x / GW;
    uint32_t* bm = smem_bm + (size_t)grp * nw;
    const uint64_t m = (uint64_t)blockIdx.x * (blockDim.x / GW) + grp;
    if (__all_sync(FULL, m >= M)) return;
    const bool on = m < M;
    for (uint32_t w = gl; w < nw; w += GW) bm[w] = 0;
    __syncwarp();
    uint32_t acc[WPL];
#pragma unroll
    for (int u = 0; u < WPL; ++u) acc[u] = 0;
    // [p0, pend): the records a group goes through, GW of them every `stride`,
    // into its registers and the bitmap `to`: first its own union's, then, one
    // long union of the warp after another, its share of that one's rest
    const uint64_t pe = on ? mend[m] : 0;
    uint64_t p0 = on ? mbeg[m] : 0, pend = pe, rest = pe;
    uint32_t stride = GW, longs = 0;
    uint32_t* to = bm;
    if constexpr (GW < 32) {
        if (p0 + 4 * GW < pe) rest = pend = p0 + 4 * GW;
        longs = __ballot_sync(FULL, gl == 0 && rest < pe);
    }
    int own = gs;          // the first lane of the group whose union the records belong to
    uint32_t keep[WPL];    // the words of a group's own union while it helps another's
    for (;;) {
        for (; __any_sync(FULL, p0 < pend); p0 += stride) {
            const uint64_t p = p0 + gl;
            bool heavy = false, light = false;
            uint64_t src = 0, c0 = 0, c1 = 0;
            if (p < pend) {
                const uint32_t r = urec[p];
                heavy = hflag && hflag[r - R0] != 0;
                light = !heavy;
                if (heavy) {
                    src = hpos[r - R0] * (uint64_t)nw;
                } else {
                    c0 = col_off[r];
                    c1 = col_off[r + 1];
                }
            }
            uint32_t hm = (__ballot_sync(FULL, heavy) >> gs) & GMASK;
            while (__any_sync(FULL, hm != 0)) {
                // four records' lines in flight (a record repeats when fewer remain)
                const bool any = hm != 0;
                int q[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    q[j] = hm ? __ffs(hm) - 1 : j ? q[0] : 0;
                    if (hm) hm &= hm - 1;
                }
                uint64_t s[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) s[j] = __shfl_sync(FULL, src, q[j], GW);
#pragma unroll
                for (int u = 0; u < WPL; ++u) {
                    const uint32_t w = gl + GW * u;
                    if (any && w < nw) acc[u] |= rbits[s[0] + w] | rbits[s[1] + w] | rbits[s[2] + w] | rbits[s[3] + w];
                }
            }
            // light records: their colors laid end to end over the group, GW at a
            // time (a lane finds its record by a search over the length prefix)
            const uint32_t len = light ? (uint32_t)(c1 - c0) : 0u;  // < 8192 colors in bitmap mode
            uint32_t incl = len;
#pragma unroll
            for (int o = 1; o < GW; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, incl, o, GW);
                if (gl >= o) incl += y;
            }
            const uint32_t excl = incl - len;
            const uint32_t total = __shfl_sync(FULL, incl, GW - 1, GW);
            for (uint32_t e0 = 0; __any_sync(FULL, e0 < total); e0 += GW) {
                const uint32_t e = e0 + gl;
                int q = 0;  // the last lane whose range starts at or before e
#pragma unroll
                for (int step = GW / 2; step; step >>= 1) {
                    const uint32_t ex = __shfl_sync(FULL, excl, (q + step) & (GW - 1), GW);
                    if (q + step < GW && ex <= e) q += step;
                }
                const uint64_t cq = __shfl_sync(FULL, c0, q, GW);
                const uint32_t xq = __shfl_sync(FULL, excl, q, GW);
                if (e < total) {
                    const uint32_t v = colors[cq + (e - xq)];
                    atomicOr(&to[v >> 5], 1u << (v & 31));
                }
            }
        }
        if constexpr (GW == 32) {
            break;
        } else {
            if (stride == 32) {
#pragma unroll
                for (int u = 0; u < WPL; ++u) {
#pragma unroll
                    for (int o = GW; o < 32; o <<= 1) acc[u] |= __shfl_xor_sync(FULL, acc[u], o);
                    if (gs != own) acc[u] = keep[u];
                }
            }
            if (!longs) break;
            own = __ffs(longs) - 1;
            longs &= longs - 1;
            stride = 32;
            p0 = __shfl_sync(FULL, rest, own) + gs;
            pend = __shfl_sync(FULL, pe, own);
            to = smem_bm + (size_t)((threadIdx.x - lane + own) / GW) * nw;
#pragma unroll
            for (int u = 0; u < WPL; ++u) {
                keep[u] = acc[u];
                if (gs != own) acc[u] = 0;
            }
        }
    }
    __syncwarp();
    uint32_t cnt = 0;
    uint64_t hs = 0;
    uint32_t* out = mbits + m * (uint64_t)nw;
#pragma unroll
    for (int u = 0; u < WPL; ++u) {
        const uint32_t w = gl + GW * u;
        if (on && w < nw) {
            const uint32_t x = bm[w] | acc[u];
            out[w] = x;
            cnt += __popc(x);
            if (x) hs += word_mix(w, x);
        }
    }
#pragma unroll
    for (int o = GW / 2; o; o >>= 1) {
        cnt += __shfl_xor_sync(FULL, cnt, o, GW);
        hs += __shfl_xor_sync(FULL, hs, o, GW);
    }
    if (on && gl == 0) {
        msize[m] = cnt;
        mhash[m] = set_hash_final(hs, cnt);
    }
}

// Four consecutive nodes' words from n0 (a multiple of 4; n_rec starts on 16
// bytes); NONE32 past D.
__device__ __forceinline__ void load_nodes4(uint32_t const* __restrict__ w, uint64_t n0, uint64_t D, uint32_t (&r)[4]) {
    if (n0 + 4 <= D) {
        const uint4 v = *reinterpret_cast<uint4 const*>(w + n0);
        r[0] = v.x;
        r[1] = v.y;
        r[2] = v.z;
        r[3] = v.w;
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = n0 + j < D ? w[n0 + j] : NONE32;
    }
}

// rec_first[r] = smallest node index whose color set is record r's list.
// Neighbouring nodes mostly come from one record, so a thread takes four and
// only the first of consecutive nodes with the same record sends a minimum
// (200 genomes: 1.0 ms with one for every node, 0.26 so).
__global__ void __launch_bounds__(256) k_rec_first(uint64_t D, uint32_t const* __restrict__ n_rec, uint32_t R0,
                                                   uint32_t* __restrict__ rec_first) {
    const uint64_t n0 = 4 * ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x);
    uint32_t r[4];
    load_nodes4(n_rec, n0, D, r);
    uint32_t prev = __shfl_up_sync(0xffffffffu, r[3], 1);
    if ((threadIdx.x & 31) == 0) prev = NONE32;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (r[j] != NONE32 && !(r[j] & MULTI_TAG) && r[j] != prev) atomicMin(&rec_first[r[j] - R0], (uint32_t)(n0 + j));
        prev = r[j];
    }
}

// Candidate class sources: used records then multi nodes.
struct cand_view {
    uint32_t* kind_id;   // record id (global) or MULTI_TAG | m
    uint32_t* first;     // node of first appearance
    uint64_t* hash;
};

// Records that are some k-mer's color set (rec_first set), in record order.
__global__ void __launch_bounds__(256) k_cand_records(uint64_t nrec, uint32_t R0,
                                                      uint32_t const* __restrict__ rec_first, select_ws ws,
                                                      uint64_t const* __restrict__ rhash, cand_view cv,
                                                      uint32_t* __restrict__ rec_cand, uint32_t* err) {
    __shared__ prim::ordered_select used;
    const uint64_t tile = prim::select_tile(used, ws.counter);
    uint32_t first[prim::SEL_ROUNDS], sel = 0;
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t i = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        first[r] = i < nrec ? rec_first[i] : NONE32;
        if (first[r] != NONE32) sel |= 1u << r;
    }
    prim::select_rank(used, sel, tile, ws.ntiles, ws.status, ws.total, err);
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        if (!((sel >> r) & 1u)) continue;
        const uint64_t i = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        const uint64_t c = prim::select_pos(used, r);
        cv.kind_id[c] = R0 + (uint32_t)i;
        cv.first[c] = first[r];
        cv.hash[c] = rhash[R0 + i];
        rec_cand[i] = (uint32_t)c;
    }
}

__global__ void k_cand_multi(uint64_t M, uint64_t base, uint32_t const* __restrict__ mnode,
                             uint64_t const* __restrict__ mhash, cand_view cv) {
    uint64_t m = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    cv.kind_id[base + m] = MULTI_TAG | (uint32_t)m;
    cv.first[base + m] = mnode[m];
    cv.hash[base + m] = mhash[m];
}

struct list_src {
    uint64_t const* col_off;
    uint32_t const* colors;
    uint64_t const* poff;   // list mode: multi-node unions as ascending lists
    uint32_t const* pool;
    uint32_t const* msize;
    uint32_t const* mbits;  // bitmap mode: multi-node unions as C-bit bitmaps
    uint32_t nw;            // 32-bit words per bitmap
};
__device__ __forceinline__ void cand_list(list_src const& L, uint32_t kind_id, uint32_t const*& p, uint64_t& n) {
    if (kind_id & MULTI_TAG) {
        const uint32_t m = kind_id & ~MULTI_TAG;
        p = L.pool ? L.pool + L.poff[m] : nullptr;
        n = L.msize[m];
    } else {
        p = L.colors + L.col_off[kind_id];
        n = L.col_off[kind_id + 1] - L.col_off[kind_id];
    }
}

// A candidate color set: an ascending list, or a bitmap (multi-node unions
// in bitmap mode), with its size.
struct cand_set {
    uint32_t const* list;
    uint32_t const* bm;
    uint64_t n;
};
__device__ __forceinline__ cand_set cand_get(list_src const& L, uint32_t kind_id) {
    cand_set c;
    c.bm = nullptr;
    if ((kind_id & MULTI_TAG) && L.mbits) {
        const uint32_t m = kind_id & ~MULTI_TAG;
        c.list = nullptr;
        c.bm = L.mbits + (uint64_t)m * L.nw;
        c.n = L.msize[m];
        return c;
    }
    cand_list(L, kind_id, c.list, c.n);
    return c;
}
__device__ __forceinline__ cand_set shfl_set(cand_set const& s, int src) {
    cand_set r;
    r.list = (uint32_t const*)__shfl_sync(0xffffffffu, (unsigned long long)s.list, src);
    r.bm = (uint32_t const*)__shfl_sync(0xffffffffu, (unsigned long long)s.bm, src);
    r.n = __shfl_sync(0xffffffffu, (unsigned long long)s.n, src);
    return r;
}

__device__ __forceinline__ bool sets_equal(cand_set const& a, cand_set const& b, uint32_t nw) {
    if (a.n != b.n) return false;
    if (a.bm && b.bm) {
        for (uint32_t w = 0; w < nw; ++w)
            if (a.bm[w] != b.bm[w]) return false;
        return true;
    }
    if (!a.bm && !b.bm) {
        for (uint64_t i = 0; i < a.n; ++i)
            if (a.list[i] != b.list[i]) return false;
        return true;
    }
    // list against bitmap of the same size: equal iff every element is set
    const cand_set& l = a.bm ? b : a;
    const cand_set& m = a.bm ? a : b;
    for (uint64_t i = 0; i < l.n; ++i) {
        const uint32_t v = l.list[i];
        if (!((m.bm[v >> 5] >> (v & 31)) & 1u)) return false;
    }
    return true;
}

// ---- bit ranges -------------------------------------------------------------
__device__ __forceinline__ uint64_t bits_at(uint64_t const* w, uint64_t pos) {
    const uint64_t i = pos >> 6;
    const uint32_t s = (uint32_t)(pos & 63);
    uint64_t v = w[i] >> s;
    if (s) v |= w[i + 1] << (64 - s);
    return v;
}
// Equal bit strings [pa, pa + la) of wa and [pb, pb + lb) of wb.  The hybrid
// encoding is canonical, so equal encodings <=> equal color sets.
__device__ __forceinline__ bool bits_equal(uint64_t const* wa, uint64_t pa, uint64_t la, uint64_t const* wb,
                                           uint64_t pb, uint64_t lb) {
    if (la != lb) return false;
    for (uint64_t i = 0; i < la; i += 64) {
        uint64_t x = bits_at(wa, pa + i) ^ bits_at(wb, pb + i);
        const uint64_t n = la - i;
        if (n < 64) x &= (1ull << n) - 1;
        if (x) return false;
    }
    return true;
}

// ---- hybrid encoding (hybrid_color_sets.hpp:48-95) with the delta code of
// this project's `bits` stand-in: delta(x) = Elias delta of x + 1, LSB-first.
__device__ __forceinline__ uint32_t msb64(uint64_t y) { return 63u - (uint32_t)__clzll((long long)y); }
__device__ __forceinline__ uint32_t delta_bits(uint64_t x) {
    const uint64_t y = x + 1;
    const uint32_t l = msb64(y);
    const uint32_t ll = msb64(l + 1);
    return 2 * ll + 1 + l;
}
__device__ __forceinline__ void or_bits(uint64_t* w, uint64_t pos, uint64_t val, uint32_t len) {
    if (len == 0) return;
    if (len < 64) val &= (1ull << len) - 1;
    const uint64_t i = pos >> 6;
    const uint32_t s = (uint32_t)(pos & 63);
    atomicOr((unsigned long long*)&w[i], (unsigned long long)(val << s));
    if (s && s + len > 64) atomicOr((unsigned long long*)&w[i + 1], (unsigned long long)(val >> (64 - s)));
}
// Delta code of x < 2^32: its bits (at most 43), `len` of them.
__device__ __forceinline__ uint64_t delta_code(uint64_t x, uint32_t& len) {
    const uint64_t y = x + 1;
    const uint32_t l = msb64(y);
    const uint32_t L1 = l + 1, ll = msb64(L1);
    // gamma(L1): ll zeros, a one, the low ll bits of L1; then the low l bits of y
    const uint64_t g = (1ull << ll) | ((uint64_t)(L1 & ((1u << ll) - 1u)) << (ll + 1));
    len = 2 * ll + 1 + l;
    return g | ((y & ((1ull << l) - 1)) << (2 * ll + 1));
}
__device__ __forceinline__ uint64_t put_delta(uint64_t* w, uint64_t pos, uint64_t x) {
    uint32_t len;
    const uint64_t c = delta_code(x, len);
    or_bits(w, pos, c, len);
    return pos + len;
}
// Codes one after another from bit `pos` on, stored a word at a time: the words
// in between are this writer's alone, the first and last are shared.
struct code_writer {
    uint64_t* w;
    uint64_t acc;
    uint32_t fill;
    bool shared;  // the current word holds others' bits
    __device__ __forceinline__ code_writer(uint64_t* words, uint64_t pos)
        : w(words + (pos >> 6)), acc(0), fill((uint32_t)(pos & 63)), shared(true) {}
    __device__ __forceinline__ void put(uint64_t c, uint32_t len) {
        acc |= c << fill;
        if (fill + len >= 64) {
            if (shared)
                atomicOr((unsigned long long*)w, (unsigned long long)acc);
            else
                *w = acc;
            ++w;
            shared = false;
            acc = fill ? c >> (64 - fill) : 0;
            fill = fill + len - 64;
        } else {
            fill += len;
        }
    }
    __device__ __forceinline__ void end() {
        if (acc) atomicOr((unsigned long long*)w, (unsigned long long)acc);
    }
};

// One candidate class by a group of GW consecutive lanes (a power of two; gl: the
// lane in the group; bm: the group's C-bit shared bitmap).  Groups of a warp run
// together, a group without a candidate with an empty set.  Pass 0 (ENC =
// false): encoded size -> nbits[j].  Pass 1: write at bit offset pos0 of `words`
// (zeroed).
template <int GW, typename T>
__device__ __forceinline__ T group_excl_scan(T v, T& total) {
    const int gl = threadIdx.x & (GW - 1);
    T x = v;
#pragma unroll
    for (int o = 1; o < GW; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, x, o, GW);
        if (gl >= o) x += y;
    }
    total = __shfl_sync(0xffffffffu, x, GW - 1, GW);
    return x - v;
}
template <bool ENC, int GW>
__device__ __forceinline__ void encode_one(cand_set const& cs, bool on, uint64_t j, uint64_t pos0, uint32_t C,
                                           uint32_t nw, uint32_t* bm, uint64_t* __restrict__ nbits,
                                           uint64_t* __restrict__ words) {
    const int gl = threadIdx.x & (GW - 1);
    const uint64_t N = on ? cs.n : 0;
    const uint64_t sparse_t = (uint64_t)(0.25 * (double)C);
    const uint64_t dense_t = (uint64_t)(0.75 * (double)C);
    const uint32_t hdr = delta_bits(N);
    const bool plain = N >= sparse_t && N < dense_t;       // a C-bit bitmap
    const bool gaps = !plain && cs.list && N < sparse_t;   // gap codes straight from the ascending list
    const bool walk = on && !plain && !gaps;               // gap codes of the bitmap or its complement
    if (ENC && on && gl == 0) put_delta(words, pos0, N);
    // gap codes from the list, GW at a time
    {
        uint64_t acc = 0, p = pos0 + hdr;
        const uint64_t n = on && gaps ? N : 0;
        for (uint64_t base = 0; __any_sync(0xffffffffu, base < n); base += GW) {
            const uint64_t i = base + gl;
            const uint32_t v = i < n ? cs.list[i] : 0u;
            uint32_t pv = __shfl_up_sync(0xffffffffu, v, 1, GW);
            if (gl == 0 && base && base < n) pv = cs.list[base - 1];
            const uint64_t gap = i == 0 ? (uint64_t)v : (uint64_t)(v - pv - 1);
            if (ENC) {
                uint32_t len = 0, total;
                const uint64_t c = i < n ? delta_code(gap, len) : 0;
                const uint32_t ex = group_excl_scan<GW>(len, total);
                if (i < n) or_bits(words, p + ex, c, len);
                p += total;
            } else if (i < n) {
                acc += delta_bits(gap);
            }
        }
        if (!ENC && on && gaps) {
            // (only this group's lanes are here: its own mask)
            const uint32_t gm = GW == 32 ? 0xffffffffu : ((1u << GW) - 1u) << ((threadIdx.x & 31) & ~(GW - 1));
#pragma unroll
            for (int o = GW / 2; o; o >>= 1) acc += __shfl_xor_sync(gm, acc, o, GW);
            if (gl == 0) nbits[j] = hdr + acc;
        }
    }
    if (!ENC && on && plain && gl == 0) nbits[j] = hdr + C;
    // the others through the bitmap
    const bool need_bm = walk || (ENC && on && plain);
    if (!__any_sync(0xffffffffu, need_bm)) return;
    if (need_bm)
        for (uint32_t w = gl; w < nw; w += GW) bm[w] = cs.bm ? cs.bm[w] : 0u;
    __syncwarp();
    if (need_bm && !cs.bm)
        for (uint64_t c = gl; c < N; c += GW) {
            const uint32_t v = cs.list[c];
            atomicOr(&bm[v >> 5], 1u << (v & 31));
        }
    __syncwarp();
    if (ENC && on && plain)
        for (uint32_t w = gl; w < nw; w += GW)
            or_bits(words, pos0 + hdr + (uint64_t)w * 32, bm[w], min(32u, C - w * 32));
    const bool want_ones = N < sparse_t;  // else complement: values not in the set
    const uint32_t per = (nw + GW - 1) / GW;
    const uint32_t w0 = walk ? gl * per : 0u, w1 = walk ? min(w0 + per, nw) : 0u;
    auto word_bits = [&](uint32_t w) -> uint32_t {
        uint32_t x = want_ones ? bm[w] : ~bm[w];
        const uint32_t valid = C - w * 32;
        if (valid < 32) x &= (1u << valid) - 1u;
        return x;
    };
    int32_t last = -1;
    for (uint32_t w = w0; w < w1; ++w) {
        const uint32_t x = word_bits(w);
        if (x) last = (int32_t)(w * 32 + 31 - __clz(x));
    }
    // previous element before this lane's range = max of `last` over lower lanes
    int32_t prev;
    {
        int32_t x = last;
#pragma unroll
        for (int o = 1; o < GW; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, x, o, GW);
            if (gl >= o) x = max(x, y);
        }
        prev = __shfl_up_sync(0xffffffffu, x, 1, GW);
        if (gl == 0) prev = -1;
    }
    uint64_t mybits = 0;
    {
        int32_t pv = prev;
        for (uint32_t w = w0; w < w1; ++w) {
            uint32_t x = word_bits(w);
            while (x) {
                const uint32_t b = __ffs(x) - 1;
                x &= x - 1;
                const int32_t v = (int32_t)(w * 32 + b);
                mybits += delta_bits(pv < 0 ? (uint64_t)v : (uint64_t)(v - pv - 1));
                pv = v;
            }
        }
    }
    uint64_t total;
    const uint64_t ex = group_excl_scan<GW>(mybits, total);
    if (!ENC) {
        if (walk && gl == 0) nbits[j] = hdr + total;
        return;
    }
    code_writer out(words, pos0 + hdr + ex);
    int32_t pv = prev;
    for (uint32_t w = w0; w < w1; ++w) {
        uint32_t x = word_bits(w);
        while (x) {
            const uint32_t b = __ffs(x) - 1;
            x &= x - 1;
            const int32_t v = (int32_t)(w * 32 + b);
            uint32_t len;
            const uint64_t c = delta_code(pv < 0 ? (uint64_t)v : (uint64_t)(v - pv - 1), len);
            out.put(c, len);
            pv = v;
        }
    }
    out.end();
}

// Warp per 32 candidate classes (class j = candidate order[j], or j): the lanes
// fetch the 32 candidates' sets (and pass-1 offsets) at once, then groups of GW lanes encode one each, 32 / GW
// at a time, so the dependent metadata loads are paid once per 32 candidates and a
// set of few words does not leave most of a warp idle.
// Bound: latency of the list and bitmap reads, then the bit ORs.  200 genomes (7
// bitmap words, 4.9e6 classes): whole warps 5.1 ms, groups of 8 1.8 ms;
// the first batch's classes are encoded where they stay (appending them took 0.5 ms
// more a batch).
template <bool ENC, int GW>
__global__ void k_encode(uint64_t nc, uint32_t const* __restrict__ order, cand_view cv, list_src L, uint32_t C,
                         uint64_t* __restrict__ nbits, uint64_t const* __restrict__ boff,
                         uint64_t* __restrict__ words) {
    extern __shared__ uint32_t smem_bm[];
    const uint32_t nw = (C + 31) / 32;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, grp = lane / GW;
    constexpr int GROUPS = 32 / GW;
    uint32_t* bm = smem_bm + ((size_t)wib * GROUPS + grp) * nw;
    const uint64_t j0 = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + wib) * 32;
    if (j0 >= nc) return;
    const uint64_t jl = j0 + lane;
    cand_set mine{nullptr, nullptr, 0};
    uint64_t pos = 0;
    if (jl < nc) {
        mine = cand_get(L, cv.kind_id[order ? order[jl] : jl]);
        if (ENC) pos = boff[jl];
    }
    const uint32_t cnt = nc - j0 < 32 ? (uint32_t)(nc - j0) : 32u;
    for (uint32_t q0 = 0; q0 < cnt; q0 += GROUPS) {
        const uint32_t q = q0 + grp;
        const cand_set cs = shfl_set(mine, (int)(q & 31));
        const uint64_t p = __shfl_sync(0xffffffffu, pos, (int)(q & 31));
        encode_one<ENC, GW>(cs, q < cnt, j0 + q, p, C, nw, bm, nbits, words);
        __syncwarp();  // the next candidates reuse the bitmaps
    }
}

// Global class dictionary as seen by kernels: hash slots -> class id, and the
// classes' encodings (bit_off has n + 1 entries).
struct dict_view {
    uint64_t const* slot_hash;
    uint32_t const* slot_cid;
    uint64_t mask;
    uint64_t const* bit_off;
    uint64_t const* words;
};

// Candidate encodings: cw words, cb[c] .. cb[c + 1] bit range of candidate c.
__global__ void k_dict_lookup(uint64_t nc, cand_view cv, uint64_t const* __restrict__ cw,
                              uint64_t const* __restrict__ cb, dict_view D, uint32_t* __restrict__ cid) {
    uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const uint64_t h = cv.hash[c];
    uint32_t res = NONE32;
    if (D.slot_hash) {
        uint64_t s = h & D.mask;
        for (uint64_t i = 0; i <= D.mask; ++i) {
            const uint64_t sh = D.slot_hash[s];
            if (sh == HASH_EMPTY) break;
            if (sh == h) {
                const uint32_t k = D.slot_cid[s];
                if (bits_equal(cw, cb[c], cb[c + 1] - cb[c], D.words, D.bit_off[k], D.bit_off[k + 1] - D.bit_off[k])) {
                    res = k;
                    break;
                }
            }
            s = (s + 1) & D.mask;
        }
    }
    cid[c] = res;
}

// Runs of equal hashes in the sorted candidates: run[i] of every position, the
// runs' starts, and rep_first set to none for every candidate.
__global__ void __launch_bounds__(256) k_hash_runs(uint64_t n, uint64_t const* __restrict__ key, select_ws ws,
                                                   uint32_t* __restrict__ run, uint32_t* __restrict__ run_start,
                                                   uint32_t* __restrict__ rep_first, uint32_t* err) {
    __shared__ prim::ordered_select head;
    const uint64_t tile = prim::select_tile(head, ws.counter);
    uint32_t sel = 0;
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t i = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        if (i < n && (i == 0 || key[i] != key[i - 1])) sel |= 1u << r;
    }
    prim::select_rank(head, sel, tile, ws.ntiles, ws.status, ws.total, err);
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t i = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        if (i >= n) continue;
        const bool h = (sel >> r) & 1u;
        const uint32_t q = (uint32_t)(prim::select_pos(head, r) + (h ? 1 : 0) - 1);
        run[i] = q;
        if (h) run_start[q] = (uint32_t)i;
        rep_first[i] = NONE32;
    }
}

// Set comparison split by length.  A set of at most SHORT_SET words is
// compared by its own lane, eight loads in flight at a time; a longer one by
// the whole warp, lanes reading consecutive words (one coalesced line per
// list per 32 words, four lines in flight per round).
constexpr uint64_t SHORT_SET = 32;

__device__ __forceinline__ uint64_t set_words(cand_set const& a, cand_set const& b, uint32_t nw) {
    return (a.bm && b.bm) ? nw : a.n;
}

// Lane-local equality of two sets of equal size.
__device__ __forceinline__ bool lane_sets_equal(cand_set const& a, cand_set const& b, uint32_t nw) {
    const bool ba = a.bm != nullptr, bb = b.bm != nullptr;
    if (ba == bb) {
        uint32_t const* x = ba ? a.bm : a.list;
        uint32_t const* y = ba ? b.bm : b.list;
        const uint64_t len = ba ? nw : a.n;
        for (uint64_t base = 0; base < len; base += 8) {
            uint32_t u[8], v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const bool in = base + q < len;
                u[q] = in ? x[base + q] : 0u;
                v[q] = in ? y[base + q] : 0u;
            }
            bool bad = false;
#pragma unroll
            for (int q = 0; q < 8; ++q) bad |= u[q] != v[q];
            if (bad) return false;
        }
        return true;
    }
    // list against bitmap of the same size: equal iff every element is set
    const cand_set& l = ba ? b : a;
    const cand_set& m = ba ? a : b;
    for (uint64_t base = 0; base < l.n; base += 8) {
        uint32_t u[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) u[q] = base + q < l.n ? l.list[base + q] : NONE32;
        bool bad = false;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (u[q] != NONE32) bad |= !((m.bm[u[q] >> 5] >> (u[q] & 31)) & 1u);
        if (bad) return false;
    }
    return true;
}

// Warp-wide equality of two sets of equal size (all 32 lanes call it with the
// same arguments).
__device__ __forceinline__ bool warp_sets_equal(cand_set const& a, cand_set const& b, uint32_t nw, int lane) {
    const bool ba = a.bm != nullptr, bb = b.bm != nullptr;
    if (ba == bb) {
        uint32_t const* x = ba ? a.bm : a.list;
        uint32_t const* y = ba ? b.bm : b.list;
        const uint64_t len = ba ? nw : a.n;
        for (uint64_t base = 0; base < len; base += 128) {
            uint32_t u[4], v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint64_t j = base + 32 * q + lane;
                u[q] = j < len ? x[j] : 0u;
                v[q] = j < len ? y[j] : 0u;
            }
            bool bad = false;
#pragma unroll
            for (int q = 0; q < 4; ++q) bad |= u[q] != v[q];
            if (__any_sync(0xffffffffu, bad)) return false;
        }
        return true;
    }
    const cand_set& l = ba ? b : a;
    const cand_set& m = ba ? a : b;
    for (uint64_t base = 0; base < l.n; base += 128) {
        uint32_t u[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t j = base + 32 * q + lane;
            u[q] = j < l.n ? l.list[j] : NONE32;
        }
        bool bad = false;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (u[q] != NONE32) bad |= !((m.bm[u[q] >> 5] >> (u[q] & 31)) & 1u);
        if (__any_sync(0xffffffffu, bad)) return false;
    }
    return true;
}

// Members of an equal-hash run of candidates against the run head, on the
// raw ascending color lists (or bitmaps); rep[c] = head when equal, a
// differing member marks its run for the exact fallback.  Each lane fetches
// its own pair of sets; short pairs are compared by the lane, long ones by
// the warp in turn.  The grid covers n in whole blocks of 256 threads.
__global__ void __launch_bounds__(256) k_member_match_raw(
    uint64_t n, uint32_t const* __restrict__ run_of, uint32_t const* __restrict__ run_start,
    uint32_t const* __restrict__ nidx, cand_view cv, list_src L, uint32_t* __restrict__ rep,
    uint32_t* __restrict__ rep_first, uint32_t* __restrict__ collided, uint32_t* __restrict__ any) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int need = 0;  // 0: decided, 1: lane compares, 2: warp compares
    bool eq = false;
    uint64_t run = 0;
    uint32_t c = 0, h = 0;
    cand_set sc{nullptr, nullptr, 0}, sh{nullptr, nullptr, 0};
    if (i < n) {
        run = run_of[i];
        c = nidx[i];
        h = nidx[run_start[run]];
        if (c == h) {
            rep[c] = c;
        } else {
            sc = cand_get(L, cv.kind_id[c]);
            sh = cand_get(L, cv.kind_id[h]);
            need = sc.n != sh.n ? 3 : (set_words(sc, sh, L.nw) <= SHORT_SET ? 1 : 2);
        }
    }
    if (need == 1) eq = lane_sets_equal(sc, sh, L.nw);
    uint32_t todo = __ballot_sync(0xffffffffu, need == 2);
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const bool e = warp_sets_equal(shfl_set(sc, src), shfl_set(sh, src), L.nw, lane);
        if (lane == src) eq = e;
    }
    if (need) {
        if (eq) {
            rep[c] = h;
        } else {
            rep[c] = c;
            collided[run] = 1;
            *any = 1;
        }
    }
    // rep_first[h] = min first appearance over the head and its equal
    // members.  A run's positions are consecutive, so the warp takes the
    // minimum per run first and one lane per run issues the atomic: a run of
    // millions of equal sets would otherwise serialize on one address.
    uint32_t f = (i < n && (c == h || eq)) ? cv.first[c] : NONE32;
    const uint64_t key = i < n ? run : ~0ull;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t of = __shfl_down_sync(0xffffffffu, f, o);
        const uint64_t ok = __shfl_down_sync(0xffffffffu, key, o);
        if (lane + o < 32 && ok == key) f = min(f, of);
    }
    const uint64_t pk = __shfl_up_sync(0xffffffffu, key, 1);
    if (i < n && (lane == 0 || pk != key) && f != NONE32) atomicMin(&rep_first[h], f);
}

__global__ void k_group_collided_raw(uint64_t nruns, uint32_t const* __restrict__ collided,
                                     uint32_t const* __restrict__ run_start, uint64_t n,
                                     uint32_t const* __restrict__ nidx, cand_view cv, list_src L,
                                     uint32_t* __restrict__ rep, uint32_t* __restrict__ rep_first) {
    uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nruns || !collided[r]) return;
    const uint64_t i = run_start[r];
    const uint64_t e = (r + 1 < nruns) ? run_start[r + 1] : n;
    for (uint64_t j = i; j < e; ++j) {
        const uint32_t cj = nidx[j];
        const cand_set sj = cand_get(L, cv.kind_id[cj]);
        uint32_t rr = cj;
        for (uint64_t q = i; q < j; ++q) {
            const uint32_t cq = nidx[q];
            if (rep[cq] != cq) continue;
            if (sets_equal(sj, cand_get(L, cv.kind_id[cq]), L.nw)) {
                rr = cq;
                break;
            }
        }
        rep[cj] = rr;
        const uint32_t f = cv.first[cj];
        if (rr == cj)
            rep_first[cj] = f;
        else if (f < rep_first[rr])
            rep_first[rr] = f;
    }
}

// The representatives into their own candidate view, in candidate order.
__global__ void __launch_bounds__(256) k_rep_compact(uint64_t nc, uint32_t const* __restrict__ rep, select_ws ws,
                                                     cand_view cv, uint32_t const* __restrict__ rep_first,
                                                     cand_view rv, uint32_t* __restrict__ rep_index, uint32_t* err) {
    __shared__ prim::ordered_select is_rep;
    const uint64_t tile = prim::select_tile(is_rep, ws.counter);
    uint32_t sel = 0;
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t c = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        if (c < nc && rep[c] == (uint32_t)c) sel |= 1u << r;
    }
    prim::select_rank(is_rep, sel, tile, ws.ntiles, ws.status, ws.total, err);
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        if (!((sel >> r) & 1u)) continue;
        const uint64_t c = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        const uint64_t p = prim::select_pos(is_rep, r);
        rv.kind_id[p] = cv.kind_id[c];
        rv.first[p] = rep_first[c];
        rv.hash[p] = cv.hash[c];
        rep_index[c] = (uint32_t)p;
    }
}

// New representatives (not in the dictionary): keys = first appearance.
__global__ void __launch_bounds__(256) k_new_reps(uint64_t nr, uint32_t const* __restrict__ rcid, select_ws ws,
                                                  cand_view rv, uint32_t* __restrict__ key,
                                                  uint32_t* __restrict__ idx, uint32_t* err) {
    __shared__ prim::ordered_select is_new;
    const uint64_t tile = prim::select_tile(is_new, ws.counter);
    uint32_t sel = 0;
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t j = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        if (j < nr && rcid[j] == NONE32) sel |= 1u << r;
    }
    prim::select_rank(is_new, sel, tile, ws.ntiles, ws.status, ws.total, err);
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        if (!((sel >> r) & 1u)) continue;
        const uint64_t j = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        const uint64_t p = prim::select_pos(is_new, r);
        key[p] = rv.first[j];
        idx[p] = (uint32_t)j;
    }
}

__global__ void k_cand_cid(uint64_t nc, uint32_t const* __restrict__ rep, uint32_t const* __restrict__ rep_index,
                           uint32_t const* __restrict__ rcid, uint32_t* __restrict__ cid) {
    uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c < nc) cid[c] = rcid[rep_index[rep[c]]];
}

// New class j (in first-appearance order) = candidate rcand[j]: its id base + j,
// hash, color count (summed per warp, one atomic per warp on the shared counter)
// and, with the candidates' bit offsets cb, its encoded length.
__global__ void k_new_classes(uint64_t nnew, uint32_t const* __restrict__ rcand, cand_view cv, list_src L,
                              uint64_t const* __restrict__ cb, uint64_t* __restrict__ nbits,
                              uint64_t* __restrict__ hashes, uint64_t base, uint32_t* __restrict__ cid,
                              unsigned long long* __restrict__ ints) {
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t n = 0;
    if (j < nnew) {
        const uint32_t c = rcand[j];
        uint32_t const* p;
        cand_list(L, cv.kind_id[c], p, n);
        if (cb) nbits[j] = cb[c + 1] - cb[c];
        hashes[j] = cv.hash[c];
        cid[c] = (uint32_t)(base + j);
    }
    const uint64_t sum = warp_sum64(n);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(ints, (unsigned long long)sum);
}

// Append new classes' encodings to the dictionary's bit vector (warp per class;
// words beyond the old end are zero, neighbours share boundary words).
__global__ void k_append_bits(uint64_t nnew, uint32_t const* __restrict__ rcand, uint64_t const* __restrict__ cw,
                              uint64_t const* __restrict__ cb, uint64_t const* __restrict__ dst_off,
                              uint64_t* __restrict__ dw) {
    const uint64_t j = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (j >= nnew) return;
    const uint32_t c = rcand[j];
    const uint64_t a = cb[c], len = cb[c + 1] - a, d = dst_off[j];
    for (uint64_t i = (threadIdx.x & 31) * 64ull; i < len; i += 32 * 64ull) {
        const uint64_t n = len - i < 64 ? len - i : 64;
        or_bits(dw, d + i, bits_at(cw, a + i), (uint32_t)n);
    }
}

// Bound: latency of two dependent lookups, so four nodes per thread (200 genomes:
// 1.35 ms with one, 0.53 so).
__global__ void __launch_bounds__(256) k_node_cid(uint64_t D, uint32_t const* __restrict__ n_rec, uint32_t R0,
                                                  uint32_t const* __restrict__ rec_cand, uint64_t mbase,
                                                  uint32_t const* __restrict__ mgrp, uint32_t const* __restrict__ cid,
                                                  uint32_t* __restrict__ n_cid) {
    const uint64_t n0 = 4 * ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x);
    uint32_t r[4], c[4];
    load_nodes4(n_rec, n0, D, r);
    uint64_t at[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        at[j] = r[j] == NONE32 ? 0 : (r[j] & MULTI_TAG) ? mbase + mgrp[r[j] & ~MULTI_TAG] : rec_cand[r[j] - R0];
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = r[j] == NONE32 ? NONE32 : cid[at[j]];
    if (n0 + 4 <= D) {
        *reinterpret_cast<uint4*>(n_cid + n0) = make_uint4(c[0], c[1], c[2], c[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (n0 + j < D) n_cid[n0 + j] = c[j];
    }
}

// ---- extension masks and clean links -------------------------------------
// The tables are read-only once they are filled, so the probes go through the
// read-only path.  First occurrence of x, or NONE32 when absent.
__device__ __forceinline__ uint32_t node_probe(slot_t<uint64_t> const* t, uint32_t cap, uint64_t x) {
    const uint64_t EMPTY = kmer_ops<uint64_t>::empty();
    const uint32_t pairs = cap / 2;
    uint32_t p = slot_home(x, pairs);
    for (uint32_t i = 0; i < pairs; ++i) {
        uint64_t k0, v0, k1, v1;
        asm volatile("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];"
                     : "=l"(k0), "=l"(v0), "=l"(k1), "=l"(v1)
                     : "l"(t + 2 * (uint64_t)p));
        if (k0 == x) return (uint32_t)v0;
        if (k1 == x) return (uint32_t)v1;
        if (k0 == EMPTY || k1 == EMPTY) return NONE32;
        p = p + 1 == pairs ? 0u : p + 1;
    }
    return NONE32;
}
__device__ __forceinline__ uint32_t node_probe(slot_t<u128> const* t, uint32_t cap, u128 x) {
    const u128 EMPTY = kmer_ops<u128>::empty();
    uint32_t p = slot_home(x, cap);
    for (uint32_t i = 0; i < cap; ++i) {
        slot_t<u128> const* e = t + p;
        const ulonglong2 v = __ldg(reinterpret_cast<ulonglong2 const*>(e));
        const u128 key = ((u128)v.y << 64) | (u128)v.x;
        if (key == x) return __ldg(&e->rank);
        if (key == EMPTY) return NONE32;
        p = p + 1 == cap ? 0u : p + 1;
    }
    return NONE32;
}

// The state (node << 1) | rc reached over a side from the node of canonical
// k-mer `can` (reverse complement `rev`), whose only neighbour there, by base
// nt, is `node`.
template <typename K>
__device__ __forceinline__ uint32_t right_state(K can, K rev, uint32_t nt, uint32_t k, uint32_t node) {
    const K nf = ((can << 2) | (K)nt) & kmer_ops<K>::mask(k);
    const K nr = (rev >> 2) | ((K)(3u - nt) << (2 * (k - 1)));
    return (node << 1) | (nf <= nr ? 0u : 1u);
}
// backward from (can, rc = false) = forward from (can, rc = true), then flipped
template <typename K>
__device__ __forceinline__ uint32_t left_state(K can, K rev, uint32_t nt, uint32_t k, uint32_t node) {
    return right_state<K>(rev, can, nt, k, node) ^ 1u;
}

// One bucket of k_ext_mask or k_ext_flat, its occurrences [ba, bb)
// (batch-relative): blocks from `first` on share them evenly, a block taking the
// k-mers first inserted by its share.  In k_ext_flat's packed form `first` = the
// occurrences of the list's buckets before it, and its blocks take equal stretches
// of all of them.  An item past the last holds the grid's size or the sum.
struct ext_item {
    uint32_t bucket, first, ba, bb;
};
// The last of the n items whose `first` is at most x (whole warps call; the first
// item's is 0): 32-way search.
__device__ __forceinline__ uint32_t find_item(ext_item const* __restrict__ items, uint32_t n, uint32_t x) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = n;  // the item is in [lo, hi)
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t i = lo + lane * step;
        const bool le = i < hi && items[i].first <= x;
        const uint32_t m = __ballot_sync(0xffffffffu, le);  // a prefix of the lanes, lane 0 among them
        const uint32_t at = 31 - __clz(m);
        const uint32_t l = lo + at * step;
        hi = min(l + step, hi);
        lo = l;
    }
    return lo;
}
struct ext_share {
    uint32_t bucket, oa, ob, ba, bb;
};
// The calling block's share (not packed).
__device__ __forceinline__ ext_share find_share(ext_item const* __restrict__ items, uint32_t n) {
    const uint32_t at = find_item(items, n, blockIdx.x);
    const ext_item it = items[at];
    const uint32_t parts = items[at + 1].first - it.first, c = blockIdx.x - it.first;
    const uint64_t len = it.bb - it.ba;
    return ext_share{it.bucket, it.ba + (uint32_t)(len * c / parts), it.ba + (uint32_t)(len * (c + 1) / parts), it.ba,
                     it.bb};
}
// Filter hash of a k-mer from v = x ^ revcomp(x), the same for both strands (no
// canonical form needed, and a neighbour's v is one XOR away from its node's).
// Bases i and k - 1 - i of v are equal, so its low half says it all.
__device__ __forceinline__ uint32_t strand_hash(uint64_t v) {
    const uint32_t a = (uint32_t)v;
    return (a ^ (a >> 15)) * 0x9e3779b1u;
}
__device__ __forceinline__ uint32_t strand_hash(u128 v) {
    const uint32_t a = (uint32_t)v, b = (uint32_t)((uint64_t)v >> 32);
    return ((a ^ (a >> 15)) * 0x85ebca6bu ^ b) * 0x9e3779b1u;
}
// Threads of a filter block: two blocks per SM, with 32 registers a thread (64 for
// 128-bit k-mers).
template <typename K>
struct ext_cfg {
    static constexpr int THREADS = sizeof(K) == 8 ? 1024 : 512;
};
constexpr uint32_t EXT_FILTER_WORDS = 102 * 1024 / 4;

// Extension masks: which of a node's 8 possible neighbours are nodes of its
// bucket, and per side the state over to the neighbour when it is the side's
// only one (link[2n] left, link[2n + 1] right, NONE32 otherwise), so k_links
// needs neither k-mers nor probes.  A neighbour is first compared with the nodes before and after (nodes
// are in insertion order: most neighbours along a record are there), then
// looked up in a bitmap of the bucket's keys in shared memory, two bits of one
// word per key, and only what passes is probed in the table, a warp's lookups packed over its
// lanes.
// Bound: instruction issue (70% of the ALU pipe), then the table's random sectors.
// 200 genomes, k = 31: 13.4 -> 7.4 ms, 60 genomes, k = 63: 11.6 -> 5.9 ms against
// all 8 neighbours probed; with one filter bit per key 8.9 / 6.1.  (The states
// for k_links add 0.4 and 0.6 ms.)
template <typename K, bool WIDE>
__global__ void __launch_bounds__(WIDE ? 1024 : ext_cfg<K>::THREADS, WIDE ? 1 : 2)
    k_ext_mask(ext_item const* __restrict__ items, uint32_t nitems, uint32_t t1, unsigned long long const* ne,
               tables<K> T, K const* __restrict__ n_key, uint32_t k, uint2 const* __restrict__ fw, uint8_t* __restrict__ n_mask,
               uint32_t* __restrict__ link) {
    typedef kmer_ops<K> ops;
    constexpr uint32_t THREADS = WIDE ? 1024 : ext_cfg<K>::THREADS;
    constexpr uint32_t WORDS = WIDE ? 2 * EXT_FILTER_WORDS : EXT_FILTER_WORDS;
    extern __shared__ __align__(16) uint32_t ext_filter[];
    __shared__ uint8_t queue[THREADS / 32][256];
    const ext_share it = find_share(items, nitems);
    auto nodes_before = [&](uint32_t o) { return o < t1 ? node_of(fw, o) : (uint32_t)*ne; };
    const uint32_t na = nodes_before(it.oa), nz = nodes_before(it.ob);
    if (na == nz) return;
    const uint32_t ba = nodes_before(it.ba), bb = nodes_before(it.bb);
    const uint32_t words = min(WORDS, ((bb - ba) / 2 + 4) & ~3u);  // 16 bits per key if they fit
    for (uint32_t i = threadIdx.x; i < words / 4; i += THREADS)
        reinterpret_cast<uint4*>(ext_filter)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    for (uint32_t n = ba + threadIdx.x; n < bb; n += THREADS) {
        const K x = n_key[n];
        const uint32_t h = strand_hash((K)(x ^ ops::revcomp(x, k)));
        atomicOr(&ext_filter[__umulhi(h, words)], (1u << (h & 31)) | (1u << ((h >> 5) & 31)));
    }
    __syncthreads();
    const K msk = ops::mask(k), msk1 = msk >> 2;
    const uint32_t top = 2 * (k - 1);
    const uint32_t cap = (uint32_t)T.tab_cap[it.bucket];
    slot_t<K> const* t = T.slots + (T.tab_off[it.bucket] - T.off0);
    const int lane = threadIdx.x & 31;
    uint8_t* const wq = queue[threadIdx.x >> 5];
    constexpr uint32_t NODE_TAG = 0x80000000u;
    for (uint32_t n0 = na + (threadIdx.x & ~31u); n0 < nz; n0 += THREADS) {
        const uint32_t n = n0 + lane;
        const bool on = n < nz;
        const K can = on ? n_key[n] : (K)0;
        const K rev = ops::revcomp(can, k);
        uint32_t out = 0, need = 0;
        uint32_t side[2] = {NONE32, NONE32};  // right, left: NODE_TAG | node, or first occurrence
        // neighbour c: base c & 3 appended to the k-mer (c < 4) or to its
        // reverse complement; appending nt to x prepends 3 - nt to revcomp(x).
        // A node y is neighbour c of this one in one of four ways: y or
        // revcomp(y) starts with the k-mer's last k - 1 bases, or the same for
        // the k-mer's reverse complement.
        auto adjacent = [&](K y, uint32_t m) {
            const K hi = y >> 2, lo = y & msk1;
            const uint32_t first = ops::low2(y >> top), last = ops::low2(y);
            auto hit = [&](uint32_t c) {
                out |= 1u << c;
                side[c >> 2] = NODE_TAG | m;
            };
            if (hi == (can & msk1)) hit(last);
            if (lo == (rev >> 2)) hit(3u - first);
            if (hi == (rev & msk1)) hit(4u + last);
            if (lo == (can >> 2)) hit(7u - first);
        };
        if (on && n > ba) adjacent(n_key[n - 1], n - 1);
        if (on && n + 1 < bb) adjacent(n_key[n + 1], n + 1);
        {
            const K vr = ((can << 2) & msk) ^ (rev >> 2), vl = ((rev << 2) & msk) ^ (can >> 2);
#pragma unroll
            for (uint32_t c = 0; c < 8; ++c) {
                const K v = (c < 4 ? vr : vl) ^ (K)(c & 3u) ^ ((K)(3u - (c & 3u)) << top);
                const uint32_t h = strand_hash(v), w = ext_filter[__umulhi(h, words)];
                need |= ((w >> (h & 31)) & (w >> ((h >> 5) & 31)) & 1u) << c;
            }
        }
        need = on ? need & ~out : 0u;
        // the warp's lookups, laid end to end over its lanes: entry = the
        // node's lane and c
        const uint32_t cnt = __popc(need);
        uint32_t total;
        const uint32_t at = warp_excl_scan32(cnt, total);
        __syncwarp();
        {
            uint32_t m = need;
            for (uint32_t i = at; m; ++i, m &= m - 1) wq[i] = (uint8_t)((lane << 3) | (__ffs(m) - 1));
        }
        __syncwarp();
        uint32_t next = at;
        for (uint32_t q0 = 0; q0 < total; q0 += 32) {
            const uint32_t e = q0 + lane < total ? wq[q0 + lane] : 0u;
            const int src = (int)(e >> 3);
            const uint32_t c = e & 7u, nt = c & 3u;
            const K cs = ops::shfl(can, src), rs = ops::shfl(rev, src);
            uint32_t got = NONE32;
            if (q0 + lane < total) {
                const K x = c < 4 ? cs : rs, y = c < 4 ? rs : cs;
                const K f = ((x << 2) | (K)nt) & msk, r = (y >> 2) | ((K)(3u - nt) << top);
                const K z = f <= r ? f : r;
                got = node_probe(t, cap, z);
            }
            // each node's lane takes its answers
            for (;;) {
                const bool mine = need != 0 && next < q0 + 32;
                if (!__any_sync(0xffffffffu, mine)) break;
                const uint32_t v = __shfl_sync(0xffffffffu, got, (int)(next & 31));
                if (mine) {
                    const uint32_t cc = __ffs(need) - 1;
                    need &= need - 1;
                    ++next;
                    if (v != NONE32) {
                        out |= 1u << cc;
                        side[cc >> 2] = v;
                    }
                }
            }
        }
        if (on) {
            n_mask[n] = (uint8_t)out;
            auto node = [&](uint32_t v) { return (v & NODE_TAG) ? v & ~NODE_TAG : node_of(fw, v); };
            uint2 l;
            l.x = __popc(out >> 4) == 1 ? left_state<K>(can, rev, __ffs(out >> 4) - 1, k, node(side[1])) : NONE32;
            l.y = __popc(out & 0xfu) == 1 ? right_state<K>(can, rev, __ffs(out & 0xfu) - 1, k, node(side[0])) : NONE32;
            reinterpret_cast<uint2*>(link)[n] = l;
        }
    }
}

// Node n's mask and states with all eight neighbours probed in its bucket's table.
template <typename K>
__device__ __forceinline__ void probe_neighbours(uint32_t n, slot_t<K> const* t, uint32_t cap,
                                                 K const* __restrict__ n_key, uint32_t k,
                                                 uint2 const* __restrict__ fw, uint8_t* __restrict__ n_mask,
                                                 uint32_t* __restrict__ link) {
    typedef kmer_ops<K> ops;
    const K msk = ops::mask(k);
    const uint32_t top = 2 * (k - 1);
    const K can = n_key[n];
    const K rev = ops::revcomp(can, k);
    uint32_t out = 0, right = NONE32, left = NONE32;
#pragma unroll
    for (uint32_t nt = 0; nt < 4; ++nt) {
        const K hi = (K)(3u - nt) << top;
        const K f = ((can << 2) | (K)nt) & msk;
        const K fr = (rev >> 2) | hi;
        const uint32_t a = node_probe(t, cap, f <= fr ? f : fr);
        if (a != NONE32) {
            out |= 1u << nt;
            right = a;
        }
        const K r = ((rev << 2) | (K)nt) & msk;
        const K rr = (can >> 2) | hi;
        const uint32_t b = node_probe(t, cap, r <= rr ? r : rr);
        if (b != NONE32) {
            out |= 1u << (4 + nt);
            left = b;
        }
    }
    n_mask[n] = (uint8_t)out;
    uint2 l;
    l.x = __popc(out >> 4) == 1 ? left_state<K>(can, rev, __ffs(out >> 4) - 1, k, node_of(fw, left)) : NONE32;
    l.y = __popc(out & 0xfu) == 1 ? right_state<K>(can, rev, __ffs(out & 0xfu) - 1, k, node_of(fw, right)) : NONE32;
    reinterpret_cast<uint2*>(link)[n] = l;
}

// The same without a filter, for buckets of more keys than one is good for and for
// groups of too few or too small buckets to fill the chip with filter blocks
// (ext_plan): small blocks in bucket order, so the buckets in flight stay in L2.
// PACKED: blocks of `share` occurrences of the list's buckets laid end to end, for
// buckets of less than a few blocks.
constexpr uint32_t FLAT_MOST = 1024;  // largest share
template <typename K, bool PACKED>
__global__ void __launch_bounds__(256, 8)
    k_ext_flat(ext_item const* __restrict__ items, uint32_t nitems, uint32_t share, uint32_t t1,
               unsigned long long const* ne, tables<K> T, K const* __restrict__ n_key, uint32_t k,
               uint2 const* __restrict__ fw, uint8_t* __restrict__ n_mask, uint32_t* __restrict__ link) {
    auto nodes_before = [&](uint32_t o) { return o < t1 ? node_of(fw, o) : (uint32_t)*ne; };
    if constexpr (!PACKED) {
        const ext_share it = find_share(items, nitems);
        const uint32_t na = nodes_before(it.oa), nz = nodes_before(it.ob);
        const uint32_t cap = (uint32_t)T.tab_cap[it.bucket];
        slot_t<K> const* t = T.slots + (T.tab_off[it.bucket] - T.off0);
        for (uint32_t n = na + threadIdx.x; n < nz; n += 256) probe_neighbours<K>(n, t, cap, n_key, k, fw, n_mask, link);
    } else {
        // of the block's buckets: its first node, and the block's nodes before it
        __shared__ uint32_t s_node[FLAT_MOST], s_at[FLAT_MOST], sw[256 / 32 + 1];
        const uint32_t v0 = blockIdx.x * share, v1 = min(v0 + share, items[nitems].first);
        const uint32_t lo = find_item(items, nitems, v0);
        const uint32_t cnt = find_item(items, nitems, v1 - 1) + 1 - lo;  // at most `share`: an item has an occurrence
        uint32_t total = 0;
        for (uint32_t i0 = 0; i0 < cnt; i0 += 256) {
            const uint32_t i = i0 + threadIdx.x;
            uint32_t a = 0, c = 0, all;
            if (i < cnt) {
                const ext_item it = items[lo + i];
                a = nodes_before(it.ba + (v0 > it.first ? v0 - it.first : 0u));
                c = nodes_before(it.ba + min(it.bb - it.ba, v1 - it.first)) - a;
            }
            const uint32_t at = total + prim::block_exclusive_scan<uint32_t, 256>(c, sw, all);
            if (i < cnt) {
                s_node[i] = a;
                s_at[i] = at;
            }
            total += all;
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < total; j += 256) {
            uint32_t q = 0;  // the node's bucket: the last that starts at or before it
            for (uint32_t h = cnt; h - q > 1;) {
                const uint32_t mid = (q + h) >> 1;
                if (s_at[mid] <= j)
                    q = mid;
                else
                    h = mid;
            }
            const uint32_t bucket = items[lo + q].bucket;
            probe_neighbours<K>(s_node[q] + (j - s_at[q]), T.slots + (T.tab_off[bucket] - T.off0),
                                (uint32_t)T.tab_cap[bucket], n_key, k, fw, n_mask, link);
        }
    }
}

__device__ __forceinline__ uint32_t fwd_nib(uint32_t m, bool rc) { return (rc ? (m >> 4) : m) & 0xfu; }
__device__ __forceinline__ uint32_t back_nib(uint32_t m, bool rc) { return (rc ? m : (m >> 4)) & 0xfu; }

// link[2n] = L port, link[2n+1] = R port: (node << 1) | rc of the state
// reached, NONE32 when the step is not clean.  On entry link holds the sides'
// only neighbours as k_ext_mask found them; a neighbour with more than one way
// back, or the node itself (the reference's walk meets its own visited k-mer
// there), ends the chain and leaves NONE32.  Nodes with at most one port are
// the chain ends, listed in any order.
// Bound: latency of the neighbours' masks, so four nodes per thread.  200
// genomes: 2.9 ms with one and the states taken from the k-mers here, 0.90 so
// (and 0.4 more in k_ext_mask, which has the k-mers at hand).
constexpr int LINKS_PER = 4;
template <bool EVEN_K>
__global__ void __launch_bounds__(256, 8) k_links(unsigned long long const* nb, unsigned long long const* ne,
                                                  uint8_t const* __restrict__ n_mask, uint32_t* __restrict__ link,
                                                  uint32_t* __restrict__ ends, unsigned long long* nends) {
    const uint64_t lo = *nb, hi = *ne;
    for (uint64_t n0 = lo + (uint64_t)blockIdx.x * (256 * LINKS_PER); n0 < hi;
         n0 += (uint64_t)gridDim.x * (256 * LINKS_PER)) {
        uint2 l[LINKS_PER];
        uint32_t ml[LINKS_PER], mr[LINKS_PER];
#pragma unroll
        for (int j = 0; j < LINKS_PER; ++j) {
            const uint64_t n = n0 + 256 * j + threadIdx.x;
            l[j] = n < hi ? reinterpret_cast<uint2 const*>(link)[n] : make_uint2(0, 0);
        }
#pragma unroll
        for (int j = 0; j < LINKS_PER; ++j) {
            const uint64_t n = n0 + 256 * j + threadIdx.x;
            ml[j] = n < hi && l[j].x != NONE32 ? n_mask[l[j].x >> 1] : 0u;
            mr[j] = n < hi && l[j].y != NONE32 ? n_mask[l[j].y >> 1] : 0u;
        }
        uint32_t end = 0;
#pragma unroll
        for (int j = 0; j < LINKS_PER; ++j) {
            const uint64_t n = n0 + 256 * j + threadIdx.x;
            if (n >= hi) continue;
            uint2 t = l[j];
            if (t.x != NONE32 && (__popc(fwd_nib(ml[j], t.x & 1u)) != 1 || (t.x >> 1) == (uint32_t)n)) t.x = NONE32;
            if (t.y != NONE32 && (__popc(back_nib(mr[j], t.y & 1u)) != 1 || (t.y >> 1) == (uint32_t)n)) t.y = NONE32;
            // a k-mer that is its own reverse complement (k even) has the same
            // neighbour on both sides, at one port of it: the walk ends there (it is
            // entered with rc = false, whose way on is the R port)
            if (EVEN_K && t.x != NONE32 && t.x == (t.y ^ 1u)) t.y = NONE32;
            if (t.x != l[j].x || t.y != l[j].y) reinterpret_cast<uint2*>(link)[n] = t;
            end |= (t.x == NONE32 || t.y == NONE32 ? 1u : 0u) << j;
        }
        unsigned long long at = block_reserve<256>(__popc(end), nends);
#pragma unroll
        for (int j = 0; j < LINKS_PER; ++j)
            if ((end >> j) & 1u) ends[at++] = (uint32_t)(n0 + 256 * j + threadIdx.x);
    }
}

// ---- chains ---------------------------------------------------------------
struct chain_ws {
    uint32_t const* link;
    uint8_t const* meta;
    uint8_t const* mask;
    uint32_t* ch_node;
    uint8_t* ch_rc;
    unsigned long long* ch_ord;
    uint8_t* ch_vis;
    uint32_t* fe;            // fragment elements (node << 1 | walk rc)
    uint32_t const* n_cid;
    uint32_t* seed_start;    // per seed node: offset into fe
    uint32_t* seed_len;      // per seed node: elements (0 = not a seed)
    uint32_t* seed_info;     // per seed node: color runs << 2 | open right << 1 | open left
    uint8_t* covered;
    unsigned long long* cursor;
    uint64_t D;
};

// Step forward from state (c, rc): use the R port when rc is false.
__device__ __forceinline__ bool chain_step(uint32_t const* link, uint32_t& c, bool& rc) {
    const uint32_t l = link[2 * (uint64_t)c + (rc ? 0 : 1)];
    if (l == NONE32) return false;
    c = l >> 1;
    rc = ((l & 1u) != 0) != rc;
    return true;
}

// Seed s's fragment: fe[start .. start + len), already stored, by this thread.
__device__ __forceinline__ void put_seed(chain_ws const& W, uint32_t s, uint64_t start, uint32_t len, bool open_l,
                                         bool open_r) {
    uint32_t runs = 1, prev = W.n_cid[W.fe[start] >> 1];
    for (uint32_t j = 1; j < len; ++j) {
        const uint32_t c = W.n_cid[W.fe[start + j] >> 1];
        runs += c != prev;
        prev = c;
    }
    W.seed_start[s] = (uint32_t)start;
    W.seed_len[s] = len;
    W.seed_info[s] = (runs << 2) | (open_r ? 2u : 0u) | (open_l ? 1u : 0u);
}

__device__ void heap_sort(unsigned long long* a, uint32_t n) {
    auto sift = [&](uint32_t i, uint32_t len) {
        for (;;) {
            uint32_t l = 2 * i + 1, m = i;
            if (l < len && a[l] > a[m]) m = l;
            if (l + 1 < len && a[l + 1] > a[m]) m = l + 1;
            if (m == i) return;
            unsigned long long t = a[i];
            a[i] = a[m];
            a[m] = t;
            i = m;
        }
    };
    if (n < 2) return;
    for (uint32_t i = n / 2; i-- > 0;) sift(i, n);
    for (uint32_t e = n - 1; e > 0; --e) {
        unsigned long long t = a[0];
        a[0] = a[e];
        a[e] = t;
        sift(0, e);
    }
}

// Replay the reference's seed loop on one chain stored at [c0, c0 + L).
__device__ void simulate_chain(chain_ws const& W, uint64_t c0, uint32_t L, bool cyclic) {
    uint32_t const* cn = W.ch_node + c0;
    uint8_t const* crc = W.ch_rc + c0;
    unsigned long long* ord = W.ch_ord + c0;
    uint8_t* vis = W.ch_vis + c0;
    for (uint32_t i = 0; i < L; ++i) {
        ord[i] = ((unsigned long long)cn[i] << 32) | i;
        vis[i] = 0;
    }
    heap_sort(ord, L);
    uint64_t fcur = c0;
    for (uint32_t t = 0; t < L; ++t) {
        const uint32_t p = (uint32_t)(ord[t] & 0xffffffffu);
        if (vis[p]) continue;
        vis[p] = 1;
        const uint32_t s = cn[p];
        const int df = crc[p] ? -1 : 1;  // chain direction of the seed's canonical forward
        const uint32_t sflags = W.meta[s] & 3u;
        uint32_t nb = 0, nf = 0;
        bool open_l = false, open_r = false;
        for (int dir = 0; dir < 2; ++dir) {
            const bool forward = dir == 1;
            if (!forward && sflags == M_LEFT) {
                open_l = __popc(back_nib(W.mask[s], false)) <= 1;
                continue;
            }
            if (forward && sflags == M_RIGHT) {
                open_r = __popc(fwd_nib(W.mask[s], false)) <= 1;
                continue;
            }
            const int step = forward ? df : -df;
            int64_t q = p;
            uint32_t cnt = 0;
            for (;;) {
                int64_t q2 = q + step;
                if (cyclic) {
                    if (q2 < 0) q2 += L;
                    if (q2 >= (int64_t)L) q2 -= L;
                } else if (q2 < 0 || q2 >= (int64_t)L) {
                    break;
                }
                if (vis[q2]) break;
                vis[q2] = 1;
                ++cnt;
                q = q2;
                const uint32_t nd = cn[q];
                const uint32_t f = W.meta[nd] & 3u;
                if (f == M_LEFT || f == M_RIGHT) {
                    const bool wrc = (df == 1) ? (crc[q] != 0) : (crc[q] == 0);
                    if (forward)
                        open_r = __popc(fwd_nib(W.mask[nd], wrc)) <= 1;
                    else
                        open_l = __popc(back_nib(W.mask[nd], wrc)) <= 1;
                    break;
                }
            }
            if (forward)
                nf = cnt;
            else
                nb = cnt;
        }
        const uint32_t flen = nb + 1 + nf;
        for (uint32_t j = 0; j < flen; ++j) {
            int64_t q = (int64_t)p + (int64_t)df * ((int64_t)j - (int64_t)nb);
            if (cyclic) {
                q %= (int64_t)L;
                if (q < 0) q += L;
            }
            const bool wrc = (df == 1) ? (crc[q] != 0) : (crc[q] == 0);
            W.fe[fcur + j] = (cn[q] << 1) | (wrc ? 1u : 0u);
        }
        put_seed(W, s, fcur, flen, open_l, open_r);
        fcur += flen;
    }
}

// Seed loop of a chain of at most 64 nodes: the visited set is a register
// mask and each seed is the unvisited position with the smallest node index
// (a scan instead of a sort; chains hold one or two fragments in practice).
// Same walk rules as simulate_chain.
__device__ void simulate_chain_small(chain_ws const& W, uint64_t c0, uint32_t L, bool cyclic) {
    uint32_t const* cn = W.ch_node + c0;
    uint8_t const* crc = W.ch_rc + c0;
    const uint64_t all = (L >= 64) ? ~0ull : ((1ull << L) - 1);
    uint64_t vis = 0;
    uint64_t fcur = c0;
    while (vis != all) {
        uint32_t p = 0, best = NONE32;
        for (uint32_t q = 0; q < L; ++q) {
            if ((vis >> q) & 1ull) continue;
            const uint32_t nd = cn[q];
            if (nd < best) {
                best = nd;
                p = q;
            }
        }
        vis |= 1ull << p;
        const uint32_t s = best;
        const int df = crc[p] ? -1 : 1;
        const uint32_t sflags = W.meta[s] & 3u;
        const uint32_t smask = W.mask[s];
        uint32_t nb = 0, nf = 0;
        bool open_l = false, open_r = false;
        for (int dir = 0; dir < 2; ++dir) {
            const bool forward = dir == 1;
            if (!forward && sflags == M_LEFT) {
                open_l = __popc(back_nib(smask, false)) <= 1;
                continue;
            }
            if (forward && sflags == M_RIGHT) {
                open_r = __popc(fwd_nib(smask, false)) <= 1;
                continue;
            }
            const int step = forward ? df : -df;
            int q = (int)p;
            uint32_t cnt = 0;
            for (;;) {
                int q2 = q + step;
                if (cyclic) {
                    if (q2 < 0) q2 += (int)L;
                    if (q2 >= (int)L) q2 -= (int)L;
                } else if (q2 < 0 || q2 >= (int)L) {
                    break;
                }
                if ((vis >> q2) & 1ull) break;
                vis |= 1ull << q2;
                ++cnt;
                q = q2;
                const uint32_t nd = cn[q];
                const uint32_t f = W.meta[nd] & 3u;
                if (f == M_LEFT || f == M_RIGHT) {
                    const bool wrc = (df == 1) ? (crc[q] != 0) : (crc[q] == 0);
                    if (forward)
                        open_r = __popc(fwd_nib(W.mask[nd], wrc)) <= 1;
                    else
                        open_l = __popc(back_nib(W.mask[nd], wrc)) <= 1;
                    break;
                }
            }
            if (forward)
                nf = cnt;
            else
                nb = cnt;
        }
        const uint32_t flen = nb + 1 + nf;
        for (uint32_t j = 0; j < flen; ++j) {
            int q = (int)p + df * ((int)j - (int)nb);
            if (cyclic) {
                q %= (int)L;
                if (q < 0) q += (int)L;
            }
            const bool wrc = (df == 1) ? (crc[q] != 0) : (crc[q] == 0);
            W.fe[fcur + j] = (cn[q] << 1) | (wrc ? 1u : 0u);
        }
        put_seed(W, s, fcur, flen, open_l, open_r);
        fcur += flen;
    }
}

// Each path end walks to the other end; the end with the smaller node index
// leads and reserves the chain's elements [c0, c0 + L).  Most chains are one
// fragment: no node inside the chain breaks a contig, and the seed -- the smallest
// node -- steps to both ends (a seed flagged on the side it would step to does
// not).  The leader then writes that fragment itself, on a second walk over the
// links it just read; the other chains go to `heads` (node | rc << 31, L, c0 low,
// c0 high) for k_chain_paths.
// Bound: issue (72%; half the lanes walk a chain the other end leads), then the
// latency of the link reads, mostly cache hits (a chain's nodes are
// neighbours in node order).  Finding the ends, the leaders, laying out every chain
// and replaying the seed loop on it, the cycle check, and the run counts from the
// fragments took 9.8 ms of a 200-genome build; this takes 4.1 and the ends 0.9 more
// in k_links.
__global__ void __launch_bounds__(256) k_chain_lead(chain_ws W, uint32_t const* __restrict__ ends,
                                                    unsigned long long const* __restrict__ pends,
                                                    uint4* __restrict__ heads, unsigned long long* __restrict__ nheads,
                                                    uint32_t* err) {
    const uint64_t nends = *pends;  // (the grid may be larger)
    if ((uint64_t)blockIdx.x * blockDim.x >= nends) return;
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t c = 0, L = 0;
    bool rc = false, lead = false;
    // of the walk: the smallest node with its position, orientation and flags;
    // the last node; how many nodes before the last, and after the first, break
    uint32_t seed = 0, seed_at = 0, seed_f = 0, last = 0, last_f = 0, first_f = 0, breaks = 0;
    bool seed_rc = false, last_rc = false;
    if (i < nends) {
        c = ends[i];
        const uint32_t ll = W.link[2 * (uint64_t)c], lr = W.link[2 * (uint64_t)c + 1];
        rc = (lr == NONE32);  // walk out through the linked port
        L = 1;
        lead = true;
        seed = last = c;
        seed_rc = last_rc = rc;
        seed_f = last_f = first_f = W.meta[c] & 3u;
        if (ll != NONE32 || lr != NONE32) {
            uint32_t cc = c;
            bool r = rc;
            while (chain_step(W.link, cc, r)) {
                if (L > 1) breaks += last_f == M_LEFT || last_f == M_RIGHT;  // `last` was not the first, nor is it the last
                last = cc;
                last_rc = r;
                last_f = W.meta[cc] & 3u;
                if (cc < seed) {
                    seed = cc;
                    seed_at = L;
                    seed_rc = r;
                    seed_f = last_f;
                }
                if (++L > W.D) {
                    set_error(err, ERR_CHAIN_LIMIT);
                    lead = false;
                    break;
                }
            }
            if (last < c) lead = false;  // the other end leads
        }
    }
    // the whole chain from its one seed?
    const bool inside = seed_at > 0 && seed_at + 1 < L;
    if (inside) breaks -= seed_f == M_LEFT || seed_f == M_RIGHT;
    const bool fwd = !seed_rc;  // the walk goes the way of the seed's k-mer
    const bool before = seed_at > 0, after = seed_at + 1 < L;
    const bool has_b = fwd ? before : after, has_f = fwd ? after : before;  // nodes behind / ahead of the seed
    const bool whole = lead && breaks == 0 && !(seed_f == M_LEFT && has_b) && !(seed_f == M_RIGHT && has_f);
    const unsigned long long c0 = block_reserve<256>(lead ? L : 0, W.cursor);
    const unsigned long long h = block_reserve<256>(lead && !whole ? 1 : 0, nheads);
    if (!lead) return;
    if (c0 + L > W.D) {
        // (chains partition the nodes, anything else is a bug: an error, and no
        // chain is left half described)
        set_error(err, ERR_CAPACITY);
        if (!whole) heads[h] = make_uint4(0, 0, 0, 0);
        return;
    }
    if (!whole) {
        heads[h] = make_uint4(c | (rc ? 0x80000000u : 0u), L, (uint32_t)c0, (uint32_t)(c0 >> 32));
        return;
    }
    // open ends, as the seed loop leaves them: a seed flagged there, or the last
    // node stepped to when it is flagged
    auto breaking = [](uint32_t f) { return f == M_LEFT || f == M_RIGHT; };
    bool open_l = false, open_r = false;
    if (seed_f == M_LEFT) {
        open_l = __popc(back_nib(W.mask[seed], false)) <= 1;
    } else if (has_b) {
        const uint32_t e = fwd ? c : last, ef = fwd ? first_f : last_f;
        const bool wrc = fwd ? rc : !last_rc;
        if (breaking(ef)) open_l = __popc(back_nib(W.mask[e], wrc)) <= 1;
    }
    if (seed_f == M_RIGHT) {
        open_r = __popc(fwd_nib(W.mask[seed], false)) <= 1;
    } else if (has_f) {
        const uint32_t e = fwd ? last : c, ef = fwd ? last_f : first_f;
        const bool wrc = fwd ? last_rc : !rc;
        if (breaking(ef)) open_r = __popc(fwd_nib(W.mask[e], wrc)) <= 1;
    }
    uint32_t cc = c, runs = 1, prev = W.n_cid[c];
    bool r = rc;
    for (uint32_t j = 0;;) {
        W.fe[c0 + (fwd ? j : L - 1 - j)] = (cc << 1) | ((r == fwd) ? 1u : 0u);
        if (++j == L) break;
        chain_step(W.link, cc, r);
        const uint32_t q = W.n_cid[cc];
        runs += q != prev;
        prev = q;
    }
    W.seed_start[seed] = (uint32_t)c0;
    W.seed_len[seed] = L;
    W.seed_info[seed] = (runs << 2) | (open_r ? 2u : 0u) | (open_l ? 1u : 0u);
}

// The chains of more than one fragment, a thread each: lay the chain out at c0
// and replay the seed loop.
__global__ void __launch_bounds__(128) k_chain_paths(chain_ws W, uint4 const* __restrict__ heads,
                                                     unsigned long long const* __restrict__ nheads) {
    for (uint64_t h = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; h < *nheads;
         h += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 hd = heads[h];
        uint32_t cc = hd.x & 0x7fffffffu;
        bool r = (hd.x >> 31) != 0;
        const uint32_t L = hd.y;
        const uint64_t c0 = ((uint64_t)hd.w << 32) | hd.z;
        if (L == 0) continue;
        W.ch_node[c0] = cc;
        W.ch_rc[c0] = r ? 1 : 0;
        for (uint32_t i = 1; i < L && chain_step(W.link, cc, r); ++i) {
            W.ch_node[c0 + i] = cc;
            W.ch_rc[c0 + i] = r ? 1 : 0;
        }
        if (L <= 64)
            simulate_chain_small(W, c0, L, false);
        else
            simulate_chain(W, c0, L, false);
    }
}

// The number of nodes on paths; when that is not all there are cycles, and
// k_chain_cycles needs to know the others.  (More than all: an error is set, and not
// every fragment element is written.)
__global__ void k_chain_covered(chain_ws W, unsigned long long* __restrict__ paths) {
    const uint64_t n = *W.cursor;
    if (blockIdx.x == 0 && threadIdx.x == 0) *paths = n;
    if (n >= W.D) return;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        W.covered[W.fe[i] >> 1] = 1;
}

// Cycles: nodes left uncovered; the smallest node index of a cycle leads.
// `paths` = the nodes on paths.
__global__ void k_chain_cycles(chain_ws W, unsigned long long const* __restrict__ paths, uint32_t* err) {
    if (*paths >= W.D) return;
    for (uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; n < W.D;
         n += (uint64_t)gridDim.x * blockDim.x) {
        if (W.covered[n]) continue;
        uint32_t cc = (uint32_t)n;
        bool r = false, lead = true;
        uint32_t L = 1;
        for (;;) {
            if (!chain_step(W.link, cc, r)) {
                set_error(err, ERR_CHAIN_LIMIT);  // an uncovered node must be on a cycle
                return;
            }
            if (cc == n) break;
            if (cc < n) {
                lead = false;
                break;
            }
            if (++L > W.D) {
                set_error(err, ERR_CHAIN_LIMIT);
                return;
            }
        }
        if (!lead) continue;
        const uint64_t c0 = atomicAdd(W.cursor, (unsigned long long)L);
        if (c0 + L > W.D) {
            set_error(err, ERR_CAPACITY);
            return;
        }
        cc = (uint32_t)n;
        r = false;
        W.ch_node[c0] = cc;
        W.ch_rc[c0] = 0;
        for (uint32_t i = 1; i < L; ++i) {
            chain_step(W.link, cc, r);
            W.ch_node[c0 + i] = cc;
            W.ch_rc[c0 + i] = r ? 1 : 0;
        }
        if (L <= 64)
            simulate_chain_small(W, c0, L, true);
        else
            simulate_chain(W, c0, L, true);
    }
}

// ---- fragments --------------------------------------------------------------
// Fragments in node order of their seeds, in one pass over the nodes: seed_of[f],
// and off[f], the offset of its record (frag_unitig_writer::write_batch layout);
// tot[0..2] = fragments, record bytes, sequence bases.
__global__ void __launch_bounds__(256) k_seed_list(uint64_t D, uint32_t const* __restrict__ seed_len,
                                                   uint32_t const* __restrict__ seed_info, uint32_t k, select_ws ws,
                                                   unsigned long long* status_bytes, uint32_t* __restrict__ seed_of,
                                                   uint64_t* __restrict__ off, unsigned long long* __restrict__ tot,
                                                   uint32_t* err) {
    __shared__ prim::ordered_select seeds;
    __shared__ uint64_t wbytes[prim::SEL_ROUNDS * 8], s_bytes;
    const uint64_t tile = prim::select_tile(seeds, ws.counter);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t len[prim::SEL_ROUNDS], info[prim::SEL_ROUNDS], sel = 0;
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t n = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        len[r] = n < D ? seed_len[n] : 0u;
    }
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        info[r] = 0;
        if (len[r]) {
            info[r] = seed_info[tile * prim::SEL_TILE + 256u * r + threadIdx.x];
            sel |= 1u << r;
        }
    }
    auto bytes = [&](int r) { return len[r] ? 9 + 12ull * (info[r] >> 2) + k + len[r] - 1 : 0ull; };
    uint64_t at[prim::SEL_ROUNDS], seq = 0;  // record bytes before this element in its (round, warp)
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t size = bytes(r);
        // (32-bit sums unless some record is of 64 MiB)
        if (!__any_sync(0xffffffffu, (size >> 26) != 0)) {
            const uint32_t incl = prim::warp_inclusive_scan((uint32_t)size);
            at[r] = incl - (uint32_t)size;
        } else {
            at[r] = prim::warp_inclusive_scan(size) - size;
        }
        if (lane == 31) wbytes[r * 8 + warp] = at[r] + size;
        if (len[r]) seq += (uint64_t)k + len[r] - 1;
    }
    prim::select_put(seeds, sel);
    __syncthreads();
    if (warp == 0) {
        prim::select_scan(seeds, tile, ws.ntiles, ws.status, tot, err);
    } else if (warp == 1) {
        const uint64_t c0 = wbytes[2 * lane], c1 = wbytes[2 * lane + 1];
        const uint64_t x = prim::warp_inclusive_scan(c0 + c1);
        const uint64_t sum = __shfl_sync(0xffffffffu, x, 31);
        wbytes[2 * lane] = x - c0 - c1;
        wbytes[2 * lane + 1] = x - c1;
        uint64_t excl = 0;
        const bool ok = prim::lookback_exclusive(status_bytes, tile, sum, excl);
        if (lane == 0) {
            if (!ok) set_error(err, ERR_CHAIN_LIMIT);
            s_bytes = excl;
            if (tile == ws.ntiles - 1) tot[1] = excl + sum;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < prim::SEL_ROUNDS; ++r) {
        const uint64_t n = tile * prim::SEL_TILE + 256u * r + threadIdx.x;
        const bool f = (sel >> r) & 1u;
        if (!f && n != D - 1) continue;
        const uint64_t at_f = prim::select_pos(seeds, r), o = s_bytes + wbytes[r * 8 + warp] + at[r];
        if (f) {
            seed_of[at_f] = (uint32_t)n;
            off[at_f] = o;
        }
        // the total closes the offsets
        if (n == D - 1) off[at_f + (f ? 1 : 0)] = o + bytes(r);
    }
    for (int o = 16; o; o >>= 1) seq += __shfl_xor_sync(0xffffffffu, seq, o);
    if (lane == 0 && seq) atomicAdd(tot + 2, (unsigned long long)seq);
}

// Bytes one after another at any address (shared or global memory), stored by
// aligned 4-byte words; the words at the two ends, which hold others' bytes, byte
// by byte.
struct byte_writer {
    uint8_t* p;      // next word (aligned)
    uint64_t acc;    // bytes not yet stored
    uint32_t fill;   // of them (< 4), counting the first word's bytes before the start
    uint32_t skip;   // bytes of the next word before the start
    __device__ __forceinline__ explicit byte_writer(uint8_t* o) {
        skip = fill = (uint32_t)(reinterpret_cast<uintptr_t>(o) & 3);
        p = o - fill;
        acc = 0;
    }
    __device__ __forceinline__ void word() {
        const uint32_t w = (uint32_t)acc;
        if (skip == 0) {
            *reinterpret_cast<uint32_t*>(p) = w;
        } else {
            for (uint32_t i = skip; i < 4; ++i) p[i] = (uint8_t)(w >> (8 * i));
            skip = 0;
        }
        p += 4;
        acc >>= 32;
    }
    __device__ __forceinline__ void put4(uint32_t v) {
        acc |= (uint64_t)v << (8 * fill);
        word();
    }
    __device__ __forceinline__ void put1(uint32_t v) {
        acc |= (uint64_t)v << (8 * fill);
        if (++fill == 4) {
            word();
            fill = 0;
        }
    }
    __device__ __forceinline__ void end() {
        for (uint32_t i = skip; i < fill; ++i) p[i] = (uint8_t)(acc >> (8 * i));
    }
};

// ASCII of the four 2-bit bases of b, the first in the low bits.
__device__ __forceinline__ uint32_t ascii4(uint32_t b) {
    uint32_t s = (b | (b << 4)) & 0x0f0fu;
    s = (s | (s << 2)) & 0x3333u;
    return __byte_perm(0x54474341u, 0u, s);  // byte i = "ACGT"[nibble i]
}
// Bases of a k-mer, base i at bits 2i.
__device__ __forceinline__ void bases_of(uint64_t w, uint32_t k, uint64_t& lo, uint64_t& hi) {
    lo = rev2_64(w) >> (64 - 2 * k);
    hi = 0;
}
__device__ __forceinline__ void bases_of(u128 w, uint32_t k, uint64_t& lo, uint64_t& hi) {
    const u128 x = kmer_ops<u128>::rev2_128(w) >> (128 - 2 * k);
    lo = (uint64_t)x;
    hi = (uint64_t)(x >> 64);
}

// One fragment record (unitig_spill.hpp:491-522 layout) at `o` (shared or
// global memory).  Each base after the first k-mer is the last base of the
// oriented k-mer: the low 2 bits of the key, or the complement of its first
// base when the walk is reverse -- no reverse complement per element.
template <typename K>
__device__ __forceinline__ void emit_fragment(uint8_t* o, uint32_t n, uint32_t const* __restrict__ seed_start,
                                              uint32_t const* __restrict__ seed_len,
                                              uint32_t const* __restrict__ seed_info, uint32_t const* __restrict__ fe,
                                              uint32_t const* __restrict__ n_cid, K const* __restrict__ n_key,
                                              uint32_t k) {
    typedef kmer_ops<K> ops;
    const uint32_t len = seed_len[n], info = seed_info[n];
    uint32_t const* el = fe + seed_start[n];
    byte_writer w(o);
    w.put1(info & 3u);
    w.put4(info >> 2);
    auto run = [&](uint32_t cid, uint32_t cnt) {
        w.put4(cid);
        w.put4(cid == NONE32 ? 0xffffffffu : 0u);
        w.put4(cnt);
    };
    uint32_t prev = n_cid[el[0] >> 1], cnt = len;
    if ((info >> 2) > 1) {
        cnt = 1;
        for (uint32_t j = 1; j < len; ++j) {
            const uint32_t c = n_cid[el[j] >> 1];
            if (c != prev) {
                run(prev, cnt);
                prev = c;
                cnt = 0;
            }
            ++cnt;
        }
    }
    run(prev, cnt);
    w.put4(k + len - 1);
    uint64_t lo, hi;
    {
        const uint32_t e = el[0];
        K x = n_key[e >> 1];
        if (e & 1u) x = ops::revcomp(x, k);
        bases_of(x, k, lo, hi);
    }
    uint32_t left = k;
    for (; left >= 4; left -= 4) {
        w.put4(ascii4((uint32_t)lo & 0xffu));
        lo >>= 8;
        if constexpr (sizeof(K) == 16) {
            lo |= hi << 56;
            hi >>= 8;
        }
    }
    uint32_t b = (uint32_t)lo;  // `left` < 4 bases not yet written
    const uint32_t top = 2 * (k - 1);
    for (uint32_t j = 1; j < len; ++j) {
        const uint32_t e = el[j];
        const K x = n_key[e >> 1];
        b |= ((e & 1u) ? 3u - ops::low2(x >> top) : ops::low2(x)) << (2 * left);
        if (++left == 4) {
            w.put4(ascii4(b));
            b = left = 0;
        }
    }
    for (uint32_t x = ascii4(b); left; --left, x >>= 8) w.put1(x & 0xffu);
    w.end();
}

// Fragments [f0, f0 + FW_THREADS) of a block occupy one contiguous byte range
// of the output.  They are laid out in shared memory with the range's
// 16-byte phase and stored with aligned 16-byte writes (bytes at the two
// ragged ends one by one), instead of a few dozen scattered byte stores per
// fragment.  A block whose range does not fit writes directly.
// Bound: the gathers of a fragment's elements (its keys and color sets).  With the
// records put together byte by byte 5.7 ms for 2.3 GB of a 200-genome build, by
// words 3.9 (0.6 TB/s), with 24 KB of buffer and 64 registers for 8 blocks per SM
// (32 KB and 76: 6) 3.4.
constexpr int FW_THREADS = 128;
constexpr int FW_BYTES = 24 * 1024;

template <typename K>
__global__ void __launch_bounds__(FW_THREADS, 8)
    k_frag_write(uint64_t F, uint32_t const* __restrict__ seed_of, uint32_t const* __restrict__ seed_start,
                 uint32_t const* __restrict__ seed_len, uint32_t const* __restrict__ seed_info,
                 uint32_t const* __restrict__ fe, uint32_t const* __restrict__ n_cid, K const* __restrict__ n_key,
                 uint32_t k, uint64_t const* __restrict__ off, uint64_t base, uint8_t* __restrict__ out) {
    __shared__ __align__(16) uint8_t buf[FW_BYTES];
    const uint64_t f0 = (uint64_t)blockIdx.x * FW_THREADS;
    const uint64_t f1 = (f0 + FW_THREADS < F) ? f0 + FW_THREADS : F;
    const uint64_t g0 = base + off[f0], g1 = base + off[f1];  // out is 16-byte aligned, out + base need not be
    const uint32_t phase = (uint32_t)(g0 & 15);
    const uint64_t f = f0 + threadIdx.x;
    if (g1 - g0 + phase > (uint64_t)FW_BYTES) {  // block-uniform
        if (f < F) emit_fragment<K>(out + base + off[f], seed_of[f], seed_start, seed_len, seed_info, fe, n_cid, n_key, k);
        return;
    }
    if (f < F)
        emit_fragment<K>(buf + phase + (base + off[f] - g0), seed_of[f], seed_start, seed_len, seed_info, fe, n_cid, n_key,
                         k);
    __syncthreads();
    const uint64_t a0 = (g0 + 15) & ~uint64_t(15);  // first aligned byte inside the range
    const uint64_t a1 = g1 & ~uint64_t(15);         // end of the aligned part
    if (a0 >= a1) {
        for (uint64_t b = g0 + threadIdx.x; b < g1; b += FW_THREADS) out[b] = buf[phase + (b - g0)];
        return;
    }
    for (uint64_t b = g0 + threadIdx.x; b < a0; b += FW_THREADS) out[b] = buf[phase + (b - g0)];
    for (uint64_t b = a1 + threadIdx.x; b < g1; b += FW_THREADS) out[b] = buf[phase + (b - g0)];
    const uint64_t nchunks = (a1 - a0) >> 4;
    uint4 const* src = reinterpret_cast<uint4 const*>(buf + phase + (a0 - g0));  // 16-byte aligned
    uint4* dst = reinterpret_cast<uint4*>(out + a0);
    for (uint64_t c = threadIdx.x; c < nchunks; c += FW_THREADS) dst[c] = src[c];
}

// ---------------------------------------------------------------------------
// ---- small helpers ----------------------------------------------------------
__global__ void k_add_offsets(uint64_t n, uint64_t const* __restrict__ src, uint64_t add,
                              uint64_t* __restrict__ dst) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[i] + add;
}
__global__ void k_copy_u64x2(unsigned long long const* src, unsigned long long* dst) {
    dst[0] = src[0];
    dst[1] = src[1];
}

void add_offsets(uint64_t const* src, uint64_t n, uint64_t add, uint64_t* dst, cudaStream_t st) {
    if (!n) return;
    k_add_offsets<<<grid(n, 256), 256, 0, st>>>(n, src, add, dst);
    CDBG_CHECK_LAUNCH();
}

void check_device_error_word(uint32_t* d_err, cudaStream_t st, char const* stage) {
    const uint32_t e = read_dev(d_err, st);
    if (e == ERR_NONE) return;
    CDBG_CUDA(cudaMemsetAsync(d_err, 0, 4, st));
    static char const* names[] = {"none", "hash table full", "field overflow", "malformed record",
                                  "capacity exceeded", "chain walk bound exceeded"};
    throw std::runtime_error(std::string("device error in ") + stage + ": " +
                             (e < 6 ? names[e] : "unknown"));
}

// ---------------------------------------------------------------------------
__global__ void k_dict_insert(uint64_t c0, uint64_t c1, uint64_t const* __restrict__ cls_hash,
                              uint64_t* __restrict__ slot_hash, uint32_t* __restrict__ slot_cid, uint64_t mask,
                              uint32_t* err) {
    uint64_t c = c0 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= c1) return;
    const uint64_t h = cls_hash[c];
    uint64_t s = h & mask;
    for (uint64_t i = 0; i <= mask; ++i) {
        const uint64_t old = atomicCAS((unsigned long long*)&slot_hash[s], (unsigned long long)HASH_EMPTY,
                                       (unsigned long long)h);
        if (old == HASH_EMPTY) {
            slot_cid[s] = (uint32_t)c;
            return;
        }
        s = (s + 1) & mask;
    }
    set_error(err, ERR_TABLE_FULL);
}

// Global color-class dictionary (persists across bucket batches): per class
// its 64-bit set hash and its bit range in the encoded .color_sets vector; an
// open-addressing table hash -> class id.  Equality is tested on encodings.
struct class_dict {
    dvec<uint64_t>& cls_hash;  // n
    dvec<uint64_t>& bit_off;   // n + 1 (last = nbits)
    dvec<uint64_t>& words;     // encoded classes, zero beyond nbits
    dvec<uint64_t>& slot_hash;
    dvec<uint32_t>& slot_cid;
    uint64_t n = 0, nbits = 0, total_integers = 0, mask = 0;
    uint64_t tabled = 0;  // classes in the table: the first batch needs none, later ones add the rest

    explicit class_dict(phase2_state& S)
        : cls_hash(S.cls_hash), bit_off(S.bit_off), words(S.words), slot_hash(S.slot_hash), slot_cid(S.slot_cid) {}

    // Start empty, keeping the storage of a previous build (words are zeroed
    // where the previous build wrote).
    void init(cudaStream_t st) {
        bit_off.reserve(1024, st);
        CDBG_CUDA(cudaMemsetAsync(bit_off.p, 0, 8, st));
        bit_off.n = 1;
        words.reserve(1024, st, true);
        if (words.n) CDBG_CUDA(cudaMemsetAsync(words.p, 0, 8 * std::min(words.n + 4, words.cap), st));
        words.n = 0;
        cls_hash.n = 0;
    }
    dict_view view() const { return dict_view{slot_hash.p, slot_cid.p, mask, bit_off.p, words.p}; }
    // Every class in the table (load <= 1/2), before a lookup.  A resized table is
    // rebuilt from every class hash.
    void ensure_table(cudaStream_t st, uint32_t* d_err) {
        uint64_t cap = 1024;
        while (cap < 2 * n) cap <<= 1;
        uint64_t from = tabled;
        if (!slot_hash.p || cap - 1 > mask) {
            slot_hash.reserve(cap, st);
            slot_cid.reserve(cap, st);
            mask = cap - 1;
            CDBG_CUDA(cudaMemsetAsync(slot_hash.p, 0xff, cap * 8, st));
            from = 0;
        }
        if (n > from) {
            k_dict_insert<<<grid(n - from, 256), 256, 0, st>>>(from, n, cls_hash.p, slot_hash.p, slot_cid.p, mask,
                                                              d_err);
            CDBG_CHECK_LAUNCH();
        }
        tabled = n;
    }
};

// A block of zeroed device words handed out piece by piece.
struct zero_block {
    unsigned long long* p;
    uint64_t used = 0, cap;
    zero_block(uint64_t words, dev_arena& A, cudaStream_t st) : cap(words) {
        p = A.alloc<unsigned long long>(words);
        CDBG_CUDA(cudaMemsetAsync(p, 0, 8 * words, st));
    }
    template <typename T>
    T* take(uint64_t count) {
        T* r = reinterpret_cast<T*>(p + used);
        used += (count * sizeof(T) + 7) / 8;
        if (used > cap) throw std::runtime_error("zero_block: block too small");
        return r;
    }
    static uint64_t tiles(uint64_t n, uint64_t tile) { return std::max<uint64_t>(1, ceil_div(n, tile)); }
    // words of an ordered selection over n elements
    static uint64_t select_words(uint64_t n, uint64_t tile = prim::SEL_TILE) { return tiles(n, tile) + 2; }
    select_ws select(uint64_t n, uint64_t tile = prim::SEL_TILE) {
        select_ws w;
        w.ntiles = tiles(n, tile);
        w.status = take<unsigned long long>(w.ntiles);
        w.total = take<unsigned long long>(1);
        w.counter = take<uint32_t>(1);
        return w;
    }
};

template <typename K>
void run_batch(record_set const& rs, rec_view const& R, phase2_params const& p, uint32_t b0, uint32_t b1,
               std::vector<uint64_t> const& bocc, dev_arena& A, cudaStream_t st, uint32_t* d_err,
               class_dict& dict, phase2_result& out, std::vector<uint64_t> const& hbstart, uint64_t* d_rhash,
               dvec<uint8_t>& dfrag, dvec<uint64_t>& dfoff) {
    const uint32_t k = p.k, C = p.num_colors;
    const uint64_t R0 = hbstart[b0], R1 = hbstart[b1];
    const uint64_t nrec = R1 - R0;
    const uint64_t O0 = bocc[b0], O1 = bocc[b1];
    const uint64_t nocc = O1 - O0;
    if (nocc == 0) return;
    auto mark = A.mark();
    // ---- tables: one open-addressing table per bucket, processed in bucket
    // groups of at most p.group_bytes of tables (one group per batch by
    // default): a group's tables are built, numbered and probed (insert, first
    // occurrences, nodes, extension masks, links) before the next group
    // reuses their memory, so a group that fits in L2 stays cache-resident
    const uint32_t nb = b1 - b0;
    const uint64_t q = std::min<uint32_t>(16, std::max<uint32_t>(5, p.table_slots_q));
    std::vector<uint64_t> toff(nb + 1), tcap(nb);
    uint64_t T = 0;
    for (uint32_t b = 0; b < nb; ++b) {
        const uint64_t o = bocc[b0 + b + 1] - bocc[b0 + b];
        // slots per occurrence q/4 > 1 (distinct <= occurrences): the default
        // 2 keeps the load factor <= 1/2 for short unsuccessful probes in the
        // neighbour lookups
        const uint64_t cap = o ? std::max<uint64_t>(64, (o * q / 4 + 17) & ~uint64_t(1)) : 0;  // whole pairs
        toff[b] = T;
        tcap[b] = cap;
        T += cap;
    }
    toff[nb] = T;
    if (T >= (1ull << 31)) throw std::runtime_error("k-mer table of one bucket batch exceeds 2^31 slots");
    if (nrec > MAX_BATCH_RECORDS) throw std::runtime_error("more than 2^28 - 2 records in one bucket");
    const uint64_t gslots = std::max<uint64_t>(1024, p.group_bytes / sizeof(slot_t<K>));
    std::vector<uint32_t> gb{0};  // group boundaries (batch-relative buckets)
    for (uint32_t b = 1; b <= nb; ++b)
        if (b == nb || toff[b + 1] - toff[gb.back()] > gslots) gb.push_back(b);
    if (gb.back() != nb) gb.push_back(nb);
    const size_t ng = gb.size() - 1;
    uint64_t Tmax = 0;
    for (size_t g = 0; g < ng; ++g) Tmax = std::max<uint64_t>(Tmax, toff[gb[g + 1]] - toff[gb[g]]);
    uint32_t* occ_slot = A.alloc<uint32_t>(nocc);
    // the buckets of k_ext_mask, of its wide form and of k_ext_flat, per group, with
    // their blocks
    std::vector<ext_item> items;
    std::vector<uint32_t> gitem(3 * ng + 1, 0), gblocks(3 * ng, 0), gshare(ng, 0);  // (share 0: not packed)
    const ext_plan plan(sizeof(K) == 16, nocc);
    for (size_t g = 0; g < ng; ++g) {
        uint64_t const* off = bocc.data() + b0 + gb[g];
        const uint32_t gn = gb[g + 1] - gb[g];
        const uint64_t cut = plan.cut(off, gn);
        const uint64_t tn = off[gn] - off[0];
        std::vector<ext_item> of[3];
        uint32_t first[3] = {0, 0, 0};
        for (uint32_t b = 0; b < gn; ++b) {
            const uint64_t ba = off[b] - O0, n = off[b + 1] - off[b];
            if (n == 0) continue;
            const int f = plan.form(n, cut);
            of[f].push_back(ext_item{b, first[f], (uint32_t)ba, (uint32_t)(ba + n)});
            first[f] += (uint32_t)(f == EXT_FLAT ? n : plan.parts(n));
        }
        const uint32_t share = plan.flat_occ(tn);
        const bool packed = plan.packed(first[EXT_FLAT], of[EXT_FLAT].size(), tn);
        if (!packed) {
            first[EXT_FLAT] = 0;
            for (ext_item& it : of[EXT_FLAT]) {
                it.first = first[EXT_FLAT];
                first[EXT_FLAT] += (it.bb - it.ba + share - 1) / share;
            }
        }
        for (int f = 0; f < 3; ++f) {
            items.insert(items.end(), of[f].begin(), of[f].end());
            items.push_back(ext_item{0, first[f], 0, 0});
            gitem[3 * g + f + 1] = (uint32_t)items.size();
            gblocks[3 * g + f] = first[f];
        }
        gshare[g] = packed ? share : 0;
        if (packed) gblocks[3 * g + EXT_FLAT] = (uint32_t)ceil_div((uint64_t)first[EXT_FLAT], (uint64_t)share);
    }
    // one upload: table offsets, capacities, items
    const size_t items_at = 8 * (2 * (size_t)nb + 1), up_bytes = items_at + items.size() * sizeof(ext_item);
    std::vector<uint8_t> up(up_bytes);
    std::memcpy(up.data(), toff.data(), 8 * ((size_t)nb + 1));
    std::memcpy(up.data() + 8 * ((size_t)nb + 1), tcap.data(), 8 * (size_t)nb);
    std::memcpy(up.data() + items_at, items.data(), items.size() * sizeof(ext_item));
    uint8_t* d_up = A.alloc<uint8_t>(up_bytes);
    CDBG_CUDA(cudaMemcpyAsync(d_up, up.data(), up_bytes, cudaMemcpyHostToDevice, st));
    uint64_t const* d_toff = reinterpret_cast<uint64_t const*>(d_up);
    uint64_t const* d_tcap = d_toff + nb + 1;
    ext_item const* d_items = reinterpret_cast<ext_item const*>(d_up + items_at);
    slot_t<K>* slots = A.alloc<slot_t<K>>(Tmax + 1);
    // record of each occurrence block's first occurrence (k_insert, k_number)
    const uint64_t nblk = ceil_div(nocc, (uint64_t)OCC_BLOCK);
    uint32_t* blk_rec = A.alloc<uint32_t>(nblk + 1);
    k_block_records<<<grid(nrec, 256), 256, 0, st>>>(R.occ, R0, nrec, O0, nblk, blk_rec);
    CDBG_CHECK_LAUNCH();
    uint2* fw = A.alloc<uint2>(ceil_div(nocc, 32) + 1);  // first occurrences, by word (node_of)
    // node arrays, sized for the worst case (every occurrence a distinct
    // k-mer): the groups number their nodes on the device, without a host
    // round trip per group
    K* n_key = A.alloc<K>(nocc);
    uint8_t* n_meta = A.alloc<uint8_t>(nocc);
    uint32_t* n_rec = A.alloc<uint32_t>(nocc);
    uint8_t* n_mask = A.alloc<uint8_t>(nocc);
    uint32_t* link = A.alloc<uint32_t>(2 * nocc);
    // (node, record) pairs of multi-record k-mers: at most one per occurrence
    uint32_t* pnode = A.alloc<uint32_t>(nocc);
    uint32_t* prec = A.alloc<uint32_t>(nocc);
    // look-back state of every group's numbering, zeroed once
    constexpr uint64_t NB_TILE = (uint64_t)NB_ROUNDS * 256;
    std::vector<uint64_t> gtile(ng + 1, 0);
    for (size_t g = 0; g < ng; ++g) {
        const uint64_t t0 = bocc[b0 + gb[g]] - O0, t1 = bocc[b0 + gb[g + 1]] - O0;
        gtile[g + 1] = gtile[g] + (t1 > t0 ? ceil_div(t1 - t0 / OCC_BLOCK * OCC_BLOCK, NB_TILE) : 0);
    }
    // zeroed together: look-back status, the node and pair counts so far
    // (alternating by group), tile counters
    // and the number of path ends
    uint32_t* ends = A.alloc<uint32_t>(nocc);
    unsigned long long* nb_status = A.alloc<unsigned long long>(gtile[ng] + 5 + (ng + 1) / 2 + 1);
    unsigned long long* ncnt = nb_status + gtile[ng];
    unsigned long long* nends = ncnt + 4;
    uint32_t* nb_counter = reinterpret_cast<uint32_t*>(ncnt + 5);
    CDBG_CUDA(cudaMemsetAsync(nb_status, 0, 8 * (gtile[ng] + 5 + (ng + 1) / 2 + 1), st));
    for (size_t g = 0; g < ng; ++g) {
        const uint32_t g0 = gb[g], g1 = gb[g + 1];
        const uint64_t t0 = bocc[b0 + g0] - O0, tn = bocc[b0 + g1] - bocc[b0 + g0];
        const uint64_t Tg = toff[g1] - toff[g0];
        if (tn == 0) {
            // no occurrence: the next group starts from the same counts
            k_copy_u64x2<<<1, 1, 0, st>>>(ncnt + 2 * (g & 1), ncnt + 2 * ((g + 1) & 1));
            CDBG_CHECK_LAUNCH();
            continue;
        }
        tables<K> TG;
        TG.slots = slots;
        TG.tab_off = d_toff + g0;
        TG.tab_cap = d_tcap + g0;
        TG.b0 = b0 + g0;
        TG.off0 = toff[g0];
        {
            CDBG_PROF("k_init_tables", st);
            k_init_tables<K><<<grid(Tg, 256), 256, 0, st>>>(Tg, slots);
        }
        CDBG_CHECK_LAUNCH();
        {
            CDBG_PROF("k_insert", st);
            k_insert<K><<<(unsigned)(ceil_div(t0 + tn, OCC_BLOCK) - t0 / OCC_BLOCK), OCC_BLOCK, 0, st>>>(
                R, TG, R0, nrec, O0, t0, t0 + tn, k, nblk, blk_rec, occ_slot, d_err);
        }
        CDBG_CHECK_LAUNCH();
        unsigned long long* nbase = ncnt + 2 * (g & 1);
        unsigned long long* nnext = ncnt + 2 * ((g + 1) & 1);
        {
            CDBG_PROF("k_number", st);
            k_number<K><<<(unsigned)(gtile[g + 1] - gtile[g]), 256, 0, st>>>(
                t0 / OCC_BLOCK * OCC_BLOCK, t0, t0 + tn, occ_slot, TG, R.occ, R0, nrec, O0, nblk, blk_rec, nbase,
                nnext, nb_counter + g, nb_status + gtile[g], fw, n_key, n_meta, n_rec, pnode, prec, d_err);
        }
        CDBG_CHECK_LAUNCH();
        {
            CDBG_PROF("k_pair_nodes", st);
            k_pair_nodes<<<(unsigned)std::min<uint64_t>(grid(tn, 256), 148 * 16), 256, 0, st>>>(nbase + 1, nnext + 1,
                                                                                               fw, pnode);
        }
        CDBG_CHECK_LAUNCH();
        {
            CDBG_PROF("k_ext_mask", st);  // (its three forms)
            constexpr int smem = EXT_FILTER_WORDS * 4;
            CDBG_CUDA(cudaFuncSetAttribute(k_ext_mask<K, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            if constexpr (sizeof(K) == 16)
                CDBG_CUDA(cudaFuncSetAttribute(k_ext_mask<K, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * smem));
            const uint32_t t1 = (uint32_t)(t0 + tn);
            auto launch = [&](auto kern, int c, int threads, int sm, auto... share) {
                const uint32_t a = gitem[3 * g + c], n = gitem[3 * g + c + 1] - a - 1;
                if (gblocks[3 * g + c])
                    kern<<<gblocks[3 * g + c], threads, sm, st>>>(d_items + a, n, share..., t1, nnext, TG, n_key, k, fw,
                                                                  n_mask, link);
            };
            launch(k_ext_mask<K, false>, EXT_FILTER, ext_cfg<K>::THREADS, smem);
            if constexpr (sizeof(K) == 16) launch(k_ext_mask<K, true>, EXT_WIDE, 1024, 2 * smem);
            if (gshare[g])
                launch(k_ext_flat<K, true>, EXT_FLAT, 256, 0, gshare[g]);
            else
                launch(k_ext_flat<K, false>, EXT_FLAT, 256, 0, 0u);
        }
        CDBG_CHECK_LAUNCH();
        {
            CDBG_PROF("k_links", st);
            const unsigned blocks = (unsigned)std::min<uint64_t>(grid(tn, 256 * LINKS_PER), 148 * 16);
            if (k & 1u)
                k_links<false><<<blocks, 256, 0, st>>>(nbase, nnext, n_mask, link, ends, nends);
            else
                k_links<true><<<blocks, 256, 0, st>>>(nbase, nnext, n_mask, link, ends, nends);
        }
        CDBG_CHECK_LAUNCH();
    }
    uint64_t counts[2];  // nodes, pairs
    uint64_t n_ends = 0;
    uint32_t derr = 0;
    mail_reader(st).add(counts, ncnt + 2 * (ng & 1), 16).add(&n_ends, nends).add(&derr, d_err).wait();
    const uint64_t D = counts[0], npairs = counts[1];
    if (D >= (1ull << 31)) throw std::runtime_error("too many distinct k-mers in one bucket batch");
    if (derr) check_device_error_word(d_err, st, "k-mer table insert");
    // zeroed together: selections over the pairs, records, nodes and fragments,
    // heavy-record flags, the chains' seed lengths and covered flags, counts
    zero_block Z(3 * zero_block::select_words(npairs) + zero_block::select_words(nrec) +
                     zero_block::select_words(D) + zero_block::tiles(D, prim::SEL_TILE) + nrec / 2 + D / 2 + D / 8 + 16,
                 A, st);
    // ---- multi-record k-mers, from their (node, record) pairs
    uint64_t M = 0;
    uint32_t* mnode = nullptr;
    uint64_t* moff = nullptr;
    uint32_t* urec = nullptr;
    uint32_t* msize = nullptr;
    uint64_t* mhash = nullptr;
    uint64_t* poff = nullptr;
    uint32_t* pool = nullptr;
    uint32_t* mbits = nullptr;
    uint64_t G = 0;              // union groups
    uint32_t* gnode = nullptr;   // first node of each group
    uint64_t* gbeg = nullptr;    // record range of each group
    uint64_t* gend = nullptr;
    uint32_t* mgrp = nullptr;    // group of each multi node
    uint64_t nu = 0;
    if (npairs) {
        // stable by node (records already ascend within a node): the node bits only
        const int node_bits = D > 1 ? 64 - __builtin_clzll(D - 1) : 1;
        prim::radix_sort_pairs<uint32_t, uint32_t>(pnode, prec, npairs, 0, node_bits, A, st, d_err);
        // (arrays sized for the pairs when those are few, else for the counts)
        select_ws wk = Z.select(npairs), wh = Z.select(npairs);
        urec = A.alloc<uint32_t>(npairs);
        mnode = A.alloc<uint32_t>(npairs);
        moff = A.alloc<uint64_t>(npairs + 1);
        {
            CDBG_PROF("k_multi_index", st);
            k_multi_index<<<(unsigned)wk.ntiles, 256, 0, st>>>(npairs, pnode, prec, wk, wh, urec, mnode, moff, n_rec,
                                                               d_err);
        }
        CDBG_CHECK_LAUNCH();
        mail_reader(st).add(&nu, wk.total).add(&M, wh.total).wait();
        // one union per run of multi nodes with the same owning records
        gnode = A.alloc<uint32_t>(M);
        gbeg = A.alloc<uint64_t>(M);
        gend = A.alloc<uint64_t>(M);
        mgrp = A.alloc<uint32_t>(M);
    }
    // ---- counts the host needs next: union groups, heavy records (with a
    // bitmap: unions of at least that many colors), records used as color sets
    const uint32_t nw = (C + 31) / 32;
    // Unless the caller names a threshold: 64 colors; where a bitmap is no longer
    // than a list of 8 colors, 8 (unions of 90 genomes in skewed buckets 2.4 ms
    // instead of 3.1; of 60 genomes of the small kind 0.29 instead of 0.40;
    // thresholds 4 and 16 within 10% of it).
    const uint32_t heavy = p.heavy_colors ? p.heavy_colors : nw <= 8 ? 8 : 64;
    const bool may_heavy = M && p.union_bitmaps && C >= heavy;
    uint32_t* hflag = nullptr;
    uint64_t* hpos = nullptr;
    select_ws wg{}, wr = Z.select(nrec);
    if (M) {
        wg = Z.select(M);
        {
            uint32_t* same = A.alloc<uint32_t>(ceil_div(M, (uint64_t)32));
            CDBG_PROF("k_multi_groups", st);  // (both)
            k_multi_same<<<grid(M, 256), 256, 0, st>>>(M, moff, urec, same);
            CDBG_CHECK_LAUNCH();
            k_multi_groups<<<(unsigned)wg.ntiles, 256, 0, st>>>(M, same, moff, mnode, wg, gnode, gbeg, gend, mgrp,
                                                                d_err);
        }
        CDBG_CHECK_LAUNCH();
    }
    if (may_heavy) {
        hflag = Z.take<uint32_t>(nrec);
        hpos = A.alloc<uint64_t>(nrec + 1);
        k_heavy_flags<<<grid(nu, 256), 256, 0, st>>>(nu, urec, R.col_off, (uint32_t)R0, heavy, hflag);
        CDBG_CHECK_LAUNCH();
        prim::exclusive_scan<uint32_t, uint64_t>(hflag, hpos, nrec, A, st, hpos + nrec);
    }
    uint32_t* rec_first = A.alloc<uint32_t>(nrec);
    CDBG_CUDA(cudaMemsetAsync(rec_first, 0xff, 4 * nrec, st));
    {
        CDBG_PROF("k_rec_first", st);
        k_rec_first<<<grid(D, 1024), 256, 0, st>>>(D, n_rec, (uint32_t)R0, rec_first);
    }
    CDBG_CHECK_LAUNCH();
    // candidates: used records, then union groups
    cand_view cv;
    cv.kind_id = A.alloc<uint32_t>(nrec + M + 1);
    cv.first = A.alloc<uint32_t>(nrec + M + 1);
    cv.hash = A.alloc<uint64_t>(nrec + M + 1);
    uint32_t* rec_cand = A.alloc<uint32_t>(nrec);
    {
        CDBG_PROF("k_cand_records", st);
        k_cand_records<<<(unsigned)wr.ntiles, 256, 0, st>>>(nrec, (uint32_t)R0, rec_first, wr, d_rhash, cv, rec_cand,
                                                            d_err);
    }
    CDBG_CHECK_LAUNCH();
    uint64_t nrc = 0, nheavy = 0;
    {
        mail_reader mr(st);
        mr.add(&nrc, wr.total);
        if (M) mr.add(&G, wg.total);
        if (may_heavy) mr.add(&nheavy, hpos + nrec);
        mr.wait();
    }
    if (M) {
        msize = A.alloc<uint32_t>(G);
        mhash = A.alloc<uint64_t>(G);
        int wpb = (int)std::max<uint64_t>(1, std::min<uint64_t>(8, (96 * 1024) / (4ull * nw)));
        const size_t shm = (size_t)wpb * nw * 4;
        if (p.union_bitmaps) {
            // heavy records used by multi-record nodes get a bitmap once
            uint32_t* rbits = A.alloc<uint32_t>(nheavy * nw + 1);
            if (shm > 48 * 1024)
                CDBG_CUDA(cudaFuncSetAttribute(k_heavy_bitmaps, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
            if (nheavy) {
                CDBG_PROF("k_heavy_bitmaps", st);
                k_heavy_bitmaps<<<grid(ceil_div(nrec, 32), wpb), wpb * 32, shm, st>>>(nrec, hflag, hpos, (uint32_t)R0, R.col_off,
                                                                        R.colors, nw, rbits);
            }
            CDBG_CHECK_LAUNCH();
            mbits = A.alloc<uint32_t>(G * nw + 1);
            {
                CDBG_PROF("k_union", st);
                auto launch = [&](auto kern, int gw) {
                    // blocks of as many warps as their groups' bitmaps leave room for
                    const int groups = 32 / gw;
                    const int wpu = (int)std::max<uint64_t>(1, std::min<uint64_t>(8, (96 * 1024) / (4ull * nw * groups)));
                    const size_t sh = (size_t)wpu * groups * nw * 4;
                    if (sh > 48 * 1024)
                        CDBG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh));
                    kern<<<grid(G, wpu * groups), wpu * 32, sh, st>>>(G, gbeg, gend, urec, R.col_off, R.colors,
                                                                      (uint32_t)R0, hflag, hpos, rbits, nw, mbits,
                                                                      msize, mhash);
                };
                // groups no wider than the bitmap's words keep their lanes
                // busy (figures at the kernel)
                if (nw <= 8)
                    launch(k_union_bm<1, 8>, 8);
                else if (nw <= 16)
                    launch(k_union_bm<1, 16>, 16);
                else if (nw <= 32)
                    launch(k_union_bm<1, 32>, 32);
                else if (nw <= 64)
                    launch(k_union_bm<2, 32>, 32);
                else if (nw <= 128)
                    launch(k_union_bm<4, 32>, 32);
                else if (nw <= 256)
                    launch(k_union_bm<8, 32>, 32);
                else
                    throw std::runtime_error("bitmap unions need at most 8192 colors");
            }
            CDBG_CHECK_LAUNCH();
        } else {
            if (shm > 48 * 1024) {
                CDBG_CUDA(cudaFuncSetAttribute(k_union<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
                CDBG_CUDA(cudaFuncSetAttribute(k_union<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
            }
            {
                CDBG_PROF("k_union", st);
                k_union<false><<<grid(G, wpb), wpb * 32, shm, st>>>(G, gbeg, gend, urec, R.col_off, R.colors, C,
                                                                     msize, mhash, nullptr, nullptr);
            }
            CDBG_CHECK_LAUNCH();
            poff = A.alloc<uint64_t>(G + 1);
            prim::exclusive_scan<uint32_t, uint64_t>(msize, poff, G, A, st, poff + G);
            const uint64_t ptot = read_dev(poff + G, st);
            pool = A.alloc<uint32_t>(ptot + 1);
            {
                CDBG_PROF("k_union", st);
                k_union<true><<<grid(G, wpb), wpb * 32, shm, st>>>(G, gbeg, gend, urec, R.col_off, R.colors, C,
                                                                    msize, mhash, poff, pool);
            }
            CDBG_CHECK_LAUNCH();
        }
    }
    out.n_multi += M;
    const uint64_t nc = nrc + G;
    if (G) {
        k_cand_multi<<<grid(G, 256), 256, 0, st>>>(G, nrc, gnode, mhash, cv);
        CDBG_CHECK_LAUNCH();
    }
    list_src L{R.col_off, R.colors, poff, pool, msize, mbits, nw};
    uint32_t* cid = A.alloc<uint32_t>(nc + 1);
    unsigned long long* ints = Z.take<unsigned long long>(1);  // colors in the new classes
    if (nc) {
        // 1. group candidates with equal color sets (sort by set hash, then
        //    compare raw lists inside equal-hash runs)
        uint64_t* skey = A.alloc<uint64_t>(nc);
        uint32_t* sidx = A.alloc<uint32_t>(nc);
        CDBG_CUDA(cudaMemcpyAsync(skey, cv.hash, 8 * nc, cudaMemcpyDeviceToDevice, st));
        prim::sort_pairs_u64_exact<uint32_t>(skey, sidx, nc, A, st, d_err, true);
        // zeroed together: selections of runs, representatives (twice) and new
        // ones, the runs' collision flags, counts
        zero_block Y(4 * zero_block::select_words(nc) + nc / 2 + 8, A, st);
        uint32_t* run = A.alloc<uint32_t>(nc);
        uint32_t* run_start = A.alloc<uint32_t>(nc);
        uint32_t* rep = A.alloc<uint32_t>(nc);
        uint32_t* rep_first = A.alloc<uint32_t>(nc);
        select_ws wq = Y.select(nc), wp = Y.select(nc), wp2 = Y.select(nc), wn = Y.select(nc);
        uint32_t* collided = Y.take<uint32_t>(nc);
        uint32_t* any_collided = Y.take<uint32_t>(1);
        {
            CDBG_PROF("k_hash_runs", st);
            k_hash_runs<<<(unsigned)wq.ntiles, 256, 0, st>>>(nc, skey, wq, run, run_start, rep_first, d_err);
        }
        CDBG_CHECK_LAUNCH();
        {
            CDBG_PROF("k_member_match", st);
            k_member_match_raw<<<grid(nc, 256), 256, 0, st>>>(nc, run, run_start, sidx, cv, L, rep, rep_first, collided,
                                                               any_collided);
        }
        CDBG_CHECK_LAUNCH();
        // 2. representatives: compact, encode, look up in the dictionary
        cand_view rv;
        rv.kind_id = A.alloc<uint32_t>(nc + 1);
        rv.first = A.alloc<uint32_t>(nc + 1);
        rv.hash = A.alloc<uint64_t>(nc + 1);
        uint32_t* rep_index = A.alloc<uint32_t>(nc);
        auto compact_reps = [&](select_ws w) {
            CDBG_PROF("k_rep_compact", st);
            k_rep_compact<<<(unsigned)w.ntiles, 256, 0, st>>>(nc, rep, w, cv, rep_first, rv, rep_index, d_err);
            CDBG_CHECK_LAUNCH();
        };
        compact_reps(wp);
        uint64_t nr = 0, nruns = 0;
        uint32_t any = 0;
        mail_reader(st).add(&nr, wp.total).add(&nruns, wq.total).add(&any, any_collided).wait();
        if (any) {
            // equal hashes of different sets: those runs grouped exactly
            k_group_collided_raw<<<grid(nruns, 128), 128, 0, st>>>(nruns, collided, run_start, nc, sidx, cv, L, rep,
                                                                   rep_first);
            CDBG_CHECK_LAUNCH();
            compact_reps(wp2);
            nr = read_dev(wp2.total, st);
        }
        uint64_t* cbits = A.alloc<uint64_t>(nr);
        // lanes per candidate: one per bitmap word, 8 at least
        auto encode = [&](auto enc, uint32_t const* order, uint64_t* nbits, uint64_t const* boff, uint64_t* words) {
            constexpr bool ENC = decltype(enc)::value;
            auto launch = [&](auto kern, int groups) {
                const uint64_t wbytes = 4ull * nw * groups;  // bitmaps of a warp
                const int wpb = (int)std::max<uint64_t>(1, std::min<uint64_t>(8, (96 * 1024) / wbytes));
                const size_t shm = wpb * wbytes;
                if (shm > 48 * 1024)
                    CDBG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
                CDBG_PROF("k_encode", st);
                kern<<<grid(ceil_div(nr, 32), wpb), wpb * 32, shm, st>>>(nr, order, rv, L, C, nbits, boff, words);
                CDBG_CHECK_LAUNCH();
            };
            if (nw <= 8)
                launch(k_encode<ENC, 8>, 4);
            else if (nw <= 16)
                launch(k_encode<ENC, 16>, 2);
            else
                launch(k_encode<ENC, 32>, 1);
        };
        uint32_t* rcid = A.alloc<uint32_t>(nr + 1);
        uint32_t* rcand = A.alloc<uint32_t>(nr);
        const int node_bits = D > 1 ? 64 - __builtin_clzll(D - 1) : 1;
        const uint64_t base = dict.n;
        uint64_t nnew = nr, badd = 0;
        auto room = [&](uint64_t classes, uint64_t words) {
            if (p.copy_st && (dict.bit_off.cap < classes + 1 || dict.words.cap < words)) {
                // growing frees the old arrays: after the host copies that read them
                CDBG_CUDA(cudaEventRecord(p.copy_ev, p.copy_st));
                CDBG_CUDA(cudaStreamWaitEvent(st, p.copy_ev, 0));
            }
            dict.cls_hash.reserve(classes, st);
            dict.bit_off.reserve(classes + 1, st);
            dict.words.reserve(words, st, true);
        };
        auto new_classes = [&](uint64_t const* cb, uint64_t* nbits) {
            CDBG_PROF("k_new_classes", st);
            k_new_classes<<<grid(nnew, 256), 256, 0, st>>>(nnew, rcand, rv, L, cb, nbits, dict.cls_hash.p + base, base,
                                                           rcid, ints);
            CDBG_CHECK_LAUNCH();
        };
        if (base == 0) {
            // an empty dictionary (the first batch): every representative is a new
            // class, encoded where it stays, in order of first appearance
            prim::radix_sort_pairs<uint32_t, uint32_t>(rv.first, rcand, nr, 0, node_bits, A, st, d_err, true);
            room(nr, 0);
            new_classes(nullptr, nullptr);
            encode(std::false_type{}, rcand, cbits, nullptr, nullptr);
            prim::exclusive_scan<uint64_t, uint64_t>(cbits, dict.bit_off.p, nr, A, st, dict.bit_off.p + nr);
            badd = read_dev(dict.bit_off.p + nr, st);
            room(nr, (badd + 63) / 64 + 4);
            encode(std::true_type{}, rcand, nullptr, dict.bit_off.p, dict.words.p);
        } else {
            // 3. the dictionary is asked by encoding; the classes it does not hold
            // are new, in order of first appearance
            uint64_t* cb = A.alloc<uint64_t>(nr + 1);
            encode(std::false_type{}, nullptr, cbits, nullptr, nullptr);
            prim::exclusive_scan<uint64_t, uint64_t>(cbits, cb, nr, A, st, cb + nr);
            const uint64_t ctot = read_dev(cb + nr, st);
            const uint64_t cwn = ctot / 64 + 4;
            uint64_t* cw = A.alloc<uint64_t>(cwn);
            CDBG_CUDA(cudaMemsetAsync(cw, 0, 8 * cwn, st));
            encode(std::true_type{}, nullptr, nullptr, cb, cw);
            dict.ensure_table(st, d_err);
            {
                CDBG_PROF("k_dict_lookup", st);
                k_dict_lookup<<<grid(nr, 256), 256, 0, st>>>(nr, rv, cw, cb, dict.view(), rcid);
            }
            CDBG_CHECK_LAUNCH();
            uint32_t* rkey = A.alloc<uint32_t>(nr);
            wn.ntiles = zero_block::tiles(nr, prim::SEL_TILE);
            {
                CDBG_PROF("k_new_reps", st);
                k_new_reps<<<(unsigned)wn.ntiles, 256, 0, st>>>(nr, rcid, wn, rv, rkey, rcand, d_err);
            }
            CDBG_CHECK_LAUNCH();
            nnew = read_dev(wn.total, st);
            if (nnew) {
                prim::radix_sort_pairs<uint32_t, uint32_t>(rkey, rcand, nnew, 0, node_bits, A, st, d_err);
                uint64_t* nbits = A.alloc<uint64_t>(nnew);
                uint64_t* boff = A.alloc<uint64_t>(nnew + 1);
                room(base + nnew, 0);
                new_classes(cb, nbits);
                prim::exclusive_scan<uint64_t, uint64_t>(nbits, boff, nnew, A, st, boff + nnew);
                badd = read_dev(boff + nnew, st);
                add_offsets(boff, nnew + 1, dict.nbits, boff, st);  // absolute bit offsets
                room(base + nnew, (dict.nbits + badd + 63) / 64 + 4);
                CDBG_CUDA(cudaMemcpyAsync(dict.bit_off.p + base, boff, 8 * (nnew + 1), cudaMemcpyDeviceToDevice, st));
                {
                    CDBG_PROF("k_append_bits", st);
                    k_append_bits<<<grid(nnew, 8), 256, 0, st>>>(nnew, rcand, cw, cb, boff, dict.words.p);
                }
                CDBG_CHECK_LAUNCH();
            }
        }
        dict.n = base + nnew;
        dict.cls_hash.n = dict.n;
        dict.bit_off.n = dict.n + 1;
        dict.nbits += badd;
        dict.words.n = (dict.nbits + 63) / 64;
        // 4. every candidate takes its representative's class id
        k_cand_cid<<<grid(nc, 256), 256, 0, st>>>(nc, rep, rep_index, rcid, cid);
        CDBG_CHECK_LAUNCH();
    }
    // ---- node class ids
    uint32_t* n_cid = A.alloc<uint32_t>(D);
    {
        CDBG_PROF("k_node_cid", st);
        k_node_cid<<<grid(D, 1024), 256, 0, st>>>(D, n_rec, (uint32_t)R0, rec_cand, nrc, mgrp, cid, n_cid);
    }
    CDBG_CHECK_LAUNCH();
    // ---- chains (extension masks and links were made with the tables)
    chain_ws W;
    W.link = link;
    W.meta = n_meta;
    W.mask = n_mask;
    W.ch_node = A.alloc<uint32_t>(D);
    W.ch_rc = A.alloc<uint8_t>(D);
    W.ch_ord = A.alloc<unsigned long long>(D);
    W.ch_vis = A.alloc<uint8_t>(D);
    W.fe = A.alloc<uint32_t>(D);
    W.seed_start = A.alloc<uint32_t>(D);
    W.seed_len = Z.take<uint32_t>(D);
    W.seed_info = A.alloc<uint32_t>(D);
    W.covered = Z.take<uint8_t>(D);
    W.n_cid = n_cid;
    W.cursor = Z.take<unsigned long long>(1);
    W.D = D;
    {
        uint4* heads = A.alloc<uint4>(n_ends + 1);
        unsigned long long* cnt2 = Z.take<unsigned long long>(2);  // heads, nodes on paths
        if (n_ends) {
            CDBG_PROF("k_chain_lead", st);
            k_chain_lead<<<grid(n_ends, 256), 256, 0, st>>>(W, ends, nends, heads, cnt2, d_err);
        }
        CDBG_CHECK_LAUNCH();
        {
            CDBG_PROF("k_chain_paths", st);
            k_chain_paths<<<(unsigned)std::min<uint64_t>(grid(n_ends + 1, 128), 148 * 16), 128, 0, st>>>(W, heads, cnt2);
        }
        CDBG_CHECK_LAUNCH();
        {
            CDBG_PROF("k_chain_cycles", st);
            const unsigned blocks = (unsigned)std::min<uint64_t>(grid(D, 128), 148 * 16);
            k_chain_covered<<<blocks, 128, 0, st>>>(W, cnt2 + 1);
            CDBG_CHECK_LAUNCH();
            k_chain_cycles<<<blocks, 128, 0, st>>>(W, cnt2 + 1, d_err);
        }
        CDBG_CHECK_LAUNCH();
    }
    // ---- fragments, in seed order (offsets and seeds sized for D of them)
    uint32_t* seed_of = A.alloc<uint32_t>(D);
    uint64_t* foff = A.alloc<uint64_t>(D + 1);
    select_ws wseed = Z.select(D);
    unsigned long long* byte_status = Z.take<unsigned long long>(wseed.ntiles);
    unsigned long long* ftot = Z.take<unsigned long long>(3);
    {
        CDBG_PROF("k_seed_list", st);
        k_seed_list<<<(unsigned)wseed.ntiles, 256, 0, st>>>(D, W.seed_len, W.seed_info, k, wseed, byte_status, seed_of,
                                                            foff, ftot, d_err);
    }
    CDBG_CHECK_LAUNCH();
    uint64_t ft[3], new_ints = 0;
    mail_reader(st).add(ft, ftot, 24).add(&new_ints, ints).add(&derr, d_err).wait();
    if (derr) check_device_error_word(d_err, st, "unitig walk");
    const uint64_t nfr = ft[0], fbytes = ft[1], seq_total = ft[2];
    dict.total_integers += new_ints;
    const uint64_t frag_old = dfrag.n;
    uint8_t* fb = nullptr;  // the fragments: scratch on their way to the host, or where the output stays
    if (p.take_frag) {
        fb = A.alloc<uint8_t>(fbytes + 16);
    } else {
        if (p.copy_st && dfrag.n + fbytes + 16 > dfrag.cap) {
            // growing frees the old buffer: after the host copies that read it
            CDBG_CUDA(cudaEventRecord(p.copy_ev, p.copy_st));
            CDBG_CUDA(cudaStreamWaitEvent(st, p.copy_ev, 0));
        }
        dfrag.reserve(dfrag.n + fbytes + 16, st);
        fb = dfrag.p;
    }
    if (nfr) {
        CDBG_PROF("k_frag_write", st);
        k_frag_write<K><<<grid(nfr, FW_THREADS), FW_THREADS, 0, st>>>(nfr, seed_of, W.seed_start, W.seed_len,
                                                                       W.seed_info, W.fe, n_cid, n_key, k, foff,
                                                                       p.take_frag ? 0 : frag_old, fb);
    }
    CDBG_CHECK_LAUNCH();
    out.n_fragments += nfr;
    out.total_seq_bytes += seq_total;
    out.n_occ += nocc;
    out.n_distinct += D;
    if (p.take_frag) {
        check_device_error_word(d_err, st, "phase-2 batch");
        if (fbytes) p.take_frag(p.take_frag_ctx, fb, fbytes);
    } else {
        const uint64_t old_n = frag_old;
        dfrag.n += fbytes;
        if (p.keep_frag_offsets && nfr) {
            dfoff.reserve(dfoff.n + nfr + 1, st);
            add_offsets(foff, nfr, old_n, dfoff.p + dfoff.n, st);
            dfoff.n += nfr;
        }
        if (p.copy_st && p.frag_host && out.frag_host_copied == old_n && dfrag.n <= p.frag_host_cap && fbytes) {
            // this batch's fragments go to the host while the next batch runs
            CDBG_CUDA(cudaEventRecord(p.copy_ev, st));
            CDBG_CUDA(cudaStreamWaitEvent(p.copy_st, p.copy_ev, 0));
            CDBG_CUDA(cudaMemcpyAsync(p.frag_host + old_n, dfrag.p + old_n, fbytes, cudaMemcpyDeviceToHost,
                                      p.copy_st));
            out.frag_host_copied = dfrag.n;
            if (p.on_frag) p.on_frag(p.on_frag_ctx, old_n, fbytes);
        }
    }
    if (!p.take_frag && p.copy_st) {
        // completed class words (all but the one later classes still fill) and
        // class offsets go to the host while the next batch runs
        const uint64_t wdone = dict.nbits / 64;
        const bool words_go = p.words_host && out.words_host_copied < wdone && wdone <= p.words_host_cap;
        const bool offs_go = p.offs_host && out.offs_host_copied < dict.n && dict.n <= p.offs_host_cap;
        if (words_go || offs_go) {
            CDBG_CUDA(cudaEventRecord(p.copy_ev, st));
            CDBG_CUDA(cudaStreamWaitEvent(p.copy_st, p.copy_ev, 0));
        }
        if (words_go) {
            CDBG_CUDA(cudaMemcpyAsync(p.words_host + out.words_host_copied, dict.words.p + out.words_host_copied,
                                      8 * (wdone - out.words_host_copied), cudaMemcpyDeviceToHost, p.copy_st));
            out.words_host_copied = wdone;
        }
        if (offs_go) {
            CDBG_CUDA(cudaMemcpyAsync(p.offs_host + out.offs_host_copied, dict.bit_off.p + out.offs_host_copied,
                                      8 * (dict.n - out.offs_host_copied), cudaMemcpyDeviceToHost, p.copy_st));
            out.offs_host_copied = dict.n;
        }
    }
    out.frag_nbytes += fbytes;
    if (!p.take_frag) check_device_error_word(d_err, st, "phase-2 batch");
    A.release(mark);
}

}  // namespace
}  // namespace cdbg

namespace cdbg {

namespace {
template <typename K>
void run_all(record_set const& rs, phase2_params const& p, dev_arena& A, cudaStream_t st, uint32_t* d_err,
             phase2_result& out) {
    const uint64_t n = rs.n;
    const uint32_t B = rs.B;
    auto mark = A.mark();
    uint64_t* nk = A.alloc<uint64_t>(n + 1);
    uint32_t* rbucket = A.alloc<uint32_t>(n + 1);
    uint64_t* rhash = A.alloc<uint64_t>(n + 1);
    uint64_t* occ = A.alloc<uint64_t>(n + 1);
    if (n) {
        {
            CDBG_PROF("k_rec_prep", st);
            k_rec_prep<<<grid(n, 256), 256, 0, st>>>(n, rs.len, p.k, rs.bucket_start, B, nk, rbucket, rs.col_off,
                                                     rs.colors, rhash);
        }
        CDBG_CHECK_LAUNCH();
    }
    prim::exclusive_scan<uint64_t, uint64_t>(nk, occ, n, A, st, occ + n);
    uint64_t* d_bocc = A.alloc<uint64_t>(B + 1);
    k_gather_u64<<<grid(B + 1, 256), 256, 0, st>>>(B + 1, occ, rs.bucket_start, d_bocc);
    CDBG_CHECK_LAUNCH();
    std::vector<uint64_t> bocc(B + 1), hbstart(B + 1);
    mail_reader(st)
        .add(bocc.data(), d_bocc, 8ull * (B + 1))
        .add(hbstart.data(), rs.bucket_start, 8ull * (B + 1))
        .wait();
    uint64_t budget = p.batch_occ;
    if (budget == 0) {
        int dev = 0;
        CDBG_CUDA(cudaGetDevice(&dev));
        const uint64_t avail = std::min<uint64_t>(device_available(dev) + A.cached_free(), A.headroom());
        // ~200 B of device memory per k-mer occurrence in the batch, worst
        // case; keep 45% of the available memory for outputs and the dictionary
        budget = std::max<uint64_t>(1ull << 22, std::min<uint64_t>(1ull << 28, (uint64_t)(avail * 0.5) / 220));
    }
    rec_view R{rs.start, rs.len, rs.flags, rs.col_off, rs.colors, rbucket, occ, rs.words};
    phase2_state local_state;
    phase2_state& S = out.state ? *out.state : local_state;
    class_dict dict(S);
    if (p.keep_dict) {
        dict.n = S.n;
        dict.nbits = S.nbits;
        dict.total_integers = S.total_integers;
        dict.mask = S.mask;
        dict.tabled = S.tabled;
    } else {
        dict.init(st);
    }
    dvec<uint8_t>& dfrag = S.frag;
    dfrag.n = 0;
    S.frag_off.n = 0;
    uint32_t b = 0;
    while (b < B) {
        const uint32_t s = b;
        uint64_t acc = 0, recs = 0;
        while (b < B) {
            const uint64_t ob = bocc[b + 1] - bocc[b];
            const uint64_t rb = hbstart[b + 1] - hbstart[b];
            if (b > s && (acc + ob > budget || recs + rb > MAX_BATCH_RECORDS)) break;
            acc += ob;
            recs += rb;
            ++b;
        }
        run_batch<K>(rs, R, p, s, b, bocc, A, st, d_err, dict, out, hbstart, rhash, dfrag, S.frag_off);
    }
    // outputs
    S.n = dict.n;
    S.nbits = dict.nbits;
    S.total_integers = dict.total_integers;
    S.mask = dict.mask;
    S.tabled = dict.tabled;
    out.n_classes = dict.n;
    out.nbits = dict.nbits;
    out.total_integers = dict.total_integers;
    const uint64_t nwords = (dict.nbits + 63) / 64;
    if (p.take_frag && p.copy_dict) {
        out.words.resize(nwords);
        out.offsets.resize(dict.n);
        if (nwords)
            CDBG_CUDA(cudaMemcpyAsync(out.words.data(), dict.words.p, 8 * nwords, cudaMemcpyDeviceToHost, st));
        if (dict.n)
            CDBG_CUDA(cudaMemcpyAsync(out.offsets.data(), dict.bit_off.p, 8 * dict.n, cudaMemcpyDeviceToHost, st));
    }
    CDBG_CUDA(cudaStreamSynchronize(st));
    A.release(mark);
    if (!p.take_frag) {
        // outputs stay in the persistent state
        out.d_frag = S.frag.p;
        out.d_words = S.words.p;
        out.d_offsets = S.bit_off.p;
    }
}
}  // namespace

void run_phase2(record_set const& rs, phase2_params const& p, dev_arena& A, cudaStream_t st, uint32_t* d_err,
                phase2_result& out) {
    {
        // keep the caller's persistent storage across the reset
        phase2_state* S = out.state;
        out = phase2_result();
        out.state = S;
    }
    if (!p.take_frag && !out.state) throw std::runtime_error("device-resident phase-2 outputs need persistent storage");
    if (p.k < 2 || p.k > 63) throw std::runtime_error("k must be in [2, 63]");
    if (p.num_colors == 0) throw std::runtime_error("num_colors must be > 0");
    if (rs.n >= (1ull << 31)) throw std::runtime_error("more than 2^31 bucket records in one build");
    phase2_params q = p;
    // bitmaps cost C/8 bytes per multi-record k-mer: lists above 8192 colors
    if (q.num_colors > 8192) q.union_bitmaps = false;
    if (q.k <= 31)
        run_all<uint64_t>(rs, q, A, st, d_err, out);
    else
        run_all<u128>(rs, q, A, st, d_err, out);
}

namespace {
// One value per thread: its l low bits OR-ed into the low vector (a value
// spans at most two words) and its bit in the high vector.
__global__ void k_ef_encode(uint64_t const* __restrict__ offsets, uint64_t nclasses, uint64_t total, uint64_t l,
                            unsigned long long* __restrict__ low, unsigned long long* __restrict__ high) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i > nclasses) return;
    const uint64_t v = i < nclasses ? offsets[i] : total;
    if (l) {
        const uint64_t pos = i * l, lo = v & ((uint64_t(1) << l) - 1);
        atomicOr(&low[pos >> 6], (unsigned long long)(lo << (pos & 63)));
        if ((pos & 63) + l > 64) atomicOr(&low[(pos >> 6) + 1], (unsigned long long)(lo >> (64 - (pos & 63))));
    }
    const uint64_t hp = (v >> l) + i;
    atomicOr(&high[hp >> 6], 1ull << (hp & 63));
}
}  // namespace

void ef_encode(uint64_t const* d_offsets, uint64_t nclasses, uint64_t total_bits, dev_arena& A, cudaStream_t st,
               ef_encoded& out) {
    out = ef_encoded();
    const uint64_t n = nclasses + 1, U = total_bits;
    uint64_t l = 0;
    if (U > n) {
        const uint64_t q = U / n;
        while ((uint64_t(1) << (l + 1)) <= q) ++l;
    }
    out.n = n;
    out.l = l;
    out.high_bits = n + (U >> l) + 1;
    out.low_words = (n * l + 63) / 64;
    out.high_words = (out.high_bits + 63) / 64;
    out.low = A.alloc<uint64_t>(out.low_words + 1);
    out.high = A.alloc<uint64_t>(out.high_words + 1);
    CDBG_CUDA(cudaMemsetAsync(out.low, 0, 8 * (out.low_words + 1), st));
    CDBG_CUDA(cudaMemsetAsync(out.high, 0, 8 * (out.high_words + 1), st));
    {
        CDBG_PROF("k_ef_encode", st);
        k_ef_encode<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d_offsets, nclasses, U, l,
                                                                  (unsigned long long*)out.low,
                                                                  (unsigned long long*)out.high);
    }
    CDBG_CHECK_LAUNCH();
}

}  // namespace cdbg
