// gzip (RFC 1952) / DEFLATE (RFC 1951) decoding on the device, one CTA per
// file, and the FASTA record rules of the reference's reader (kseq, as used by
// seq_reader.hpp:66 and restated by the host reader in host/io.cpp) applied
// to the inflated bytes in place.
//
// The host reader inflates with zlib on the host threads; for collections of
// many files of a few Mbp (the pangenome shape: a file per genome) one warp
// per file on the device is several times faster, the compressed bytes are
// all that cross PCIe, and the decoded sequences are already in HBM for
// phase 1.  Everything here is a decoder written from the two RFCs; nothing
// decides a result the host reader would decide differently: streams this
// decoder does not accept go back to the host reader whole.
//
// Decoder layout (per CTA): warp 0 parses member and block headers, two warps
// build the block's codes and all threads its lookup tables.
// A block's symbols are decoded a window of IF_THREADS x WIN_LANE_BITS bits at
// a time, a sub-window per thread.  Every thread but the first starts at a
// guessed bit; a Huffman stream falls back into step with the true symbol
// boundaries after a few symbols, and threads whose guess was wrong decode
// again from their predecessor's exit until all agree (3 rounds for gzip -1
// genomes, 5 for gzip -6).  The threads then write their symbols at their
// output positions, one literal or distance per output byte -- every byte of a
// match that overlaps itself points before the match -- and every byte of the
// window finds its literal by following distances, independent of the others; a
// source before the window is read from HBM.  A literal/length
// lookup of 11 bits yields up to three literals at once, or a whole match
// length; a distance lookup of 11 bits a whole distance (gzip -1 writes DNA as
// matches of about 4 bytes at a few hundred bytes' distance, whose codes and
// extra bits fit the indexes); codes longer than the tables fall back to a
// canonical decode by length.
//
// Bound: the latency of one thread's dependent lookups, about 60 symbols per
// window of 14 KB.  130 gzip -1 files of 2.4 MB (one per SM): 14.2 ms; symbol by
// symbol with one warp per file 228 ms, windows of one warp per file 58.6 ms.
// Runs (N gaps on one line, short tandem repeats) would follow one match's bytes
// one by one.  Eight files of 2.4 MB, ms at gzip -1 / -6, 1 MB of each one run 12.3 /
// 11.0, all of it 10.1 / 12.0; with the bytes of a match pointing a distance back
// each 36.6 / 480 and 61 / 1263; without the stop at the window's last byte (guesses
// between equal symbols stay out of step) 36.3 / 17.6 and 61 / 32; with a match
// written by its thread alone 12.7 / 17.5 and 11.4 / 32.

#include <cuda_runtime.h>
#include <stdint.h>

#include "inflate.cuh"

namespace cdbg {

namespace {

constexpr uint32_t FULL = 0xffffffffu;
constexpr int LB_LIT = 11;     // literal/length table index bits
constexpr int LB_DIST = 11;    // distance table index bits
constexpr int LB_CLEN = 7;     // code-length code table index bits (its longest code)
constexpr int IF_THREADS = 256;
constexpr int IF_WARPS = IF_THREADS / 32;
// Bits decoded per thread and window: about a dozen symbols of genome data, so
// most guesses are back in step by their sub-window's end; an odd number of
// 32-bit words, so a warp's reads of the staged bits fall into different banks.
constexpr uint32_t WIN_LANE_BITS = 160;
constexpr int WIN_STAGE = 648;  // staged 64-bit words of input
static_assert(IF_THREADS * WIN_LANE_BITS + 63 + 48 + 96 <= 64 * WIN_STAGE, "a window's bits and its last symbols fit");
// Output bytes of a window, at most: a thread's symbols always fit (a match
// takes at least 2 bits), so every window makes progress.
constexpr uint32_t WIN_OUT = 24576;
static_assert((WIN_LANE_BITS / 2 + 1) * 258 <= WIN_OUT, "one thread's symbols fit the window");
// Matches of at least this many bytes are written by the whole CTA: in a long run
// one thread has all of a window's bytes.
constexpr uint32_t LONG_MATCH = 192;
static_assert(WIN_OUT / LONG_MATCH * 2 <= IF_THREADS, "a window's long matches fit cta_state::exits");

// RFC 1951 3.2.5: length codes 257..285 and distance codes 0..29
__constant__ uint16_t c_len_base[29] = {3,  4,  5,  6,  7,  8,  9,  10, 11,  13,  15,  17,  19,  23, 27,
                                        31, 35, 43, 51, 59, 67, 83, 99, 115, 131, 163, 195, 227, 258};
__constant__ uint8_t c_len_extra[29] = {0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 2, 2, 2,
                                        2, 3, 3, 3, 3, 4, 4, 4, 4, 5, 5, 5, 5, 0};
__constant__ uint16_t c_dist_base[30] = {1,   2,   3,   4,   5,   7,    9,    13,   17,   25,   33,   49,   65,    97,    129,
                                         193, 257, 385, 513, 769, 1025, 1537, 2049, 3073, 4097, 6145, 8193, 12289, 16385, 24577};
__constant__ uint8_t c_dist_extra[30] = {0, 0, 0, 0, 1, 1, 2, 2, 3, 3, 4, 4, 5, 5, 6,
                                         6, 7, 7, 8, 8, 9, 9, 10, 10, 11, 11, 12, 12, 13, 13};
// RFC 1951 3.2.7: order of the code-length code lengths
__constant__ uint8_t c_clen_order[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};

// Canonical code (RFC 1951 3.2.2) by length: codes of length l are
// first[l] .. first[l] + cnt[l] - 1, for symbols sym[base[l] ..] in order.
struct code_aux {
    uint16_t cnt[16];
    uint16_t first[16];
    uint16_t base[16];
    uint16_t sym[288];
};

// Header fields and the position, from the parsing warp to the CTA.
struct block_ctl {
    uint64_t bit;      // next bit of the stream
    uint32_t status;   // stream_status
    uint32_t type;     // block type, or BLK_DONE after the stream's last member
    uint32_t last;     // the member's last block
    uint32_t nlit, ndist;
    uint32_t stored;   // bytes of a stored block
    uint32_t member0;  // output position of the member's first byte
};
constexpr uint32_t BLK_DONE = 4;

struct __align__(16) cta_state {
    // literal/length lookups (LB_LIT bits of input): bits 0-4 bits consumed,
    // bits 5-7 kind: 1-3 literals (bytes at bits 8, 16, 24), K_LEN a match
    // length (bits 8-16, extra bits that fit the index already added; bits
    // 17-19 extra bits still to read), K_END end of block, K_BAD no valid
    // symbol, 0 a code longer than the index (decode by length)
    uint32_t lit[1 << LB_LIT];
    // distance lookups (LB_DIST bits): bits 0-4 bits consumed, bits 5-8
    // extra bits still to read, bits 9-24 distance (folded extra added),
    // bits 25-26 kind: 1 valid, 2 no valid distance, 0 decode by length
    uint32_t dist[1 << LB_DIST];
    union {
        struct {  // while tables are built: one symbol per lookup, (length << 9) | symbol
            uint16_t one_l[1 << LB_LIT];
            uint16_t one_d[1 << LB_DIST];
            uint16_t one_c[1 << LB_CLEN];
        };
        // window output: 0x8000 | literal byte, or match distance - 1
        uint16_t ent[WIN_OUT];
    };
    uint64_t stage[WIN_STAGE];  // the window's input bits
    code_aux la, da, ca;
    uint32_t hist[2][16];
    uint8_t lens[320];
    uint32_t exits[IF_THREADS];  // bit after each thread's symbols; then the long matches (start | length << 16, distance)
    uint32_t warp_sum[IF_WARPS];
    uint32_t stop[2];
    uint32_t total, end;  // of a window: bytes, bit after the last symbol
    uint32_t ok[2];
    uint32_t nlong;       // long matches of the window
    block_ctl ctl;
};

constexpr uint32_t K_LEN = 4, K_END = 5, K_BAD = 6;

// Little-endian bit reader over the input (RFC 1951 3.1.1: bits from the
// least significant end of each byte).  All lanes of the parsing warp hold the same state.  The
// buffer above the `nb` valid bits holds either zeros or the input bits that
// follow (a refill ORs the next eight bytes in place, so repeated bytes land
// on identical bits); code that moves `ip` by hand clears it.
struct bit_reader {
    uint8_t const* in;  // 8-byte aligned, readable 32 bytes past `end`
    uint64_t ip;        // byte of bit `nb` of the buffer
    uint64_t end;       // end of this stream's bytes
    uint64_t bb;
    uint32_t nb;
    // afterwards at least 56 bits are buffered (bytes past `end` read as
    // whatever follows; callers check ip against end)
    __device__ __forceinline__ void refill() {
        if (nb < 56) {
            const uint64_t a = ip & ~uint64_t(7);
            const uint32_t sh = (uint32_t)(ip & 7) * 8u;
            const uint64_t w0 = __ldg(reinterpret_cast<unsigned long long const*>(in + a));
            const uint64_t w1 = __ldg(reinterpret_cast<unsigned long long const*>(in + a) + 1);
            const uint64_t v = sh ? (w0 >> sh) | (w1 << (64u - sh)) : w0;
            bb |= v << nb;
            const uint32_t take = (63u - nb) >> 3;
            ip += take;
            nb += 8u * take;
        }
    }
    __device__ __forceinline__ void drop(uint32_t n) {
        bb >>= n;
        nb -= n;
    }
    // n <= 16, at least n bits buffered
    __device__ __forceinline__ uint32_t get(uint32_t n) {
        const uint32_t v = (uint32_t)bb & ((1u << n) - 1u);
        drop(n);
        return v;
    }
    __device__ __forceinline__ bool overrun() const { return ip > end + 8; }
    // first byte not consumed (the buffer holds whole bytes after align())
    __device__ __forceinline__ uint64_t pos() const { return ip - nb / 8; }
    __device__ __forceinline__ void align() { drop(nb & 7u); }
    // continue at byte position p (nothing buffered)
    __device__ __forceinline__ void seek(uint64_t p) {
        ip = p;
        bb = 0;
        nb = 0;
    }
};

// The canonical code with lengths lens[0, n) by length: counts, first codes and
// symbols in order.  Returns false for an over-subscribed set, and for an
// incomplete one unless it is a single code of one bit or no code at all (with
// `strict`, for the code-length code, any incomplete set) -- the sets zlib also
// refuses.  Warp-collective.
__device__ bool build_aux(uint8_t const* lens, int n, code_aux& a, uint32_t* hist, int lane, bool strict) {
    if (lane < 16) hist[lane] = 0;
    __syncwarp();
    for (int s0 = 0; s0 < n; s0 += 32) {
        const int s = s0 + lane;
        const uint32_t l = s < n ? lens[s] : 0u;
        const uint32_t grp = __match_any_sync(FULL, l);
        if (l && lane == __ffs(grp) - 1) hist[l] += __popc(grp);
        __syncwarp();
    }
    int ok = 1;
    if (lane == 0) {
        int left = 1, maxl = 0;
        uint32_t code = 0, idx = 0, prev = 0;
        a.cnt[0] = 0;
        for (int l = 1; l < 16; ++l) {
            const uint32_t c = hist[l];
            left = 2 * left - (int)c;
            if (left < 0) ok = 0;
            code = (code + prev) << 1;
            a.cnt[l] = (uint16_t)c;
            a.first[l] = (uint16_t)code;
            a.base[l] = (uint16_t)idx;
            idx += c;
            prev = c;
            if (c) maxl = l;
        }
        if (left > 0 && (strict || maxl > 1)) ok = 0;
    }
    ok = __shfl_sync(FULL, ok, 0);
    if (!ok) return false;
    if (lane < 16) hist[lane] = 0;
    __syncwarp();
    for (int s0 = 0; s0 < n; s0 += 32) {
        const int s = s0 + lane;
        const uint32_t l = s < n ? lens[s] : 0u;
        const uint32_t grp = __match_any_sync(FULL, l);
        const uint32_t before = l ? hist[l] : 0u;
        const uint32_t rank = before + __popc(grp & ((1u << lane) - 1u));
        __syncwarp();
        if (l) {
            if (lane == __ffs(grp) - 1) hist[l] = before + __popc(grp);
            a.sym[a.base[l] + rank] = (uint16_t)s;
        }
        __syncwarp();
    }
    return true;
}

// Canonical decode of the next bits `bb` by length, codes of at most `maxlen`
// bits: (bits used << 16) | symbol, or -1 for a bit string that starts with no
// such code.
__device__ __forceinline__ int decode_canonical(uint64_t bb, code_aux const& a, int maxlen) {
    uint32_t code = 0;
    for (int len = 1; len <= maxlen; ++len) {
        code = (code << 1) | ((uint32_t)bb & 1u);
        bb >>= 1;
        const uint32_t off = code - a.first[len];
        if (off < a.cnt[len]) return (len << 16) | a.sym[a.base[len] + off];
    }
    return -1;
}
__device__ __noinline__ int decode_slow(uint64_t bb, code_aux const& a) { return decode_canonical(bb, a, 15); }

// One-symbol lookups of `lb` index bits from thread t of `nt` on.
__device__ __forceinline__ void fill_one(uint16_t* tab, int lb, code_aux const& a, uint32_t t, uint32_t nt) {
    for (uint32_t x = t; x < (1u << lb); x += nt) {
        const int r = decode_canonical(x, a, lb);
        tab[x] = r < 0 ? (uint16_t)0 : (uint16_t)(((uint32_t)r >> 16 << 9) | ((uint32_t)r & 511u));
    }
}

// Literal/length lookups from the one-symbol table.  A literal whose code
// leaves room in the index for the next code(s), when those are literals too,
// yields two or three (the bits after a code are the index shifted right by
// its length, upper bits zero, which select the same entry for any code that
// fits); a length code whose extra bits fit in the index comes with them
// added.
__device__ __forceinline__ void pack_litlen(cta_state& w, uint32_t t) {
    for (uint32_t x = t; x < (1u << LB_LIT); x += IF_THREADS) {
        const uint32_t e1 = w.one_l[x];
        const uint32_t l1 = e1 >> 9, s1 = e1 & 511u;
        uint32_t out = 0;
        if (l1 == 0) {
            out = 0;
        } else if (s1 < 256) {
            uint32_t tot = l1, cnt = 1;
            out = s1 << 8;
            const uint32_t e2 = w.one_l[x >> tot];
            const uint32_t l2 = e2 >> 9, s2 = e2 & 511u;
            if (l2 && s2 < 256 && tot + l2 <= (uint32_t)LB_LIT) {
                out |= s2 << 16;
                ++cnt;
                tot += l2;
                const uint32_t e3 = w.one_l[x >> tot];
                const uint32_t l3 = e3 >> 9, s3 = e3 & 511u;
                if (l3 && s3 < 256 && tot + l3 <= (uint32_t)LB_LIT) {
                    out |= s3 << 24;
                    ++cnt;
                    tot += l3;
                }
            }
            out |= (cnt << 5) | tot;
        } else if (s1 == 256) {
            out = (K_END << 5) | l1;
        } else if (s1 <= 285) {
            const uint32_t i = s1 - 257, ex = c_len_extra[i];
            uint32_t len = c_len_base[i], c = l1, rem = ex;
            if (l1 + ex <= (uint32_t)LB_LIT) {
                len += (x >> l1) & ((1u << ex) - 1u);
                c = l1 + ex;
                rem = 0;
            }
            out = (rem << 17) | (len << 8) | (K_LEN << 5) | c;
        } else {
            out = (K_BAD << 5) | l1;
        }
        w.lit[x] = out;
    }
}

// Distance lookups from the one-symbol table.
__device__ __forceinline__ void pack_dist(cta_state& w, uint32_t t) {
    for (uint32_t x = t; x < (1u << LB_DIST); x += IF_THREADS) {
        const uint32_t e1 = w.one_d[x];
        const uint32_t l1 = e1 >> 9, s1 = e1 & 511u;
        uint32_t out = 0;
        if (l1 && s1 < 30) {
            const uint32_t ex = c_dist_extra[s1];
            uint32_t d = c_dist_base[s1], c = l1, rem = ex;
            if (l1 + ex <= (uint32_t)LB_DIST) {
                d += (x >> l1) & ((1u << ex) - 1u);
                c = l1 + ex;
                rem = 0;
            }
            out = (1u << 25) | (d << 9) | (rem << 5) | c;
        } else if (l1) {
            out = (2u << 25) | l1;
        }
        w.dist[x] = out;
    }
}

// One thread's symbols from staged bit `pos` until it reaches `limit`: the bit
// after the last symbol in `pos`, the bytes they stand for in `out`.  Returns
// LANE_MORE, LANE_END after an end-of-block symbol, or LANE_BAD at a bit
// string that is no symbol (or past `bits_end`, the stream's last bit).  With
// WRITE, the symbols' entries go to ent[o ..] and `back` is the bytes of this
// member before the window: a distance past them is LANE_BAD.  A symbol takes
// at most 48 bits, and the stage holds the bits that follow the window.
enum : uint32_t { LANE_MORE = 0, LANE_END = 1, LANE_BAD = 2 };
template <bool WRITE>
__device__ __forceinline__ uint32_t lane_symbols(cta_state& w, uint32_t& pos, uint32_t limit, uint32_t bits_end,
                                                 uint32_t& out, uint32_t o, uint32_t back) {
    uint32_t const* sw = reinterpret_cast<uint32_t const*>(w.stage);
    uint32_t p = pos, n = 0, st = LANE_MORE;
    uint32_t wi = (p >> 5) + 2;
    uint64_t bb = (((uint64_t)sw[wi - 1] << 32) | sw[wi - 2]) >> (p & 31);
    uint32_t nb = 64 - (p & 31);
    auto refill = [&]() {  // afterwards at least 33 bits
        if (nb <= 32) {
            bb |= (uint64_t)sw[wi++] << nb;
            nb += 32;
        }
    };
    auto drop = [&](uint32_t c) {
        bb >>= c;
        nb -= c;
        p += c;
    };
    while (p < limit) {
        if (p > bits_end) {
            st = LANE_BAD;
            break;
        }
        refill();
        const uint32_t e = w.lit[(uint32_t)bb & ((1u << LB_LIT) - 1u)];
        const uint32_t kind = (e >> 5) & 7u;
        uint32_t L;
        if (kind - 1u < 3u) {  // one to three literals
            if (WRITE) {
                w.ent[o + n] = (uint16_t)(0x8000u | ((e >> 8) & 0xffu));
                if (kind > 1) w.ent[o + n + 1] = (uint16_t)(0x8000u | ((e >> 16) & 0xffu));
                if (kind > 2) w.ent[o + n + 2] = (uint16_t)(0x8000u | (e >> 24));
            }
            n += kind;
            drop(e & 31u);
            continue;
        }
        if (kind == K_LEN) {
            drop(e & 31u);
            const uint32_t x = (e >> 17) & 7u;
            L = ((e >> 8) & 511u) + ((uint32_t)bb & ((1u << x) - 1u));
            drop(x);
        } else if (kind == K_END) {
            drop(e & 31u);
            st = LANE_END;
            break;
        } else if (kind == K_BAD) {
            st = LANE_BAD;
            break;
        } else {
            // a code longer than the index
            const int r = decode_slow(bb, w.la);
            if (r < 0) {
                st = LANE_BAD;
                break;
            }
            drop((uint32_t)r >> 16);
            const uint32_t sym = (uint32_t)r & 0xffffu;
            if (sym < 256) {
                if (WRITE) w.ent[o + n] = (uint16_t)(0x8000u | sym);
                ++n;
                continue;
            }
            if (sym == 256) {
                st = LANE_END;
                break;
            }
            if (sym > 285) {
                st = LANE_BAD;
                break;
            }
            const uint32_t x = c_len_extra[sym - 257];
            L = c_len_base[sym - 257] + ((uint32_t)bb & ((1u << x) - 1u));
            drop(x);
        }
        refill();
        const uint32_t de = w.dist[(uint32_t)bb & ((1u << LB_DIST) - 1u)];
        const uint32_t dk = de >> 25;
        uint32_t d, x;
        if (dk == 1) {
            drop(de & 31u);
            d = (de >> 9) & 0xffffu;
            x = (de >> 5) & 15u;
        } else if (dk == 0) {
            const int r = decode_slow(bb, w.da);
            if (r < 0 || (r & 0xffff) >= 30) {
                st = LANE_BAD;
                break;
            }
            drop((uint32_t)r >> 16);
            const uint32_t ds = (uint32_t)r & 0xffffu;
            d = c_dist_base[ds];
            x = c_dist_extra[ds];
        } else {
            st = LANE_BAD;
            break;
        }
        d += (uint32_t)bb & ((1u << x) - 1u);
        drop(x);
        if (WRITE) {
            if (d > back + o + n) {
                st = LANE_BAD;
                break;
            }
            if (L >= LONG_MATCH) {  // by the CTA, after the window's symbols
                const uint32_t at = 2 * atomicAdd(&w.nlong, 1u);
                w.exits[at] = (o + n) | (L << 16);
                w.exits[at + 1] = d;
            } else if (d >= L) {
                for (uint32_t i = 0; i < L; ++i) w.ent[o + n + i] = (uint16_t)(d - 1);
            } else {
                // an overlapping match: all its bytes point before it, byte i at its
                // period's distance (d < 258 here, so at most 514)
                for (uint32_t i = 0, c = 0, q = d; i < L; ++i) {
                    w.ent[o + n + i] = (uint16_t)(q - 1);
                    if (++c == d) {
                        c = 0;
                        q += d;
                    }
                }
            }
        }
        n += L;
    }
    pos = p;
    out = n;
    return st;
}

// The next window of a block's symbols (up to IF_THREADS x WIN_LANE_BITS bits
// from bit `bit`, moved past the symbols taken), written to o[op ..].
// WIN_MORE: the block goes on; WIN_DONE: its end-of-block symbol was the last.
// CTA-collective, with the same arguments.
enum : uint32_t { WIN_MORE = 0, WIN_DONE = 1, WIN_BAD = 2, WIN_OVERFLOW = 3 };
__device__ __forceinline__ uint32_t window_decode(cta_state& w, uint8_t const* in, uint64_t end, uint64_t& bit,
                                                  uint8_t* o, uint32_t cap, uint32_t& op, uint32_t member0) {
    const uint32_t t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    // input bits from the 8-byte word of the first bit on
    const uint64_t a0 = (bit >> 6) * 8;
    const uint32_t ph = (uint32_t)(bit & 63);
    for (uint32_t i = t; i < (uint32_t)WIN_STAGE; i += IF_THREADS) {
        const uint64_t a = a0 + 8ull * i;
        w.stage[i] = a < end + 16 ? __ldg(reinterpret_cast<unsigned long long const*>(in + a)) : 0ull;
    }
    if (t < 2) w.stop[t] = IF_THREADS - 1;
    if (t == 2) w.total = w.nlong = 0;
    __syncthreads();
    // bits of the stream left from a0 on (a window past them is refused)
    const uint64_t left = end > a0 ? (end - a0) * 8 : 0;
    const uint32_t bits_end = left < 0xffffffffull ? (uint32_t)left : 0xffffffffu;
    uint32_t start = ph + t * WIN_LANE_BITS;
    const uint32_t limit = start + WIN_LANE_BITS;
    uint32_t pos = start, n = 0;
    uint32_t st = lane_symbols<false>(w, pos, limit, bits_end, n, 0, 0);
    // Thread 0 started right; each round every thread up to the first that
    // stopped takes its predecessor's exit as its start, so after r rounds
    // threads 0..r are right whatever the guesses were: the loop ends by itself
    // within IF_THREADS rounds.  Thread r adds its bytes when it is known to be
    // right, and the first one past the window's bytes stops the rest: in long
    // runs a few threads fill the window, while guesses between symbols that
    // repeat do not fall into step.
    uint32_t stop = 0;
    bool full = false;
    for (int r = 0; r <= IF_THREADS; ++r) {
        w.exits[t] = pos;
        if ((int)t == r) {
            w.total += n;
            full = w.total > WIN_OUT;
        }
        if (st != LANE_MORE || full) atomicMin(&w.stop[r & 1], t);
        __syncthreads();
        stop = w.stop[r & 1];
        const uint32_t want = t ? w.exits[t - 1] : start;
        const bool stale = t <= stop && want != start;
        if (!__syncthreads_or(stale)) break;
        if (t == 0) w.stop[r & 1] = IF_THREADS - 1;  // for the round after the next
        if (stale) {
            start = pos = want;
            st = lane_symbols<false>(w, pos, limit, bits_end, n, 0, 0);
        }
    }
    // output offsets; threads 0 .. take - 1 are right, complete and within
    // the entry array (a prefix of the threads, by construction)
    uint32_t incl = n;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, incl, s);
        if (lane >= s) incl += y;
    }
    if (lane == 31) w.warp_sum[warp] = incl;
    __syncthreads();
    for (int i = 0; i < warp; ++i) incl += w.warp_sum[i];
    const uint32_t take = (uint32_t)__syncthreads_count(t <= stop && st != LANE_BAD && incl <= WIN_OUT);
    if (take == 0) return WIN_BAD;  // thread 0's first symbol is none (its bytes always fit)
    if (t == take - 1) {
        w.total = incl;
        w.end = pos;
        w.ok[0] = st == LANE_END;
    }
    uint32_t wst = LANE_MORE;
    if (t < take) {
        uint32_t p = start, m;
        wst = lane_symbols<true>(w, p, limit, bits_end, m, incl - n, op - member0);
    }
    if (__syncthreads_or(wst == LANE_BAD)) return WIN_BAD;  // a distance before the member's first byte
    const uint32_t nlong = w.nlong;
    if (nlong) {
        for (uint32_t m = warp; m < nlong; m += IF_WARPS) {
            const uint32_t x = w.exits[2 * m], d = w.exits[2 * m + 1], L = x >> 16;
            uint16_t* en = w.ent + (x & 0xffffu);
            for (uint32_t i = lane; i < L; i += 32) en[i] = (uint16_t)((d >= L ? d : i - i % d + d) - 1);
        }
        __syncthreads();
    }
    const uint32_t total = w.total;
    const bool done = w.ok[0] != 0;
    if ((uint64_t)op + total > cap) return WIN_OVERFLOW;
    // Every byte follows its match distances back to a literal of the window
    // or to a byte before it, which is in HBM; a thread takes the four bytes of
    // an aligned output word.
    const uint32_t ph4 = op & 3u;  // regions start 16-byte aligned
    for (uint32_t g = t; 4 * g < total + ph4; g += IF_THREADS) {
        uint32_t p[4], e[4];
        const uint32_t j0 = 4 * g - ph4;  // (wraps below 0 in the first word)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            p[u] = j0 + u;
            e[u] = p[u] < total ? w.ent[p[u]] : 0x8000u;
        }
        for (;;) {
            bool more = false;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (e[u] < 0x8000u && p[u] > e[u]) {  // distance e + 1 <= p: a byte of the window
                    p[u] -= e[u] + 1;
                    e[u] = w.ent[p[u]];
                    more = true;
                }
            }
            if (!more) break;
        }
        uint32_t v = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            uint32_t b = e[u] & 0xffu;
            if (e[u] < 0x8000u) b = o[op + p[u] - (e[u] + 1)];
            v |= b << (8 * u);
        }
        if (j0 < total && j0 + 4 <= total) {
            *reinterpret_cast<uint32_t*>(o + op + j0) = v;
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j0 + u < total) o[op + j0 + u] = (uint8_t)(v >> (8 * u));
        }
    }
    op += total;
    bit = a0 * 8 + w.end;
    __syncthreads();  // the entries, the stage and the totals are reused; the bytes are visible to the CTA
    return done ? WIN_DONE : WIN_MORE;
}

// gzip member header (RFC 1952 2.3.1) at a byte boundary.
__device__ bool read_member_header(bit_reader& br) {
    br.refill();
    if (br.get(8) != 0x1f || br.get(8) != 0x8b || br.get(8) != 8) return false;
    const uint32_t flg = br.get(8);
    if (flg & 0xe0u) return false;
    br.refill();
    br.get(16);
    br.get(16);  // MTIME
    br.refill();
    br.get(8);
    br.get(8);  // XFL, OS
    if (flg & 4u) {  // FEXTRA
        const uint32_t xlen = br.get(16);
        const uint64_t p = br.pos() + xlen;
        br.seek(p);
        if (br.overrun()) return false;
    }
    for (uint32_t bit = 8; bit <= 16; bit <<= 1) {  // FNAME, FCOMMENT: zero-terminated
        if (!(flg & bit)) continue;
        for (;;) {
            br.refill();
            if (br.overrun()) return false;
            if (br.get(8) == 0) break;
        }
    }
    if (flg & 2u) {  // FHCRC
        br.refill();
        br.get(16);
    }
    return !br.overrun();
}

// The next block header from bit ctl.bit on -- after the member header when
// `member_start`, after the trailer checks of a member's last block and the
// next member's header when `trailer` -- into ctl and the code lengths.  `op`
// is the output position.  Warp-collective (the parsing warp).
__device__ __forceinline__ void parse_block_header(cta_state& w, uint8_t const* in, uint64_t end, bool member_start,
                                                   bool trailer, uint32_t op, int lane) {
    block_ctl& c = w.ctl;
    bit_reader br{in, 0, end, 0, 0};
    br.seek(c.bit >> 3);
    br.refill();
    br.drop((uint32_t)(c.bit & 7));
    uint32_t st = STREAM_OK, type = BLK_DONE, last = 0, nlit = 0, ndist = 0, stored = 0;
    uint32_t member0 = c.member0;
    __syncwarp();  // every lane has read ctl
    do {
        if (trailer) {
            // trailer: CRC-32 (not checked here) and ISIZE = member size mod 2^32
            br.align();
            br.refill();
            br.get(16);
            br.get(16);
            br.refill();
            const uint32_t lo = br.get(16), isize = lo | (br.get(16) << 16);
            if (br.overrun() || isize != op - member0) {
                st = STREAM_BAD;
                break;
            }
            const uint64_t p = br.pos();
            if (p > br.end) {
                st = STREAM_BAD;
                break;
            }
            if (p == br.end) break;  // BLK_DONE
            // another member follows (anything else fails its header check)
            br.seek(p);
        }
        if (member_start || trailer) {
            if (!read_member_header(br)) {
                st = STREAM_BAD;
                break;
            }
            member0 = op;
        }
        br.refill();
        if (br.overrun()) {
            st = STREAM_BAD;
            break;
        }
        last = br.get(1);
        type = br.get(2);
        if (type == 0) {
            // stored: LEN, NLEN at the next byte boundary, then LEN bytes
            br.align();
            stored = br.get(16);
            const uint32_t nlen = br.get(16);
            if ((stored ^ 0xffffu) != nlen || br.pos() + stored > br.end) st = STREAM_BAD;
        } else if (type == 1) {
            // fixed codes (RFC 1951 3.2.6); 32 distance codes of 5 bits
            // (30 and 31 never valid) keep the set complete
            for (int i = lane; i < 288 + 32; i += 32)
                w.lens[i] = i < 144 ? 8 : i < 256 ? 9 : i < 280 ? 7 : i < 288 ? 8 : 5;
            nlit = 288;
            ndist = 32;
        } else if (type == 2) {
            // dynamic codes (RFC 1951 3.2.7)
            nlit = br.get(5) + 257;
            ndist = br.get(5) + 1;
            const uint32_t hclen = br.get(4) + 4;
            if (nlit > 286 || ndist > 30) {
                st = STREAM_BAD;
                break;
            }
            if (lane < 19) w.lens[lane] = 0;
            __syncwarp();
            for (uint32_t i = 0; i < hclen; ++i) {
                br.refill();
                const uint32_t v = br.get(3);
                if (lane == 0) w.lens[c_clen_order[i]] = (uint8_t)v;
            }
            __syncwarp();
            if (!build_aux(w.lens, 19, w.ca, w.hist[0], lane, true)) {
                st = STREAM_BAD;
                break;
            }
            __syncwarp();
            fill_one(w.one_c, LB_CLEN, w.ca, (uint32_t)lane, 32);
            __syncwarp();
            const uint32_t total = nlit + ndist;
            uint32_t n = 0, prev = 0;
            while (n < total) {
                br.refill();
                if (br.overrun()) {
                    st = STREAM_BAD;
                    break;
                }
                const uint32_t e = w.one_c[(uint32_t)br.bb & ((1u << LB_CLEN) - 1u)];
                if (e == 0) {  // no code of this bit string
                    st = STREAM_BAD;
                    break;
                }
                br.drop(e >> 9);
                const uint32_t sym = e & 511u;
                uint32_t rep = 1, val = sym;
                if (sym >= 16) {
                    if (sym == 16) {
                        if (n == 0) {
                            st = STREAM_BAD;
                            break;
                        }
                        val = prev;
                        rep = 3 + br.get(2);
                    } else {
                        val = 0;
                        rep = sym == 17 ? 3 + br.get(3) : 11 + br.get(7);
                    }
                    if (n + rep > total) {
                        st = STREAM_BAD;
                        break;
                    }
                }
                for (uint32_t j = (uint32_t)lane; j < rep; j += 32) w.lens[n + j] = (uint8_t)val;
                prev = val;
                n += rep;
            }
            __syncwarp();
            if (st == STREAM_OK && w.lens[256] == 0) st = STREAM_BAD;
        } else {
            st = STREAM_BAD;
        }
    } while (false);
    if (lane == 0) {
        c.bit = br.ip * 8 - br.nb;
        c.status = st;
        c.type = type;
        c.last = last;
        c.nlit = nlit;
        c.ndist = ndist;
        c.stored = stored;
        c.member0 = member0;
    }
}

__global__ void __launch_bounds__(IF_THREADS) k_inflate(stream_set s) {
    extern __shared__ __align__(16) unsigned char if_raw[];
    cta_state& w = *reinterpret_cast<cta_state*>(if_raw);
    const uint32_t f = blockIdx.x, t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const uint64_t cap64 = s.out_cap[f];
    const uint32_t cap = (uint32_t)(cap64 < 0xfffff000ull ? cap64 : 0xfffff000ull);  // (4 GiB: the host reader)
    uint8_t* o = s.out + s.out_off[f];
    const uint64_t in0 = s.in_off[f], end = in0 + s.in_len[f];
    if (!s.gz[f]) {
        // plain file: copied as is
        const uint64_t n = end - in0;
        uint32_t st = STREAM_OK;
        if (n > cap)
            st = STREAM_OVERFLOW;
        else
            for (uint64_t i = t; i < n; i += IF_THREADS) o[i] = s.in[in0 + i];
        if (t == 0) {
            s.out_len[f] = st == STREAM_OK ? n : 0;
            s.status[f] = st;
        }
        return;
    }
    uint32_t op = 0, st = STREAM_OK;
    uint64_t bit = in0 * 8;
    bool member_start = true, trailer = false;
    if (t == 0) w.ctl.member0 = 0;
    for (;;) {  // blocks
        if (t == 0) w.ctl.bit = bit;
        __syncthreads();
        if (warp == 0) parse_block_header(w, s.in, end, member_start, trailer, op, lane);
        __syncthreads();
        const block_ctl c = w.ctl;
        st = c.status;
        if (st != STREAM_OK || c.type == BLK_DONE) break;
        member_start = false;
        bit = c.bit;
        if (c.type == 0) {
            if ((uint64_t)op + c.stored > cap) {
                st = STREAM_OVERFLOW;
                break;
            }
            const uint64_t p = bit >> 3;
            for (uint32_t i = t; i < c.stored; i += IF_THREADS) o[op + i] = s.in[p + i];
            op += c.stored;
            bit = (p + c.stored) * 8;
            __syncthreads();  // every thread has read ctl
        } else {
            if (warp < 2) {
                const bool lc = warp == 0;
                const bool ok = build_aux(lc ? w.lens : w.lens + c.nlit, (int)(lc ? c.nlit : c.ndist),
                                          lc ? w.la : w.da, w.hist[warp], lane, false);
                if (lane == 0) w.ok[warp] = ok ? 1u : 0u;
            }
            __syncthreads();
            if (!w.ok[0] || !w.ok[1]) {
                st = STREAM_BAD;
                break;
            }
            fill_one(w.one_l, LB_LIT, w.la, t, IF_THREADS);
            fill_one(w.one_d, LB_DIST, w.da, t, IF_THREADS);
            __syncthreads();
            pack_litlen(w, t);
            pack_dist(w, t);
            __syncthreads();
            uint32_t ws = WIN_MORE;
            while (ws == WIN_MORE) ws = window_decode(w, s.in, end, bit, o, cap, op, c.member0);
            if (ws != WIN_DONE) {
                st = ws == WIN_OVERFLOW ? STREAM_OVERFLOW : STREAM_BAD;
                break;
            }
        }
        trailer = c.last != 0;
    }
    if (t == 0) {
        s.out_len[f] = st == STREAM_OK ? op : 0;
        s.status[f] = st;
    }
}

// ------------------------------------------------------------ FASTA records
constexpr int FC_THREADS = 256;
constexpr uint32_t FC_CHUNK = FC_THREADS * 16;  // bytes per round
enum : uint32_t { FS_NONE = 0, FS_SEQ = 1, FS_HDR = 2, FS_FASTQ = 3 };

// Right-most event wins: inclusive scan over the CTA of `v` (FS_NONE = no
// event); returns this thread's exclusive value (`carry` for thread 0) and
// the chunk's last state in *last.
__device__ __forceinline__ uint32_t last_event_scan(uint32_t v, uint32_t carry, uint32_t* sw, uint32_t* last) {
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, o);
        if (lane >= o && x == FS_NONE) x = y;
    }
    if (lane == 31) sw[wi] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t c = carry;
        for (int i = 0; i < FC_THREADS / 32; ++i) {
            const uint32_t t = sw[i];
            sw[i] = c;  // exclusive state entering warp i
            if (t != FS_NONE) c = t;
        }
        sw[FC_THREADS / 32] = c;
    }
    __syncthreads();
    uint32_t ex = __shfl_up_sync(FULL, x, 1);
    if (lane == 0 || ex == FS_NONE) ex = sw[wi];  // nothing earlier in the warp: the warp's incoming state
    *last = sw[FC_THREADS / 32];
    return ex;
}

__device__ __forceinline__ uint32_t block_sum_excl(uint32_t v, uint32_t* sw, uint32_t* total) {
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sw[wi] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t c = 0;
        for (int i = 0; i < FC_THREADS / 32; ++i) {
            const uint32_t t = sw[i];
            sw[i] = c;
            c += t;
        }
        sw[FC_THREADS / 32] = c;
    }
    __syncthreads();
    const uint32_t r = sw[wi] + x - v;
    *total = sw[FC_THREADS / 32];
    return r;
}

// One CTA per stream, 4 KiB per round.  The record rules (the host reader's
// parse_fasta_fast): the first '>' anywhere starts the first header; a header
// runs to the end of its line; after it, a line starting with '>' starts the
// next record, one starting with '@' or '+' is FASTQ, and every other line is
// sequence (its bytes without the '\n'; empty lines add nothing).  A record's
// '>' is kept as its separator; bytes before the first header are dropped.
__global__ void __launch_bounds__(FC_THREADS) k_fasta_compact(stream_set s, uint64_t* seq_bytes) {
    __shared__ __align__(16) uint8_t chunk[FC_CHUNK];
    __shared__ __align__(16) uint8_t stage[FC_CHUNK + 32];
    __shared__ uint32_t sw[FC_THREADS / 32 + 1], sw2[FC_THREADS / 32 + 1];
    __shared__ uint32_t s_first, s_fastq;
    const uint32_t f = blockIdx.x;
    if (f >= s.n || s.status[f] != STREAM_OK) return;  // whole CTA
    const int t = threadIdx.x;
    uint8_t* base = s.out + s.out_off[f];
    const uint64_t L = s.out_len[f];
    const uint64_t C16 = (s.out_cap[f] + 15) & ~uint64_t(15);
    uint64_t cur = 0, hdrs = 0;
    uint32_t carry_n = 0, state = FS_NONE;
    uint8_t prev = '\n';
    if (t == 0) s_fastq = 0;
    for (uint64_t q = 0; q < L; q += FC_CHUNK) {
        const uint32_t cn = (L - q) < FC_CHUNK ? (uint32_t)(L - q) : FC_CHUNK;
        if (q + 16u * (uint32_t)t < C16)
            reinterpret_cast<uint4*>(chunk)[t] = reinterpret_cast<uint4 const*>(base + q)[t];
        if (t == 0) s_first = FC_CHUNK;
        __syncthreads();
        uint32_t lo = 0;
        if (state == FS_NONE) {
            uint32_t mine = FC_CHUNK;
            for (int j = 0; j < 16; ++j) {
                const uint32_t i = 16u * (uint32_t)t + (uint32_t)j;
                if (i < cn && (chunk[i] == '>' || chunk[i] == '@')) {
                    mine = i;
                    break;
                }
            }
            if (mine < FC_CHUNK) atomicMin(&s_first, mine);
            __syncthreads();
            lo = s_first;
            if (lo == FC_CHUNK) {  // no header yet
                prev = chunk[cn - 1];
                __syncthreads();
                continue;
            }
            if (chunk[lo] == '@') {
                if (t == 0) s_fastq = 1;
                break;
            }
        }
        // events: at lo (the first header) and at line starts after it
        uint32_t ev[16];
        uint32_t tl = FS_NONE;
        for (int j = 0; j < 16; ++j) {
            const uint32_t i = 16u * (uint32_t)t + (uint32_t)j;
            uint32_t e = FS_NONE;
            if (i < cn && i >= lo) {
                const uint8_t b = chunk[i];
                if (state == FS_NONE && i == lo) {
                    e = FS_HDR;
                } else {
                    const uint8_t pb = i ? chunk[i - 1] : prev;
                    if (pb == '\n') e = b == '>' ? FS_HDR : (b == '@' || b == '+') ? FS_FASTQ : FS_SEQ;
                }
            }
            if (e == FS_FASTQ) s_fastq = 1;
            ev[j] = e;
            if (e != FS_NONE) tl = e;
        }
        uint32_t last;
        uint32_t cs = last_event_scan(tl, state, sw, &last);
        uint32_t keep = 0, kc = 0, hc = 0;
        for (int j = 0; j < 16; ++j) {
            const uint32_t i = 16u * (uint32_t)t + (uint32_t)j;
            if (ev[j] != FS_NONE) cs = ev[j];
            const bool k = i < cn && i >= lo &&
                           (ev[j] == FS_HDR || (ev[j] != FS_FASTQ && cs == FS_SEQ && chunk[i] != '\n'));
            keep |= (uint32_t)k << j;
            kc += k;
            hc += ev[j] == FS_HDR;
        }
        uint32_t K;
        const uint32_t at = carry_n + block_sum_excl(kc, sw2, &K);
        uint32_t o = at;
        for (int j = 0; j < 16; ++j)
            if ((keep >> j) & 1u) stage[o++] = chunk[16u * (uint32_t)t + (uint32_t)j];
        // header count of this round (for the sequence-byte total)
        uint32_t H;
        block_sum_excl(hc, sw, &H);
        __syncthreads();
        const uint32_t S = carry_n + K, G = S / 16;
        uint4* dst = reinterpret_cast<uint4*>(base + (cur & ~uint64_t(15)));
        for (uint32_t g = (uint32_t)t; g < G; g += FC_THREADS) dst[g] = reinterpret_cast<uint4 const*>(stage)[g];
        __syncthreads();
        const uint32_t c2 = S - 16 * G;
        uint8_t mv = 0;
        if ((uint32_t)t < c2) mv = stage[16 * G + (uint32_t)t];
        __syncthreads();
        if ((uint32_t)t < c2) stage[t] = mv;
        cur += K;
        hdrs += H;
        carry_n = c2;
        state = last;
        prev = chunk[cn - 1];
        __syncthreads();
        if (s_fastq) break;
    }
    __syncthreads();
    if (s_fastq) {
        if (t == 0) s.status[f] = STREAM_FASTQ;
        return;
    }
    // the partial last group, then '\n' up to the end of the region
    const uint64_t g0 = cur & ~uint64_t(15);
    if (g0 < C16) {
        if ((uint32_t)t < 16 && (uint32_t)t >= carry_n) stage[t] = '\n';
        __syncthreads();
        if (t == 0) *reinterpret_cast<uint4*>(base + g0) = *reinterpret_cast<uint4 const*>(stage);
        const uint4 nl = make_uint4(0x0a0a0a0au, 0x0a0a0a0au, 0x0a0a0a0au, 0x0a0a0a0au);
        for (uint64_t g = g0 + 16 + 16u * (uint64_t)t; g < C16; g += 16u * FC_THREADS)
            *reinterpret_cast<uint4*>(base + g) = nl;
    }
    if (t == 0) {
        s.out_len[f] = cur;
        seq_bytes[f] = cur - hdrs;
    }
}

}  // namespace

void inflate_streams(stream_set const& s, cudaStream_t st) {
    if (!s.n) return;
    CDBG_CUDA(cudaFuncSetAttribute(k_inflate, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(cta_state)));
    k_inflate<<<s.n, IF_THREADS, sizeof(cta_state), st>>>(s);
    CDBG_CHECK_LAUNCH();
}

void fasta_compact(stream_set const& s, uint64_t* seq_bytes, cudaStream_t st) {
    if (!s.n) return;
    k_fasta_compact<<<s.n, FC_THREADS, 0, st>>>(s, seq_bytes);
    CDBG_CHECK_LAUNCH();
}

}  // namespace cdbg
