// The distinct words of a corpus, counted on the device, and what the merge loop of word_merge.cuh starts from.
//
// A pair is only ever counted or merged inside a word (src/bpe/train.wgsl:393-398,482-485,492-495 of the reference: the right
// symbol must not carry the word-start bit), so equal words behave alike for the whole run: every distinct word is kept once,
// with its multiplicity as the weight of its pairs, and the merge loop works on the dictionary.  Natural text repeats its words:
// 64 MiB of the benchmark text are 9.0 M words but 0.40 M distinct ones, 5.7 M symbols instead of 67 M.
//
// One pass over the bytes (k_dict_words): a CTA takes 4 KB tiles, turns the word-start mask into a list of starts in shared
// memory, and every thread looks its words up.  Words of up to 15 bytes carry their bytes in a 16-byte key (length in the last
// byte): first in a per-CTA cache in shared memory, which takes the frequent words' counts off the global atomics, then in a
// global table with 128-bit compare-and-swap inserts.  Longer words go to a second table whose 64-bit slots hold (hash, length,
// position of the first occurrence); a match is always verified against the bytes at that position.
#pragma once

#include "common.cuh"

namespace b200bpe {

constexpr int WD_THREADS = 256;
constexpr int WD_TILE = 4096;                 // bytes per tile: 16 per thread
constexpr int WD_CACHE_LOG2 = 11;             // words cached per CTA
constexpr uint32_t WD_MAX_WORD = 4096;        // a longer word is looked up by nobody: the corpus is not a text of words
constexpr int WD_MAX_PROBE = 512;

// Status bits of the dictionary pass (DictState::status).
enum : uint32_t { WD_FULL = 1u, WD_GIANT = 2u, WD_SYMBOL = 4u };

struct __align__(16) WordKey { uint32_t w[4]; };   // up to 15 bytes, zero padded; byte 15 = length (never 0)

struct DictState {
    uint32_t status;
    uint32_t positions;      // symbols of all distinct words
    uint32_t words;          // distinct words
    uint32_t pairs;          // distinct byte pairs
    unsigned long long split;   // "literal" runs: where the tail begins
    unsigned long long sampled, squares;   // of a sample of byte pairs: their number, and the sum of the squares of each pair's
};

struct DictTables {
    WordKey* short_key; uint32_t* short_cnt; uint32_t* short_base; uint32_t short_log2;
    unsigned long long* long_key; uint32_t* long_cnt; uint32_t* long_base; uint32_t long_log2;
    DictState* st;
};

__device__ __forceinline__ uint32_t wd_mix(uint32_t h, uint32_t v) {
    h = (h ^ v) * 0x9E3779B1u;
    return h ^ (h >> 15);
}
__device__ __forceinline__ bool wd_equal(const WordKey& a, const WordKey& b) {
    return a.w[0] == b.w[0] && a.w[1] == b.w[1] && a.w[2] == b.w[2] && a.w[3] == b.w[3];
}
__device__ __forceinline__ uint32_t wd_hash(const WordKey& k) {
    uint32_t h = wd_mix(wd_mix(wd_mix(wd_mix(0x85EBCA77u, k.w[0]), k.w[1]), k.w[2]), k.w[3]);
    return h * 0xC2B2AE3Du;
}
__device__ __forceinline__ WordKey wd_load(const WordKey* p) {
    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p));
    return WordKey{{v.x, v.y, v.z, v.w}};
}

// ── tiles of words ──
struct WordTile {
    alignas(16) uint8_t bytes[WD_TILE + 32];   // the tile and the 16 bytes behind it
    uint16_t start[WD_TILE];         // offsets of the words that start in the tile
    uint32_t warp_sum[WD_THREADS / 32];
    uint32_t n;                      // how many
    uint32_t next;                   // tile-relative start of the first word behind the tile (WD_TILE + WD_MAX_WORD: none near)
};

__device__ __forceinline__ uint32_t wd_nonzero_bits(uint32_t w) {   // bit k = byte k of w is not 0
    const uint32_t nz = __vsetne4(w, 0u);
    return ((nz * 0x01020408u) >> 24) & 0xFu;
}

// Fills `t` for the tile at `lo` (every thread of the CTA calls; ends with a barrier).  Word starts are the non-zero mask bytes
// and position 0.
__device__ __forceinline__ void wd_load_tile(WordTile& t, const uint8_t* __restrict__ bytes, const uint8_t* __restrict__ mask,
                                             uint64_t n, uint64_t lo, bool aligned) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t at = lo + (uint64_t)tid * 16;
    uint32_t bits = 0;
    if (aligned && at + 16 <= n) {
        *reinterpret_cast<uint4*>(t.bytes + tid * 16) = __ldcs(reinterpret_cast<const uint4*>(bytes + at));
        const uint4 m = __ldcs(reinterpret_cast<const uint4*>(mask + at));
        bits = wd_nonzero_bits(m.x) | wd_nonzero_bits(m.y) << 4 | wd_nonzero_bits(m.z) << 8 | wd_nonzero_bits(m.w) << 12;
    } else {
        for (int k = 0; k < 16; k++) {
            const bool in = at + k < n;
            t.bytes[tid * 16 + k] = in ? bytes[at + k] : (uint8_t)0;
            if (in && mask[at + k]) bits |= 1u << k;
        }
    }
    if (at == 0) bits |= 1u;
    if (warp == WD_THREADS / 32 - 1) {
        // the halo, and the first start behind the tile (the last warp has the least else to do on the last, partial tile)
        if (lane < 16) t.bytes[WD_TILE + lane] = lo + WD_TILE + lane < n ? bytes[lo + WD_TILE + lane] : (uint8_t)0;
        uint32_t found = WD_TILE + WD_MAX_WORD + 1u;
        for (uint32_t k = 0; k <= WD_MAX_WORD; k += 32) {
            const uint64_t g = lo + WD_TILE + k + lane;
            const uint32_t hit = __ballot_sync(0xFFFFFFFFu, g >= n || mask[g] != 0);   // the end of the text ends a word too
            if (hit) { found = WD_TILE + k + (uint32_t)__ffs((int)hit) - 1u; break; }
        }
        if (lane == 0) t.next = (uint64_t)found + lo > n ? (uint32_t)(n - lo) : found;
    }
    const uint32_t mine = (uint32_t)__popc(bits);
    uint32_t inc = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, d);
        if (lane >= d) inc += v;
    }
    if (lane == 31) t.warp_sum[warp] = inc;
    __syncthreads();
    uint32_t off = inc - mine, total = 0;
#pragma unroll
    for (int w = 0; w < WD_THREADS / 32; w++) {
        const uint32_t v = t.warp_sum[w];
        if (w < warp) off += v;
        total += v;
    }
    while (bits) {
        t.start[off++] = (uint16_t)(tid * 16 + __ffs((int)bits) - 1);
        bits &= bits - 1;
    }
    if (tid == 0) t.n = total;
    __syncthreads();
}

// End of the i-th word of the tile, tile-relative.
__device__ __forceinline__ uint32_t wd_end(const WordTile& t, uint32_t i) { return i + 1 < t.n ? t.start[i + 1] : t.next; }

// The 16-byte key of a word of 1..15 bytes at tile offset s (its bytes lie in the tile or its halo).
__device__ __forceinline__ WordKey wd_key(const WordTile& t, uint32_t s, uint32_t len) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(t.bytes) + (s >> 2);
    const uint32_t sh = (s & 3u) * 8u;
    const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[4];
    WordKey k{{__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh)}};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int left = (int)len - 4 * i;      // bytes of this word that belong to the key
        if (left <= 0) k.w[i] = 0u;
        else if (left < 4) k.w[i] &= (1u << (8 * left)) - 1u;
    }
    k.w[3] |= len << 24;
    return k;
}

// Slot of a short word (inserted if `insert`), or ~0u (not there / no room).
__device__ __forceinline__ uint32_t wd_find_short(const DictTables& d, const WordKey& key, uint32_t h, bool insert) {
    const uint32_t mask = (1u << d.short_log2) - 1u;
    uint32_t s = h >> (32u - d.short_log2);
    for (int p = 0; p < WD_MAX_PROBE; p++) {
        WordKey k = wd_load(d.short_key + s);
        if (k.w[3] == 0u) {
            if (!insert) return ~0u;
            k = atomicCAS(d.short_key + s, WordKey{{0u, 0u, 0u, 0u}}, key);
            if (k.w[3] == 0u) return s;
        }
        if (wd_equal(k, key)) return s;
        s = (s + 1u) & mask;
    }
    return ~0u;
}

// The same for a word of 16..WD_MAX_WORD bytes at text position pos.
__device__ __forceinline__ uint32_t wd_find_long(const DictTables& d, const uint8_t* __restrict__ bytes, const uint8_t* __restrict__ mask,
                                                 uint64_t n, uint64_t pos, uint32_t len, bool insert) {
    uint32_t h = wd_mix(0x27D4EB2Fu, len);
    for (uint32_t i = 0; i < len; i++) h = wd_mix(h, bytes[pos + i]);
    const uint32_t cap_mask = (1u << d.long_log2) - 1u;
    const uint32_t len8 = len < 255u ? len : 255u;
    // (hash, length) of a word is never 0 in the upper half: the length is at least 16
    const unsigned long long mine = (unsigned long long)((h & 0xFFFFFF00u) | len8) << 32 | (uint32_t)pos;
    uint32_t s = (h * 0xC2B2AE3Du) >> (32u - d.long_log2);
    for (int p = 0; p < WD_MAX_PROBE; p++) {
        unsigned long long k = __ldcg(d.long_key + s);
        if (k == 0ull) {
            if (!insert) return ~0u;
            k = atomicCAS(d.long_key + s, 0ull, mine);
            if (k == 0ull) return s;
        }
        if ((k >> 32) == (mine >> 32)) {
            const uint64_t rep = (uint32_t)k;
            bool same = true;
            if (rep != pos) {
                if (len8 == 255u) {   // the lengths agree only if the first occurrence ends where this one does
                    same = rep + len <= n && (rep + len == n || mask[rep + len] != 0);
                    for (uint32_t i = 1; same && i < len; i++) same = mask[rep + i] == 0;
                }
                for (uint32_t i = 0; same && i < len; i++) same = bytes[rep + i] == bytes[pos + i];
            }
            if (same) return s;
        }
        s = (s + 1u) & cap_mask;
    }
    return ~0u;
}

// Counts every word of the text.
__global__ void __launch_bounds__(WD_THREADS)
k_dict_words(const uint8_t* __restrict__ bytes, const uint8_t* __restrict__ mask, uint64_t n, DictTables d, int aligned) {
    extern __shared__ __align__(16) unsigned char wd_smem[];
    WordTile& t = *reinterpret_cast<WordTile*>(wd_smem);
    constexpr uint32_t NC = 1u << WD_CACHE_LOG2;
    WordKey* ckey = reinterpret_cast<WordKey*>(wd_smem + ((sizeof(WordTile) + 15) & ~(size_t)15));
    uint32_t* ctag = reinterpret_cast<uint32_t*>(ckey + NC);    // 0 free, 1 being filled, else the word's hash | 2
    uint32_t* ccnt = ctag + NC;
    for (uint32_t i = threadIdx.x; i < NC; i += WD_THREADS) { ctag[i] = 0u; ccnt[i] = 0u; }
    __syncthreads();
    const uint64_t tiles = (n + WD_TILE - 1) / WD_TILE;
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t lo = tile * WD_TILE;
        wd_load_tile(t, bytes, mask, n, lo, aligned != 0);
        for (uint32_t i = threadIdx.x; i < t.n; i += WD_THREADS) {
            const uint32_t s = t.start[i], len = wd_end(t, i) - s;
            if (len > 15u) {
                if (len > WD_MAX_WORD) { atomicOr(&d.st->status, (uint32_t)WD_GIANT); continue; }
                const uint32_t g = wd_find_long(d, bytes, mask, n, lo + s, len, true);
                if (g == ~0u) atomicOr(&d.st->status, (uint32_t)WD_FULL);
                else atomicAdd(d.long_cnt + g, 1u);
                continue;
            }
            const WordKey key = wd_key(t, s, len);
            const uint32_t h = wd_hash(key);
            bool done = false;
#pragma unroll
            for (uint32_t way = 0; way < 2 && !done; way++) {
                const uint32_t c = (h >> (32 - WD_CACHE_LOG2)) ^ way;
                uint32_t tag = *reinterpret_cast<volatile uint32_t*>(ctag + c);
                if (tag == 0u) {
                    tag = atomicCAS(ctag + c, 0u, 1u);
                    if (tag == 0u) {    // this thread fills the entry; until the tag is out the others pass it by
                        ckey[c] = key;
                        __threadfence_block();
                        atomicExch(ctag + c, h | 2u);
                        atomicAdd(ccnt + c, 1u);
                        done = true;
                    }
                } else if (tag == (h | 2u)) {
                    __threadfence_block();
                    if (wd_equal(ckey[c], key)) { atomicAdd(ccnt + c, 1u); done = true; }
                }
            }
            if (done) continue;
            const uint32_t g = wd_find_short(d, key, h, true);
            if (g == ~0u) atomicOr(&d.st->status, (uint32_t)WD_FULL);
            else atomicAdd(d.short_cnt + g, 1u);
        }
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < NC; i += WD_THREADS) {
        if (ccnt[i] == 0u) continue;
        const WordKey key = ckey[i];
        const uint32_t g = wd_find_short(d, key, wd_hash(key), true);
        if (g == ~0u) atomicOr(&d.st->status, (uint32_t)WD_FULL);
        else atomicAdd(d.short_cnt + g, ccnt[i]);
    }
}
constexpr size_t WD_SMEM_BYTES = ((sizeof(WordTile) + 15) & ~(size_t)15) + (size_t)(1u << WD_CACHE_LOG2) * (sizeof(WordKey) + 8);

// Gives every distinct word its place among the dictionary's positions (short_base / long_base) and counts them; no word is
// written yet, because the positions are only allocated once their number is known.
__global__ void __launch_bounds__(256)
k_dict_places(const uint8_t* __restrict__ mask, uint64_t n, DictTables d) {
    __shared__ uint32_t wsum[8], s_base;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t slots = (1ull << d.short_log2) + (1ull << d.long_log2);
    for (uint64_t b = (uint64_t)blockIdx.x * 1024; b < slots; b += (uint64_t)gridDim.x * 1024) {
        uint32_t len[4], sum = 0, words = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint64_t i = b + threadIdx.x * 4 + k;
            len[k] = 0;
            if (i < (1ull << d.short_log2)) {
                len[k] = d.short_key[i].w[3] >> 24;
            } else if (i < slots) {
                const unsigned long long key = d.long_key[i - (1ull << d.short_log2)];
                if (key) {
                    len[k] = (uint32_t)(key >> 32) & 0xFFu;
                    if (len[k] == 255u) {
                        const uint64_t pos = (uint32_t)key;
                        while (pos + len[k] < n && mask[pos + len[k]] == 0) len[k]++;
                    }
                }
            }
            sum += len[k];
            words += len[k] != 0;
        }
        uint32_t inc = sum;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, s);
            if (lane >= (uint32_t)s) inc += v;
        }
        words = __reduce_add_sync(0xFFFFFFFFu, words);
        if (lane == 31) wsum[warp] = inc;
        if (lane == 0 && words) atomicAdd(&d.st->words, words);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t total = 0;
            for (int w = 0; w < 8; w++) { const uint32_t v = wsum[w]; wsum[w] = total; total += v; }
            s_base = total ? atomicAdd(&d.st->positions, total) : 0u;
        }
        __syncthreads();
        uint32_t at = s_base + wsum[warp] + inc - sum;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint64_t i = b + threadIdx.x * 4 + k;
            if (len[k]) {
                if (i < (1ull << d.short_log2)) d.short_base[i] = at;
                else d.long_base[i - (1ull << d.short_log2)] = at;
            }
            at += len[k];
        }
        __syncthreads();
    }
}

// ── the dictionary's positions ──
// One 32-bit record per position: symbol (16 bits) | span << 16 (15 bits) | word start << 31.  A symbol that covers `span`
// positions has its record at the first of them; the last one carries the span too, so that the neighbour on the right finds the
// start of the symbol on its left; the records in between, and the symbol of the last, are 0 (no symbol 0 ever pairs).
constexpr uint32_t WP_START = 0x80000000u;
constexpr uint32_t WP_MAX_SPAN = 0x7FFFu;
static_assert(WD_MAX_WORD <= WP_MAX_SPAN, "a symbol never covers more than its word");
__device__ __forceinline__ uint32_t wp_sym(uint32_t r) { return r & 0xFFFFu; }
__device__ __forceinline__ uint32_t wp_span(uint32_t r) { return (r >> 16) & WP_MAX_SPAN; }

// Writes the words at their places: a record and a weight (the word's multiplicity) per position.
__global__ void __launch_bounds__(256)
k_dict_fill(const uint8_t* __restrict__ bytes, const uint8_t* __restrict__ mask, uint64_t n, DictTables d, uint32_t* __restrict__ rec,
            uint32_t* __restrict__ weight) {
    const uint64_t slots = (1ull << d.short_log2) + (1ull << d.long_log2);
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < slots; i += (uint64_t)gridDim.x * 256) {
        if (i < (1ull << d.short_log2)) {
            const WordKey k = d.short_key[i];
            const uint32_t len = k.w[3] >> 24;
            if (!len) continue;
            const uint32_t base = d.short_base[i], w = d.short_cnt[i];
            for (uint32_t j = 0; j < len; j++) {
                rec[base + j] = ((k.w[j >> 2] >> (8 * (j & 3))) & 0xFFu) | 1u << 16 | (j ? 0u : WP_START);
                weight[base + j] = w;
            }
        } else {
            const uint64_t s = i - (1ull << d.short_log2);
            const unsigned long long key = d.long_key[s];
            if (!key) continue;
            const uint64_t pos = (uint32_t)key;
            const uint32_t base = d.long_base[s], w = d.long_cnt[s];
            uint32_t j = 0;
            do {
                rec[base + j] = bytes[pos + j] | 1u << 16 | (j ? 0u : WP_START);
                weight[base + j] = w;
                j++;
            } while (pos + j < n && mask[pos + j] == 0);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) rec[d.st->positions] = WP_START;   // ends the last word
}

// Per byte pair: occurrences in the dictionary (upper half) and weighted count (lower half; the corpus has fewer than 2^32 symbols).
__global__ void __launch_bounds__(256)
k_dict_count(const uint32_t* __restrict__ rec, const uint32_t* __restrict__ weight, uint32_t positions, unsigned long long* __restrict__ bins) {
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < positions; i += gridDim.x * 256) {
        const uint32_t r = rec[i], nx = rec[i + 1];
        const uint32_t a = wp_sym(r), b = wp_sym(nx);
        if ((nx & WP_START) || a == 0u || b == 0u) continue;
        atomicAdd(bins + (a << 8 | b), 1ull << 32 | weight[i]);
    }
}

// Offsets of the byte pairs' occurrence lists (off has 65,537 entries, cursor 65,536), and the number of distinct byte pairs.
__global__ void __launch_bounds__(1024)
k_dict_offsets(const unsigned long long* __restrict__ bins, uint32_t* __restrict__ off, uint32_t* __restrict__ cursor, DictState* __restrict__ st) {
    __shared__ uint32_t wsum[32], wpairs[32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t sum = 0, pairs = 0;
    for (int k = 0; k < 64; k += 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(bins + threadIdx.x * 64 + k);
        sum += (uint32_t)(v.x >> 32) + (uint32_t)(v.y >> 32);
        pairs += (v.x != 0) + (v.y != 0);
    }
    uint32_t inc = sum;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, s);
        if (lane >= (uint32_t)s) inc += v;
    }
    pairs = __reduce_add_sync(0xFFFFFFFFu, pairs);
    if (lane == 31) wsum[warp] = inc;
    if (lane == 0) wpairs[warp] = pairs;
    __syncthreads();
    uint32_t at = inc - sum, total = 0, np = 0;
    for (uint32_t w = 0; w < 32; w++) {
        if (w < warp) at += wsum[w];
        total += wsum[w];
        np += wpairs[w];
    }
    for (int k = 0; k < 64; k++) {
        const uint32_t i = threadIdx.x * 64 + k;
        off[i] = at;
        cursor[i] = at;
        at += (uint32_t)(bins[i] >> 32);
    }
    if (threadIdx.x == 0) { off[65536] = total; st->pairs = np; }
}

// The occurrence lists themselves: positions, grouped by byte pair.
__global__ void __launch_bounds__(256)
k_dict_lists(const uint32_t* __restrict__ rec, uint32_t positions, uint32_t* __restrict__ cursor, uint32_t* __restrict__ list) {
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < positions; i += gridDim.x * 256) {
        const uint32_t r = rec[i], nx = rec[i + 1];
        const uint32_t a = wp_sym(r), b = wp_sym(nx);
        if ((nx & WP_START) || a == 0u || b == 0u) continue;
        list[atomicAdd(cursor + (a << 8 | b), 1u)] = i;
    }
}

// ── inputs other than (bytes, mask) ──
// No mask: the byte-class heuristic of the reference (train.wgsl:111-186), as a mask.
__device__ __forceinline__ uint32_t wd_class(uint32_t t) {
    if (t == 0x0Au) return 4u;
    if (t == 0x20u) return 2u;
    if (t - 0x30u <= 9u) return 1u;
    return (t >= 0x80u || t - 0x61u <= 25u || t - 0x41u <= 25u) ? 0u : 3u;
}
__global__ void __launch_bounds__(256)
k_dict_heuristic(const uint8_t* __restrict__ bytes, uint64_t n, uint8_t* __restrict__ mask) {
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (uint64_t)gridDim.x * 256) {
        uint32_t start = 1u;
        if (i > 0) {
            const uint32_t c = wd_class(bytes[i]), p = wd_class(bytes[i - 1]);
            start = c != p;
            if (p == 2u && c <= 1u) start = 0u;
            if (p == 4u || c == 4u) start = 1u;
        }
        mask[i] = (uint8_t)start;
    }
}
// Tagged symbols: bytes and mask, if every symbol is a byte value (WD_SYMBOL otherwise).
__global__ void __launch_bounds__(256)
k_dict_split(const uint32_t* __restrict__ sym, uint64_t n, uint8_t* __restrict__ bytes, uint8_t* __restrict__ mask, DictState* __restrict__ st) {
    bool bad = false;
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (uint64_t)gridDim.x * 256) {
        const uint32_t s = sym[i];
        bad |= (s & ~(WORD_START_BIT | 0xFFu)) != 0u;
        bytes[i] = (uint8_t)s;
        mask[i] = (s & WORD_START_BIT) ? 1 : 0;
    }
    if (bad) atomicOr(&st->status, (uint32_t)WD_SYMBOL);
}

// ── the tail of a "literal" run ──
// First word start at or behind `from`, or n (one CTA; a text without one within WD_MAX_WORD bytes is not one of words).
__global__ void __launch_bounds__(256)
k_dict_split_at(const uint8_t* __restrict__ mask, uint64_t n, uint64_t from, DictState* __restrict__ st) {
    for (uint64_t b = from; b < n && b <= from + WD_MAX_WORD; b += 256) {
        __shared__ uint32_t best;
        if (threadIdx.x == 0) best = 256u;
        __syncthreads();
        if (b + threadIdx.x < n && mask[b + threadIdx.x]) atomicMin(&best, threadIdx.x);
        __syncthreads();
        if (best < 256u) { if (threadIdx.x == 0) st->split = b + best; return; }
        __syncthreads();
    }
    if (threadIdx.x == 0) st->split = n;
}
// Tagged symbols of the tail, and its byte pairs in the lower halves of the bins.
__global__ void __launch_bounds__(256)
k_dict_tail(const uint8_t* __restrict__ bytes, const uint8_t* __restrict__ mask, uint64_t at, uint64_t n, uint32_t* __restrict__ tail,
            unsigned long long* __restrict__ bins) {
    for (uint64_t i = at + (uint64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (uint64_t)gridDim.x * 256) {
        const uint32_t l = bytes[i];
        tail[i - at] = l | (mask[i] ? WORD_START_BIT : 0u);
        if (i + 1 >= n || mask[i + 1]) continue;
        const uint32_t r = bytes[i + 1];
        if (l && r) atomicAdd(bins + (l << 8 | r), 1ull);
    }
}

// ── how many byte pairs a text uses ──
// A place in each of WD_SAMPLE equal parts of the text (scattered, so that no column of a table is all there is): the pairs of different
// bytes there, inside words, counted in the bins.  A pair of equal bytes does not count, because a run of them is gone with one merge.  One CTA.
constexpr uint32_t WD_SAMPLE = 32768;
__global__ void __launch_bounds__(1024)
k_dict_sample(const uint8_t* __restrict__ bytes, const uint8_t* __restrict__ mask, uint64_t n, unsigned long long* __restrict__ bins, DictState* __restrict__ st) {
    const uint64_t step = n / WD_SAMPLE + 1;
    unsigned long long squares = 0ull, taken = 0ull;
#pragma unroll 8
    for (uint32_t k = threadIdx.x; k < WD_SAMPLE; k += 1024) {
        const uint64_t i = k * step + k * 0x9E3779B1u % step;
        if (i + 1 >= n || mask[i + 1]) continue;
        const uint32_t l = bytes[i], r = bytes[i + 1];
        if (l == r || l == 0u || r == 0u) continue;
        squares += 2ull * atomicAdd(bins + (l << 8 | r), 1ull) + 1ull;      // (k + 1)^2 - k^2
        taken++;
    }
    atomicAdd(&st->squares, squares);
    atomicAdd(&st->sampled, taken);
}

// ── the live symbols, in text order ──
// Two passes with a scan of the tiles' counts in between: k_dict_expand<false> counts, <true> writes.
__device__ __forceinline__ uint32_t wd_place(const DictTables& d, const WordTile& t, const uint8_t* bytes, const uint8_t* mask, uint64_t n,
                                             uint64_t lo, uint32_t s, uint32_t len) {
    if (len > 15u) {
        const uint32_t g = wd_find_long(d, bytes, mask, n, lo + s, len, false);
        return g == ~0u ? ~0u : d.long_base[g];
    }
    const WordKey key = wd_key(t, s, len);
    const uint32_t g = wd_find_short(d, key, wd_hash(key), false);
    return g == ~0u ? ~0u : d.short_base[g];
}
template <bool WRITE>
__global__ void __launch_bounds__(WD_THREADS)
k_dict_expand(const uint8_t* __restrict__ bytes, const uint8_t* __restrict__ mask, uint64_t n, DictTables d, const uint32_t* __restrict__ rec,
              uint32_t* __restrict__ tile_count, uint32_t* __restrict__ out, int aligned) {
    __shared__ WordTile t;
    __shared__ uint32_t wsum[WD_THREADS / 32], s_at;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t tiles = (n + WD_TILE - 1) / WD_TILE;
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t lo = tile * WD_TILE;
        wd_load_tile(t, bytes, mask, n, lo, aligned != 0);
        if (threadIdx.x == 0) s_at = WRITE ? tile_count[tile] : 0u;
        for (uint32_t b = 0; b < t.n; b += WD_THREADS) {
            const uint32_t i = b + threadIdx.x;
            uint32_t live = 0, base = ~0u, len = 0;
            if (i < t.n) {
                len = wd_end(t, i) - t.start[i];
                base = wd_place(d, t, bytes, mask, n, lo, t.start[i], len);
                if (base != ~0u) for (uint32_t p = 0; p < len; p += wp_span(rec[base + p])) live++;
            }
            uint32_t inc = live;
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, s);
                if (lane >= (uint32_t)s) inc += v;
            }
            if (lane == 31) wsum[warp] = inc;
            __syncthreads();
            uint32_t at = s_at + inc - live, total = 0;
            for (uint32_t w = 0; w < WD_THREADS / 32; w++) {
                if (w < warp) at += wsum[w];
                total += wsum[w];
            }
            if (WRITE && base != ~0u) {
                for (uint32_t p = 0; p < len; p += wp_span(rec[base + p]))
                    out[at++] = wp_sym(rec[base + p]) | (mask[lo + t.start[i] + p] ? WORD_START_BIT : 0u);
            }
            __syncthreads();
            if (threadIdx.x == 0) s_at += total;
            __syncthreads();
        }
        if (!WRITE && threadIdx.x == 0) tile_count[tile] = s_at;
        __syncthreads();
    }
}
// Exclusive sums of n counts in place, the total behind them (one CTA; read-backs only).
__global__ void __launch_bounds__(1024)
k_dict_scan(uint32_t* __restrict__ v, uint64_t n) {
    __shared__ uint32_t wsum[32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint64_t b = 0; b < n; b += 1024) {
        const uint64_t i = b + threadIdx.x;
        const uint32_t x = i < n ? v[i] : 0u;
        uint32_t inc = x;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, s);
            if (lane >= (uint32_t)s) inc += y;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        uint32_t at = carry + inc - x;
        for (uint32_t w = 0; w < 32; w++) {
            if (w < warp) at += wsum[w];
            carry += wsum[w];
        }
        if (i < n) v[i] = at;
        __syncthreads();
    }
    if (threadIdx.x == 0) v[n] = carry;
}

}  // namespace b200bpe
