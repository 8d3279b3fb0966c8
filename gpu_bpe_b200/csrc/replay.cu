// Merge-replay encoding on the device: the other encode(text) of the reference, the one behind its
// Tokenizer tab (TokenizerManager.encode, src/ui/tokenizer-manager.js:13-61 of toprakdeviren/gpu-bpe).
//
// The reference starts from one token per UTF-8 byte and applies every merge rule [a, b, newId] in
// the order it was learned, each as one left-to-right pass over the WHOLE token list that replaces
// a matching adjacent pair and steps over both tokens (:45-58).  There are no word boundaries and
// no chunks on this path, and with a == b a run of k equal tokens pairs up from the left:
// floor(k / 2) new tokens, then the odd one out.  This differs from the trie encoder (greedy
// longest match) and from the trainer's merge (snapshot rule, runs collapse).
//
// Two bytes next to each other can only ever end up in one token if some rule joins a token that
// ends with the first to a token that begins with the second.  Where no rule does (for a list
// learned on words that is nearly every place between two words) the text falls apart into
// segments that the rules treat independently, so k_replay_segments encodes each of them by
// itself: always its smallest rank, leftmost first, which is the order in which the passes find
// the pairs.  A text with a segment too long for that (RS_HALO) goes through the rounds below.
//
// Rounds: a rule only does anything if its pair is present, so instead of one pass per rule the
// device works in rounds.  A round (1) looks every adjacent pair of the current list up in a hash
// table pair → (rank, newId) and takes the smallest rank present, (2) applies that one rule with a
// single-pass scan + compaction (decoupled look-back, bounded waits) from the ping into the pong
// buffer.  Both are equivalent to the reference's rule-by-rule loop when no rule refers to an id
// that is only made by a later rule and every rule makes an id of its own (then a pair that appears
// after rule r can only match rules after r, which is all the in-order loop would still try);
// every merge list a trainer produces is like that, and b200bpe_replay_create refuses the others.
// For a == b the pairing from the left needs, per token, the parity of the run of `a` that ends
// right before it: inside a tile that is a segmented scan over (all tokens are `a`, parity of the
// trailing run); for the run that reaches the tile's first token one thread reads backwards from
// the tile's start until the run ends (runs are short in text).
#include <algorithm>
#include <cstring>
#include <string>
#include <unordered_map>
#include <vector>

#include "ctx.cuh"

namespace b200bpe {

constexpr int RP_THREADS = 256;
constexpr int RP_PER_THREAD = 8;
constexpr int RP_TILE = RP_THREADS * RP_PER_THREAD;   // tokens per tile
constexpr int RP_ROUNDS_PER_GRAPH = 64;
constexpr uint32_t RP_NO_RANK = 0xFFFFFFFFu;
constexpr uint32_t RP_MAX_SPINS = 1u << 22;

struct ReplayState {
    uint32_t n[2];        // tokens in the ping / pong buffer, indexed by (epoch & 1)
    uint32_t epoch;       // rounds applied so far
    uint32_t done;        // no pair of the list has a rule any more
    uint32_t best_rank;   // smallest rank among the pairs present (RP_NO_RANK: none)
    uint32_t a, b, new_id;
    uint32_t ticket;      // next tile of the apply kernel
    uint32_t status;      // 0 ok, 2 a look-back wait ran out
    uint32_t rounds;      // statistics
    uint32_t pad;
};

struct RankSlot { unsigned long long key; uint32_t rank, new_id; };   // key 0 = empty (a pair (0, 0) is stored as ~0)

__device__ __forceinline__ uint32_t rp_hash(unsigned long long key) {
    uint32_t x = (uint32_t)key ^ ((uint32_t)(key >> 32) * 0x9E3779B1u);
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}
__device__ __forceinline__ unsigned long long rp_key(uint32_t a, uint32_t b) {
    const unsigned long long k = ((unsigned long long)a << 32) | b;
    return k ? k : ~0ull;
}

__global__ void k_replay_bytes(const uint8_t* __restrict__ bytes, uint32_t* __restrict__ tok, uint64_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) tok[i] = bytes[i];
}

// (1) the smallest rank among the adjacent pairs of the current list
__global__ void __launch_bounds__(RP_THREADS)
k_replay_rank(ReplayState* __restrict__ st, const uint32_t* buf0, const uint32_t* buf1, const RankSlot* __restrict__ table, uint32_t mask) {
    if (st->done | st->status) return;
    const uint32_t e = st->epoch, N = st->n[e & 1];
    const uint32_t* __restrict__ src = (e & 1) ? buf1 : buf0;
    uint32_t best = RP_NO_RANK;
    for (uint32_t i = blockIdx.x * RP_THREADS + threadIdx.x; i + 1 < N; i += gridDim.x * RP_THREADS) {
        const unsigned long long key = rp_key(src[i], src[i + 1]);
        uint32_t slot = rp_hash(key) & mask;
        for (;;) {
            const RankSlot s = table[slot];
            if (s.key == key) { best = min(best, s.rank); break; }
            if (s.key == 0ull) break;
            slot = (slot + 1) & mask;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xFFFFFFFFu, best, o));
    if ((threadIdx.x & 31) == 0 && best != RP_NO_RANK) atomicMin(&st->best_rank, best);
}

// between (1) and (2): the rule of this round
__global__ void k_replay_setup(ReplayState* __restrict__ st, const uint32_t* __restrict__ rules) {
    if (st->done | st->status) return;
    const uint32_t r = st->best_rank;
    if (r == RP_NO_RANK) { st->done = 1u; return; }
    st->a = rules[3 * r]; st->b = rules[3 * r + 1]; st->new_id = rules[3 * r + 2];
    st->best_rank = RP_NO_RANK;
    st->ticket = 0u;
    st->rounds += 1u;
}

// Tokens kept by the tiles before `tile`, by decoupled look-back; called by one whole warp.  The tile's own count `agg` goes out
// first.  A wait that runs out sets *status to 2 and gives 0.
// desc[tile] = (tag << 34) | (flag << 32) | kept, flag 1 aggregate / 2 inclusive prefix.
__device__ __forceinline__ uint32_t rp_look_back(unsigned long long* __restrict__ desc, uint32_t tile, uint32_t tag, uint32_t agg, int lane,
                                                 uint32_t* status) {
    unsigned long long excl = 0ull;
    if (tile == 0u) {
        if (lane == 0)
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(desc), "l"(((unsigned long long)((tag << 2) | 2u) << 32) | agg) : "memory");
    } else {
        if (lane == 0) {
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(desc + tile), "l"(((unsigned long long)((tag << 2) | 1u) << 32) | agg) : "memory");
        }
        int pos = (int)tile - 1;
        uint32_t spins = 0u;
        bool timed_out = false;
        for (;;) {
            const int idx = pos - lane;
            uint32_t hi = (tag << 2) | 2u, val = 0u;   // before tile 0: a zero prefix
            for (;;) {
                if (idx >= 0) {
                    unsigned long long d;
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(d) : "l"(desc + idx) : "memory");
                    hi = (uint32_t)(d >> 32); val = (uint32_t)d;
                }
                const bool ready = (hi >> 2) == tag && (hi & 3u) != 0u;
                if (__all_sync(0xFFFFFFFFu, ready)) break;
                if (++spins > RP_MAX_SPINS) { timed_out = true; break; }
                __nanosleep(40);
            }
            if (timed_out) break;
            const uint32_t pmask = __ballot_sync(0xFFFFFFFFu, (hi & 3u) == 2u);
            const int first = pmask ? (__ffs(pmask) - 1) : 32;
            uint32_t contrib = lane <= first ? val : 0u;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(0xFFFFFFFFu, contrib, o);
            excl += contrib;
            if (pmask) break;
            pos -= 32;
        }
        if (timed_out) { if (lane == 0) atomicExch(status, 2u); excl = 0ull; }
        if (lane == 0)
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(desc + tile), "l"(((unsigned long long)((tag << 2) | 2u) << 32) | (uint32_t)(excl + agg)) : "memory");
    }
    return (uint32_t)excl;
}

// (2) apply the rule: left-to-right pairing, stable compaction ping → pong.
// The tag of the look-back is round + 1.
__global__ void __launch_bounds__(RP_THREADS)
k_replay_apply(ReplayState* __restrict__ st, uint32_t* buf0, uint32_t* buf1, unsigned long long* __restrict__ desc) {
    __shared__ uint32_t s_tile, s_warp[RP_THREADS / 32], s_excl, s_run[RP_THREADS / 32], s_before;
    if (st->done | st->status) return;
    const uint32_t e = st->epoch, N = st->n[e & 1];
    const uint32_t* __restrict__ src = (e & 1) ? buf1 : buf0;
    uint32_t* __restrict__ dst = (e & 1) ? buf0 : buf1;
    const uint32_t A = st->a, B = st->b, NW = st->new_id;
    const uint32_t ntiles = (N + RP_TILE - 1) / RP_TILE;
    const uint32_t tag = (e + 1u) & 0x3FFFFFFFu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_tile = atomicAdd(&st->ticket, 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= ntiles) return;
        const uint32_t i0 = tile * RP_TILE + threadIdx.x * RP_PER_THREAD;   // this thread's first token
        // a token is the second of a pair (dropped) or the first (rewritten) or neither.
        // a != b: pairs cannot overlap.  a == b: within a run of `a`, the tokens at odd distance from
        // the run's start are the second halves; the distance's parity is carried along.
        uint32_t t[RP_PER_THREAD + 1];
#pragma unroll
        for (int k = 0; k <= RP_PER_THREAD; k++) t[k] = i0 + k < N ? src[i0 + k] : 0xFFFFFFFFu;   // (0xFFFFFFFF is no token)
        uint32_t odd = 0u;   // a == b: parity of the run of `a` that ends right before this thread's first token
        const uint32_t prev = i0 > 0u && i0 <= N ? src[i0 - 1u] : 0xFFFFFFFFu;
        if (A == B) {
            // this thread's tokens as one element (bit 1: all of them are `a`, bit 0: parity of the trailing run of `a`);
            // combine(left, right) = right is all `a` ? (left.all, left.parity ^ right.parity) : right
            uint32_t tr = 0u;
#pragma unroll
            for (int k = RP_PER_THREAD - 1; k >= 0; k--) { if (t[k] == A && tr == (uint32_t)(RP_PER_THREAD - 1 - k)) tr++; }
            const uint32_t mine = (tr == (uint32_t)RP_PER_THREAD ? 2u : 0u) | (tr & 1u);
            uint32_t inc = mine;   // inclusive scan within the warp
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t left = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o && (inc & 2u)) inc = (left & 2u) | ((left ^ inc) & 1u);
            }
            if (lane == 31) s_run[warp] = inc;
            if (threadIdx.x == 0) {
                // the run that ends right before the tile
                uint32_t len = 0u;
                if (prev == A) { len = 1u; for (uint32_t j = i0 - 1u; j > 0u && src[j - 1u] == A; j--) len++; }
                s_before = len & 1u;
            }
            __syncthreads();
            uint32_t ex = __shfl_up_sync(0xFFFFFFFFu, inc, 1);   // exclusive: everything of the warp before this thread
            if (lane == 0) ex = 2u;                               // nothing: all `a` (vacuously), parity 0
            uint32_t pre = 2u;                                    // the warps before this one
            for (int w2 = 0; w2 < warp; w2++) { const uint32_t r = s_run[w2]; pre = (r & 2u) ? ((pre & 2u) | ((pre ^ r) & 1u)) : r; }
            const uint32_t all_before = (ex & 2u) ? ((pre & 2u) | ((pre ^ ex) & 1u)) : ex;   // the tile's tokens before this thread
            odd = (all_before & 1u) ^ ((all_before & 2u) ? s_before : 0u);
        }
        uint32_t keep = 0u, rew = 0u;
        bool prev_first = A != B ? (prev == A && t[0] == B && i0 < N) : false;   // the token before is the first of a pair that takes t[0]
        if (A == B) prev_first = odd != 0u && t[0] == A;
#pragma unroll
        for (int k = 0; k < RP_PER_THREAD; k++) {
            const bool live = i0 + k < N;
            bool first = false;
            if (!prev_first) first = live && t[k] == A && t[k + 1] == B;   // t[k + 1] is 0xFFFFFFFF beyond the end
            if (live && !prev_first) keep |= 1u << k;
            if (first) rew |= 1u << k;
            prev_first = first;
        }
        const uint32_t cnt = __popc(keep);
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += x;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        uint32_t warp_off = 0u, agg = 0u;
#pragma unroll
        for (int w = 0; w < RP_THREADS / 32; w++) { if (w < warp) warp_off += s_warp[w]; agg += s_warp[w]; }
        if (warp == 0) {
            const uint32_t excl = rp_look_back(desc, tile, tag, agg, lane, &st->status);
            if (lane == 0) {
                s_excl = excl;
                if (tile == ntiles - 1u) {
                    st->n[(e + 1u) & 1u] = excl + agg;
                    st->epoch = e + 1u;
                }
            }
        }
        __syncthreads();
        uint32_t o = s_excl + warp_off + incl - cnt;
#pragma unroll
        for (int k = 0; k < RP_PER_THREAD; k++)
            if ((keep >> k) & 1u) dst[o++] = ((rew >> k) & 1u) ? NW : t[k];
    }
}

// ── segments ──
// Inside the kernel a token is a byte value, or 256 + the rank of the rule that made it: 21 bits, so that a rule fits 8 bytes
// (left << 43 | right << 22 | rank + 1, 0 = empty slot; table at most half full) and applying it needs no second load.
constexpr int RS_THREADS = 256;
constexpr int RS_TILE = 1024;                 // bytes whose segments one CTA takes at a time
constexpr int RS_HALO = 512;                  // how far the last of them may reach behind the tile
constexpr int RS_SPAN = RS_TILE + RS_HALO + 32;
constexpr uint32_t RS_SHORT = 32;             // a segment of up to so many bytes is one thread's, a longer one a warp's
constexpr uint32_t RS_MAX_RULES = (1u << 21) - 257u;   // (token 2^21 - 1 stays free)
constexpr uint32_t RS_NONE = 0xFFFFFFFFu;

struct SegmentState {
    uint32_t ticket;
    uint32_t status;       // 0 ok, 1 a segment is too long, 2 a look-back wait ran out
    uint32_t n_tokens;
    uint32_t pad;
};
struct SegmentRules {
    const uint32_t* join;              // bit (x << 8 | y): some rule joins a token that ends with byte x to one that begins with y
    const unsigned long long* table;
    uint32_t mask;
    const uint32_t* rules;             // [a, b, id] by rank
};

__host__ __device__ __forceinline__ uint32_t rs_hash(unsigned long long pair) {   // pair = left << 21 | right
    uint32_t x = (uint32_t)pair * 0x9E3779B1u ^ (uint32_t)(pair >> 21) * 0x85EBCA77u;
    x ^= x >> 15;
    return (x * 0xC2B2AE3Du) >> 7;
}
__device__ __forceinline__ bool rs_joins(const SegmentRules& R, uint32_t x, uint32_t y) {
    const uint32_t i = x << 8 | y;
    return (__ldg(R.join + (i >> 5)) >> (i & 31u)) & 1u;
}
// Rank of the rule for a pair, given its first table slot and what is there.
__device__ __forceinline__ uint32_t rs_rank(const SegmentRules& R, unsigned long long pair, uint32_t slot, unsigned long long v) {
    while (v != 0ull) {
        if ((v >> 22) == pair) return ((uint32_t)v & 0x3FFFFFu) - 1u;
        slot = (slot + 1u) & R.mask;
        v = __ldg(R.table + slot);
    }
    return RS_NONE;
}
__device__ __forceinline__ unsigned long long rs_pair(uint32_t l, uint32_t r) { return (unsigned long long)l << 21 | r; }

// One tile of bytes per turn: the segments that begin in it.  A few hundred segments of a few bytes, each a serial chain of
// (smallest rank, two look-ups) steps; what bounds the kernel is that chain in the longest segment of a warp, so every segment is
// in flight at once, and the look-ups of the byte pairs, which are most of them, are made beforehand by all threads together.
// A call on 192 KiB of text with 4,000 rules: 56.2 ms in some 3,300 rounds of three launches, 0.185 ms in segments, which is the two
// copies and one launch of this kernel.
__global__ void __launch_bounds__(RS_THREADS)
k_replay_segments(SegmentState* __restrict__ st, const uint8_t* __restrict__ bytes, uint64_t n, SegmentRules R, uint8_t* __restrict__ applied,
                  unsigned long long* __restrict__ desc, uint32_t* __restrict__ out) {
    __shared__ uint32_t tok[RS_SPAN], rnk[RS_SPAN];     // rnk[i]: rank of the rule for tokens i and i + 1 of the same segment
    __shared__ uint16_t start[RS_TILE], cnt[RS_TILE], longs[RS_TILE / RS_SHORT + 1];
    __shared__ uint32_t s_tile, s_warp[RS_THREADS / 32], s_next, s_longs, s_excl, s_over;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t ntiles = (uint32_t)((n + RS_TILE - 1) / RS_TILE);
    auto ranks2 = [&](unsigned long long p0, unsigned long long p1, uint32_t& r0, uint32_t& r1) {
        const uint32_t a0 = rs_hash(p0) & R.mask, a1 = rs_hash(p1) & R.mask;
        const unsigned long long v0 = __ldg(R.table + a0), v1 = __ldg(R.table + a1);   // both in flight
        r0 = rs_rank(R, p0, a0, v0);
        r1 = rs_rank(R, p1, a1, v1);
    };
    for (;;) {
        __syncthreads();
        if (tid == 0) { s_over = *reinterpret_cast<volatile uint32_t*>(&st->status); s_tile = atomicAdd(&st->ticket, 1u); s_longs = 0u; }
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= ntiles) return;
        const uint64_t lo = (uint64_t)tile * RS_TILE;
        // the tile's bytes, and where segments begin
        uint32_t bits = 0u;
        {
            const uint64_t at = lo + tid * 4u;
            uint32_t prev = at > 0 && at < n ? bytes[at - 1] : 0u;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t c = at + k < n ? bytes[at + k] : 0u;
                tok[tid * 4u + k] = c;
                if (at + k < n && (at + k == 0 || !rs_joins(R, prev, c))) bits |= 1u << k;
                prev = c;
            }
        }
        if (warp == RS_THREADS / 32 - 1) {   // the bytes behind the tile up to the first beginning there
            uint32_t found = RS_NONE;
            for (uint32_t k = 0; k <= (uint32_t)RS_HALO && found == RS_NONE; k += 32) {
                const uint64_t g = lo + RS_TILE + k + lane;
                const uint32_t c = g < n ? bytes[g] : 0u;
                if (k < (uint32_t)RS_HALO) tok[RS_TILE + k + lane] = c;
                const uint32_t hit = __ballot_sync(0xFFFFFFFFu, g >= n || !rs_joins(R, bytes[g - 1], c));
                if (hit) found = RS_TILE + k + (uint32_t)__ffs((int)hit) - 1u;
            }
            if (lane == 0) s_next = found != RS_NONE && lo + found > n ? (uint32_t)(n - lo) : found;
        }
        uint32_t inc = (uint32_t)__popc(bits);
        const uint32_t mine = inc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= (uint32_t)o) inc += x;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        uint32_t at = inc - mine, segments = 0u;
#pragma unroll
        for (uint32_t w = 0; w < RS_THREADS / 32; w++) { const uint32_t v = s_warp[w]; if (w < warp) at += v; segments += v; }
        while (bits) {
            start[at++] = (uint16_t)(tid * 4u + (uint32_t)__ffs((int)bits) - 1u);
            bits &= bits - 1u;
        }
        uint32_t end = s_next;               // of the last segment that begins here
        if (end == RS_NONE || end > (uint32_t)(RS_TILE + RS_HALO)) {
            end = RS_TILE + RS_HALO;
            if (segments) {
                if (tid == 0) atomicMax(&st->status, 1u);
                segments = 0u;
            }
        }
        // A text with a segment too long goes through the rounds: nothing that is left is worth doing but to tell the tiles behind that
        // there are no tokens here.
        if (s_over) segments = 0u;
        __syncthreads();
        // the byte pairs' ranks
        if (segments) {
            for (uint32_t i = start[0] + tid; i < end; i += RS_THREADS) {
                uint32_t r = RS_NONE;
                if (i + 1u < end && rs_joins(R, tok[i], tok[i + 1])) {
                    const unsigned long long p = rs_pair(tok[i], tok[i + 1]);
                    const uint32_t slot = rs_hash(p) & R.mask;
                    r = rs_rank(R, p, slot, __ldg(R.table + slot));
                }
                rnk[i] = r;
            }
        }
        __syncthreads();
        // short segments: a thread each
        for (uint32_t i = tid; i < segments; i += RS_THREADS) {
            const uint32_t s = start[i];
            uint32_t m = (i + 1u < segments ? start[i + 1] : end) - s;
            if (m > RS_SHORT) { longs[atomicAdd(&s_longs, 1u)] = (uint16_t)i; continue; }
            while (m > 1u) {
                uint32_t best = RS_NONE, b = 0u;
                for (uint32_t j = 0; j + 1u < m; j++) { const uint32_t r = rnk[s + j]; if (r < best) { best = r; b = j; } }
                if (best == RS_NONE) break;
                applied[best] = 1;
                const uint32_t t = 256u + best;
                for (uint32_t j = b + 1u; j + 1u < m; j++) { tok[s + j] = tok[s + j + 1]; rnk[s + j] = rnk[s + j + 1]; }
                m--;
                tok[s + b] = t;
                // a missing neighbour is looked up as token 2^21 - 1, which no rule has
                uint32_t rl, rr;
                ranks2(rs_pair(b > 0u ? tok[s + b - 1] : 0x1FFFFFu, t), rs_pair(t, b + 1u < m ? tok[s + b + 1] : 0x1FFFFFu), rl, rr);
                if (b > 0u) rnk[s + b - 1] = rl;
                rnk[s + b] = rr;
            }
            cnt[i] = (uint16_t)m;
        }
        __syncthreads();
        // long segments: a warp each
        for (uint32_t q = warp; q < s_longs; q += RS_THREADS / 32) {
            const uint32_t i = longs[q], s = start[i];
            uint32_t m = (i + 1u < segments ? start[i + 1] : end) - s;
            // A pass applies all pairs of the smallest rank, from the left, as a rule does: in a run of matches (of two equal tokens) every other
            // one.  A segment of a repeated byte then takes as many passes as rules apply, not a step per token (1,536 x "a": a call 2.0 -> 0.11 ms, in rounds 0.27).
            uint32_t best = RS_NONE;
            for (uint32_t j = lane; j + 1u < m; j += 32) best = min(best, rnk[s + j]);
            for (;;) {
                const uint32_t all = __reduce_min_sync(0xFFFFFFFFu, best);
                if (all == RS_NONE) break;
                const uint32_t t = 256u + all, below = (1u << lane) - 1u;
                uint32_t kept = 0u, odd = 0u, drop = 0u;     // of the block before: its last run of matches has an odd length; its last token is taken
                for (uint32_t j0 = 0u; j0 < m; j0 += 32) {
                    const uint32_t j = j0 + lane;
                    const uint32_t a = j < m ? tok[s + j] : 0u, r = j + 1u < m ? rnk[s + j] : RS_NONE;
                    const uint32_t match = __ballot_sync(0xFFFFFFFFu, r == all);
                    const uint32_t gap = ~match & below;     // lanes below this one without a match
                    const uint32_t place = gap ? lane - (32u - (uint32_t)__clz((int)gap)) : lane + odd;   // in the run of matches
                    const bool take = r == all && !(place & 1u);
                    const uint32_t taken = __ballot_sync(0xFFFFFFFFu, take);
                    const bool keep = j < m && !((taken << 1 | drop) >> lane & 1u);
                    const uint32_t keeps = __ballot_sync(0xFFFFFFFFu, keep);
                    __syncwarp();                            // everybody has read the block
                    if (keep) {
                        const uint32_t p = s + kept + (uint32_t)__popc(keeps & below);
                        tok[p] = take ? t : a;
                        rnk[p] = r;
                    }
                    kept += (uint32_t)__popc(keeps);
                    odd = match == 0xFFFFFFFFu ? odd : (uint32_t)__clz((int)~match) & 1u;   // (a whole block of matches is an even number)
                    drop = taken >> 31;
                }
                m = kept;
                if (lane == 0) applied[all] = 1;
                __syncwarp();
                best = RS_NONE;                              // the ranks beside the new tokens, and the smallest of all
                for (uint32_t j = lane; j + 1u < m; j += 32) {
                    const uint32_t x = tok[s + j], y = tok[s + j + 1];
                    uint32_t r = rnk[s + j];
                    if (x == t || y == t) {
                        const unsigned long long p = rs_pair(x, y);
                        const uint32_t slot = rs_hash(p) & R.mask;
                        r = rs_rank(R, p, slot, __ldg(R.table + slot));
                        rnk[s + j] = r;
                    }
                    best = min(best, r);
                }
                __syncwarp();
            }
            if (lane == 0) cnt[i] = (uint16_t)m;
        }
        __syncthreads();
        // where the tokens go: four consecutive segments per thread
        uint32_t c[4], sum = 0u;
#pragma unroll
        for (int k = 0; k < 4; k++) { const uint32_t i = tid * 4u + k; c[k] = i < segments ? cnt[i] : 0u; sum += c[k]; }
        inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= (uint32_t)o) inc += x;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        uint32_t off = inc - sum, total = 0u;
#pragma unroll
        for (uint32_t w = 0; w < RS_THREADS / 32; w++) { const uint32_t v = s_warp[w]; if (w < warp) off += v; total += v; }
        if (warp == 0) {
            const uint32_t excl = rp_look_back(desc, tile, 1u, total, (int)lane, &st->status);
            if (lane == 0) {
                s_excl = excl;
                if (tile == ntiles - 1u) st->n_tokens = excl + total;
            }
        }
        __syncthreads();
        uint32_t o = s_excl + off;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (!c[k]) continue;
            const uint32_t s = start[tid * 4u + k];
            for (uint32_t j = 0; j < c[k]; j++) {
                const uint32_t t = tok[s + j];
                out[o++] = t < 256u ? t : __ldg(R.rules + 3u * (t - 256u) + 2u);
            }
        }
    }
}

struct Replay {
    CtxHold hold;
    Ctx* ctx = nullptr;
    uint32_t n_rules = 0;
    uint32_t* d_rules = nullptr;
    RankSlot* d_table = nullptr;
    uint32_t mask = 0;
    ReplayState* d_state = nullptr;
    ReplayState* h_state = nullptr;   // pinned
    uint32_t* buf[2] = {nullptr, nullptr};
    uint8_t* d_in = nullptr;
    unsigned long long* d_desc = nullptr;
    uint64_t cap = 0;
    cudaGraphExec_t graph = nullptr;
    uint64_t graph_cap = 0;
    uint32_t last_rounds = 0;
    // segments
    SegmentRules seg{};                   // table == nullptr: more rules than its entries can number
    uint32_t* d_join = nullptr;
    unsigned long long* d_seg_table = nullptr;
    unsigned char* d_work = nullptr;      // SegmentState, a byte per rule (was it applied?), look-back descriptors
    SegmentState* h_seg = nullptr;        // pinned
    uint64_t work_cap = 0;                // bytes of input that d_work has descriptors for
    bool by_segments = false;             // the last text went through k_replay_segments
    uint32_t* result = nullptr;           // its tokens

    ~Replay() {
        if (ctx) cudaSetDevice(ctx->device);
        if (graph) cudaGraphExecDestroy(graph);
        cudaFree(d_rules); cudaFree(d_table); cudaFree(d_state); cudaFree(buf[0]); cudaFree(buf[1]); cudaFree(d_in); cudaFree(d_desc);
        cudaFree(d_join); cudaFree(d_seg_table); cudaFree(d_work);
        if (h_state) cudaFreeHost(h_state);
        if (h_seg) cudaFreeHost(h_seg);
    }

    b200bpe_status ensure(uint64_t n) {
        if (n <= cap) return B200BPE_OK;
        B2_CUDA(cudaStreamSynchronize(ctx->stream));
        if (graph) { cudaGraphExecDestroy(graph); graph = nullptr; }
        cudaFree(buf[0]); cudaFree(buf[1]); cudaFree(d_in); cudaFree(d_desc);
        buf[0] = buf[1] = nullptr; d_in = nullptr; d_desc = nullptr;
        cap = n + n / 2 + 16;
        B2_CUDA(cudaMalloc(&buf[0], cap * 4));
        B2_CUDA(cudaMalloc(&buf[1], cap * 4));
        B2_CUDA(cudaMalloc(&d_in, cap));
        B2_CUDA(cudaMalloc(&d_desc, (cap / RP_TILE + 2) * 8));
        B2_CUDA(cudaMemsetAsync(d_desc, 0, (cap / RP_TILE + 2) * 8, ctx->stream));
        return B200BPE_OK;
    }

    void enqueue_round(int grid_rank, int grid_apply) {
        cudaStream_t s = ctx->stream;
        k_replay_rank<<<grid_rank, RP_THREADS, 0, s>>>(d_state, buf[0], buf[1], d_table, mask);
        k_replay_setup<<<1, 1, 0, s>>>(d_state, d_rules);
        k_replay_apply<<<grid_apply, RP_THREADS, 0, s>>>(d_state, buf[0], buf[1], d_desc);
    }

    size_t applied_bytes() const { return ((size_t)n_rules + 15) & ~(size_t)15; }

    // Tables for k_replay_segments from a merge list that b200bpe_replay_create has accepted.
    b200bpe_status create_segments(const uint32_t* merges, const std::unordered_map<uint32_t, uint32_t>& made_at) {
        if (n_rules == 0 || n_rules > RS_MAX_RULES) return B200BPE_OK;
        std::vector<uint32_t> join(256 * 256 / 32, 0u);
        uint32_t lg = 4;
        while ((1ull << lg) < (uint64_t)n_rules * 2 + 16) lg++;
        seg.mask = (1u << lg) - 1u;
        std::vector<unsigned long long> table((size_t)1 << lg, 0ull);
        // per rule the first and the last byte of what it makes; a rule over an id that nothing makes never applies, nor do those over its id
        std::vector<int> first(n_rules, -1), last(n_rules, -1);
        for (uint32_t r = 0; r < n_rules; r++) {
            uint32_t t[2];
            int f[2], l[2];
            bool dead = false;
            for (int k = 0; k < 2; k++) {
                const uint32_t id = merges[3 * r + k];
                if (id < 256u) { t[k] = id; f[k] = l[k] = (int)id; continue; }
                const auto it = made_at.find(id);
                if (it == made_at.end() || first[it->second] < 0) { dead = true; break; }
                t[k] = 256u + it->second; f[k] = first[it->second]; l[k] = last[it->second];
            }
            if (dead) continue;
            first[r] = f[0];
            last[r] = l[1];
            const uint32_t j = (uint32_t)l[0] << 8 | (uint32_t)f[1];
            join[j >> 5] |= 1u << (j & 31u);
            const unsigned long long pair = (unsigned long long)t[0] << 21 | t[1];
            uint32_t slot = rs_hash(pair) & seg.mask;
            bool dup = false;
            while (table[slot]) { if ((table[slot] >> 22) == pair) { dup = true; break; } slot = (slot + 1) & seg.mask; }
            if (!dup) table[slot] = pair << 22 | (r + 1u);   // the first rule of a pair wins
        }
        cudaStream_t s = ctx->stream;
        B2_CUDA(cudaMalloc(&d_join, join.size() * 4));
        B2_CUDA(cudaMalloc(&d_seg_table, table.size() * 8));
        B2_CUDA(cudaMallocHost(&h_seg, sizeof(SegmentState)));
        B2_CUDA(cudaMemcpyAsync(d_join, join.data(), join.size() * 4, cudaMemcpyHostToDevice, s));
        B2_CUDA(cudaMemcpyAsync(d_seg_table, table.data(), table.size() * 8, cudaMemcpyHostToDevice, s));
        B2_CUDA(cudaStreamSynchronize(s));
        seg.join = d_join;
        seg.table = d_seg_table;
        seg.rules = d_rules;
        return B200BPE_OK;
    }

    // tokens of `n` bytes (already in d_in or given as a device pointer) → result; returns the count
    b200bpe_status run(const uint8_t* d_bytes, uint64_t n, uint64_t* n_tokens) {
        by_segments = false;
        if (seg.table) {
            const b200bpe_status r = run_segments(d_bytes, n, n_tokens);
            if (r || by_segments) return r;
        }
        return run_rounds(d_bytes, n, n_tokens);
    }

    // by_segments stays false when a segment of the text is too long.
    b200bpe_status run_segments(const uint8_t* d_bytes, uint64_t n, uint64_t* n_tokens) {
        cudaStream_t s = ctx->stream;
        const uint64_t tiles = (n + RS_TILE - 1) / RS_TILE;
        if (n > work_cap) {
            cudaFree(d_work);       // (waits for the device: nothing uses it any more)
            d_work = nullptr;
            work_cap = 0;
            B2_CUDA(cudaMalloc(&d_work, sizeof(SegmentState) + applied_bytes() + (cap / RS_TILE + 1) * 8));
            work_cap = cap;
        }
        SegmentState* st = reinterpret_cast<SegmentState*>(d_work);
        uint8_t* applied = d_work + sizeof(SegmentState);
        unsigned long long* desc = reinterpret_cast<unsigned long long*>(applied + applied_bytes());
        B2_CUDA(cudaMemsetAsync(d_work, 0, sizeof(SegmentState) + applied_bytes() + tiles * 8, s));
        const int grid = (int)std::min<uint64_t>((uint64_t)ctx->sm_count * 8, tiles);
        k_replay_segments<<<grid, RS_THREADS, 0, s>>>(st, d_bytes, n, seg, applied, desc, buf[1]);
        B2_CUDA(cudaGetLastError());
        B2_CUDA(cudaMemcpyAsync(h_seg, st, sizeof(SegmentState), cudaMemcpyDeviceToHost, s));
        B2_CUDA(cudaStreamSynchronize(s));
        if (h_seg->status == 2u) return B200BPE_ERR_LOOKBACK_TIMEOUT;
        if (h_seg->status) return B200BPE_OK;
        by_segments = true;
        result = buf[1];
        *n_tokens = h_seg->n_tokens;
        return B200BPE_OK;
    }

    // Rounds of the last text: with segments, the rules that found something to do (a round applies one).
    b200bpe_status rounds(uint32_t* out) {
        *out = last_rounds;
        if (!by_segments) return B200BPE_OK;
        std::vector<uint8_t> h(n_rules);
        B2_CUDA(cudaSetDevice(ctx->device));
        B2_CUDA(cudaMemcpyAsync(h.data(), d_work + sizeof(SegmentState), n_rules, cudaMemcpyDeviceToHost, ctx->stream));
        B2_CUDA(cudaStreamSynchronize(ctx->stream));
        *out = (uint32_t)std::count(h.begin(), h.end(), (uint8_t)1);
        return B200BPE_OK;
    }

    b200bpe_status run_rounds(const uint8_t* d_bytes, uint64_t n, uint64_t* n_tokens) {
        cudaStream_t s = ctx->stream;
        const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)ctx->sm_count * 8, (n + RP_TILE - 1) / RP_TILE));
        k_replay_bytes<<<grid, RP_THREADS, 0, s>>>(d_bytes, buf[0], n);
        std::memset(h_state, 0, sizeof(ReplayState));
        h_state->n[0] = (uint32_t)n;
        h_state->best_rank = RP_NO_RANK;
        h_state->done = (n_rules == 0 || n < 2) ? 1u : 0u;   // no merges: the bytes are the tokens (tokenizer-manager.js:21-25,46)
        B2_CUDA(cudaMemcpyAsync(d_state, h_state, sizeof(ReplayState), cudaMemcpyHostToDevice, s));
        // the look-back descriptors are tagged with the round number, which restarts here
        B2_CUDA(cudaMemsetAsync(d_desc, 0, (n / RP_TILE + 2) * 8, s));
        if (!graph || graph_cap != cap) {
            if (graph) { cudaGraphExecDestroy(graph); graph = nullptr; }
            const int g_all = (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)ctx->sm_count * 8, (cap + RP_TILE - 1) / RP_TILE));
            cudaGraph_t g = nullptr;
            B2_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            for (int i = 0; i < RP_ROUNDS_PER_GRAPH; i++) enqueue_round(g_all, g_all);
            B2_CUDA(cudaStreamEndCapture(s, &g));
            cudaError_t e = cudaGraphInstantiate(&graph, g, 0);
            cudaGraphDestroy(g);
            B2_CUDA(e);
            graph_cap = cap;
        }
        for (;;) {
            B2_CUDA(cudaGraphLaunch(graph, s));
            B2_CUDA(cudaMemcpyAsync(h_state, d_state, sizeof(ReplayState), cudaMemcpyDeviceToHost, s));
            B2_CUDA(cudaStreamSynchronize(s));
            if (h_state->status) return B200BPE_ERR_LOOKBACK_TIMEOUT;
            if (h_state->done) break;
        }
        last_rounds = h_state->rounds;
        *n_tokens = h_state->n[h_state->epoch & 1];
        result = buf[h_state->epoch & 1];
        return B200BPE_OK;
    }
};

}  // namespace b200bpe

struct b200bpe_replay { b200bpe::Replay* r; };

using namespace b200bpe;

extern "C" {

b200bpe_status b200bpe_replay_create(b200bpe_ctx* c, const uint32_t* merges, uint32_t n_merges, b200bpe_replay** out) {
    if (!c || !out || (!merges && n_merges)) return B200BPE_ERR_BAD_ARG;
    // Rounds by smallest rank equal the reference's rule-by-rule loop only for lists in which every
    // rule makes an id of its own, no byte value among them, and uses only ids made by earlier rules.
    std::unordered_map<uint32_t, uint32_t> made_at;
    for (uint32_t r = 0; r < n_merges; r++) {
        const uint32_t nw = merges[3 * r + 2];
        if (nw < 256u || made_at.count(nw)) { set_last_error("merge list: rule " + std::to_string(r) + " makes an id that is a byte value or already made"); return B200BPE_ERR_BAD_ARG; }
        made_at[nw] = r;
    }
    for (uint32_t r = 0; r < n_merges; r++)
        for (int k = 0; k < 2; k++) {
            auto it = made_at.find(merges[3 * r + k]);
            if (it != made_at.end() && it->second >= r) { set_last_error("merge list: rule " + std::to_string(r) + " uses an id that only a later rule makes"); return B200BPE_ERR_BAD_ARG; }
        }
    B2_CUDA(cudaSetDevice(c->c.device));
    Replay* rp = new Replay();
    rp->ctx = &c->c;
    rp->hold.take(c);
    rp->n_rules = n_merges;
    auto fail = [&](b200bpe_status st) { delete rp; return st; };
    uint32_t lg = 4;
    while ((1ull << lg) < (uint64_t)n_merges * 2 + 16) lg++;
    rp->mask = (1u << lg) - 1u;
    std::vector<RankSlot> table((size_t)1 << lg, RankSlot{0ull, 0u, 0u});
    for (uint32_t r = 0; r < n_merges; r++) {
        unsigned long long key = ((unsigned long long)merges[3 * r] << 32) | merges[3 * r + 1];
        if (!key) key = ~0ull;
        uint32_t x = (uint32_t)key ^ ((uint32_t)(key >> 32) * 0x9E3779B1u);
        x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
        uint32_t slot = x & rp->mask;
        bool dup = false;
        while (table[slot].key != 0ull) { if (table[slot].key == key) { dup = true; break; } slot = (slot + 1) & rp->mask; }
        if (!dup) table[slot] = RankSlot{key, r, merges[3 * r + 2]};   // the first rule of a pair wins (tokenizer-manager.js:31-33)
    }
    cudaStream_t s = c->c.stream;
    if (cudaMalloc(&rp->d_rules, std::max<size_t>(12, (size_t)n_merges * 12)) != cudaSuccess) return fail(B200BPE_ERR_OOM);
    if (cudaMalloc(&rp->d_table, table.size() * sizeof(RankSlot)) != cudaSuccess) return fail(B200BPE_ERR_OOM);
    if (cudaMalloc(&rp->d_state, sizeof(ReplayState)) != cudaSuccess) return fail(B200BPE_ERR_OOM);
    if (cudaMallocHost(&rp->h_state, sizeof(ReplayState)) != cudaSuccess) return fail(B200BPE_ERR_OOM);
    if (n_merges && cudaMemcpyAsync(rp->d_rules, merges, (size_t)n_merges * 12, cudaMemcpyHostToDevice, s) != cudaSuccess) return fail(B200BPE_ERR_CUDA);
    if (cudaMemcpyAsync(rp->d_table, table.data(), table.size() * sizeof(RankSlot), cudaMemcpyHostToDevice, s) != cudaSuccess) return fail(B200BPE_ERR_CUDA);
    if (cudaStreamSynchronize(s) != cudaSuccess) return fail(B200BPE_ERR_CUDA);
    const b200bpe_status r = rp->create_segments(merges, made_at);
    if (r) return fail(r);
    *out = new b200bpe_replay{rp};
    return B200BPE_OK;
}

b200bpe_status b200bpe_replay_encode(b200bpe_replay* h, const uint8_t* bytes, uint64_t n, uint32_t* tokens_out, uint64_t cap,
                                     uint64_t* n_tokens_out) {
    if (!h || (!bytes && n) || !n_tokens_out) return B200BPE_ERR_BAD_ARG;
    Replay* rp = h->r;
    *n_tokens_out = 0;
    if (n == 0) return B200BPE_OK;
    if (n >= 0xFFFFFFF0ull) return B200BPE_ERR_BAD_ARG;
    B2_CUDA(cudaSetDevice(rp->ctx->device));
    b200bpe_status r = rp->ensure(n);
    if (r) return r;
    cudaStream_t s = rp->ctx->stream;
    B2_CUDA(cudaMemcpyAsync(rp->d_in, bytes, n, cudaMemcpyHostToDevice, s));
    uint64_t nt = 0;
    if ((r = rp->run(rp->d_in, n, &nt))) return r;
    *n_tokens_out = nt;
    if (nt > cap || (!tokens_out && nt)) return B200BPE_ERR_CAPACITY;
    B2_CUDA(cudaMemcpyAsync(tokens_out, rp->result, nt * 4, cudaMemcpyDeviceToHost, s));
    B2_CUDA(cudaStreamSynchronize(s));
    return B200BPE_OK;
}

b200bpe_status b200bpe_replay_encode_device(b200bpe_replay* h, const uint8_t* d_bytes, uint64_t n, uint32_t* d_tokens_out,
                                            uint64_t cap, uint64_t* n_tokens_out) {
    if (!h || (!d_bytes && n) || !n_tokens_out) return B200BPE_ERR_BAD_ARG;
    Replay* rp = h->r;
    *n_tokens_out = 0;
    if (n == 0) return B200BPE_OK;
    if (n >= 0xFFFFFFF0ull) return B200BPE_ERR_BAD_ARG;
    B2_CUDA(cudaSetDevice(rp->ctx->device));
    b200bpe_status r = rp->ensure(n);
    if (r) return r;
    uint64_t nt = 0;
    if ((r = rp->run(d_bytes, n, &nt))) return r;
    *n_tokens_out = nt;
    if (nt > cap || (!d_tokens_out && nt)) return B200BPE_ERR_CAPACITY;
    B2_CUDA(cudaMemcpyAsync(d_tokens_out, rp->result, nt * 4, cudaMemcpyDeviceToDevice, rp->ctx->stream));
    B2_CUDA(cudaStreamSynchronize(rp->ctx->stream));
    return B200BPE_OK;
}

b200bpe_status b200bpe_replay_last_rounds(b200bpe_replay* h, uint32_t* rounds) {
    if (!h || !rounds) return B200BPE_ERR_BAD_ARG;
    return h->r->rounds(rounds);
}

void b200bpe_replay_destroy(b200bpe_replay* h) {
    if (!h) return;
    delete h->r;
    delete h;
}

}  // extern "C"
