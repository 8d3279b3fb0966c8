// The merge loop on the dictionary of word_dict.cuh: one kernel launch runs a whole batch of merges.
//
// What a merge has to touch is small: the occurrences of one pair among the distinct words (a few hundred late in a run), found
// without looking at anything else, because of two facts.  An occurrence of pair (x, y) comes into being when the younger of its
// symbols is made, so the occurrences of all pairs whose younger symbol is m are written, once, by merge m: a list of (position of
// the left symbol, pair), and the merge that takes (x, y) reads the list of max(x, y) and keeps the entries of its own pair.
// Byte pairs have exact lists of their own (k_dict_lists).  And a pair's count never rises after the merge that made it, so the
// arg-max needs only the pairs above a threshold: a candidate list made by a scan of the pair table, to which a merge adds the
// new pairs that reach the threshold; when the best candidate falls below it, the table is scanned again.  ("literal" runs, whose text's
// tail is kept by itself, can raise a count again: a rise across the threshold makes a candidate whenever it happens.)
//
// What bounds a merge is then a chain of dependent memory round trips (occurrence list -> records -> pair table -> candidates'
// counts), and the barriers between its two phases, not bandwidth.  So the loop runs inside ONE thread-block cluster: 16 CTAs on
// 16 SMs, whose hardware barrier costs a fraction of a grid-wide one, with the arg-max exchanged through distributed shared
// memory.  Against full passes over the symbol buffers (train_kernels.cuh, which sharded runs take): 64 MiB,
// 8,000 merges 522 -> 64 ms; heavy-tailed 256 MiB, 4,000 merges 1,326 -> 70 ms.
// Phase 1 finds and verifies the occurrences (all reads see the state before the merge), updates the pair table and
// writes the list of the new symbol; phase 2 rewrites the records and takes the arg-max of the next merge.
#pragma once

#include <cooperative_groups.h>

#include "word_dict.cuh"

namespace b200bpe {

constexpr int WM_THREADS = 512;
constexpr int WM_CLUSTER = 16;             // CTAs (the largest cluster the hardware takes)
constexpr int WM_QUEUE = 6144;             // occurrences a CTA keeps in shared memory between the phases
constexpr int WM_UNROLL = 8;               // list entries a thread has in flight
constexpr int WM_CAND = 2048;              // candidates per CTA
constexpr uint32_t WM_CAND_GOAL = 6000;    // candidates a scan aims at, all CTAs together
constexpr int WM_BINS = 256;
constexpr int WM_MAX_PROBE = 4096;

// Why the loop stopped (WordState::status).
enum : uint32_t { WS_OK = 0, WS_GROW = 1u, WS_FULL = 2u, WS_CAND = 4u, WS_TAIL = 8u };

struct __align__(16) WordState {
    unsigned long long tau;      // threshold of the candidate list, as count << 32 | ~pair; ~0 = no list
    unsigned long long best;     // best pair of the present table, if best_valid
    unsigned long long touched;  // bytes of occurrence lists and tails that the merges went through (statistics)
    uint32_t best_valid;
    uint32_t merges_done;
    uint32_t next_id;
    uint32_t early_stop;
    uint32_t status;
    uint32_t entries;            // list entries written so far
    uint32_t occupied;           // pair table slots in use
    uint32_t symbols;            // live symbols of the corpus
    uint32_t scans;              // table scans so far (statistics)
    uint32_t front, front_before;   // "literal" runs: symbols of the dictionary's part, now and before the last merge
    uint32_t turn;               // and merges so far, which say which tail buffer is which
};

struct WordArgs {
    uint32_t* rec;                    // the dictionary's positions
    const uint32_t* weight;
    const uint32_t* byte_list;        // occurrences of the byte pairs
    const uint32_t* byte_off;
    uint2* entries;                   // {position of the left symbol, left << 16 | right}, room for 2 * positions
    uint2* segment;                   // [symbol] = {first entry, end}
    uint32_t* usual;                  // [symbol] = positions it usually covers (always, but for symbols made of a run of equal ones)
    uint32_t positions;               // rec[positions] begins a word, and nothing lies behind it
    unsigned long long* table;        // pair << 32 | count, pair = left << 16 | right, never 0
    uint32_t table_log2;
    uint32_t* cand;                   // candidates between launches: [WM_CLUSTER][WM_CAND + 1], count first
    uint32_t* tail[3];                // "literal" runs: the symbols behind the dictionary's words
    WordState* st;
    uint4* log;                       // {a, b, new_id, count} per merge
};

struct WordShared {
    uint2 queue[WM_QUEUE];            // {position (~0: not an occurrence), spans}
    uint32_t cand[WM_CAND];
    uint32_t hist[WM_BINS];
    unsigned long long xbest[WM_CLUSTER];
    uint32_t xflags[WM_CLUSTER];
    unsigned long long wbest[WM_THREADS / 32];
    uint32_t queued, ncand, flags, inserted;
    uint32_t c_entries, c_inserted, c_merged, c_spilled;   // the cluster's counters: those of CTA 0 are the ones in use
    uint32_t kept[WM_CLUSTER * WM_THREADS / 32];          // tail symbols that every warp of the cluster copies
    uint32_t tail_queue[4096], tail_queued;               // matches in this CTA's part of the tail
    WordState init;
};

__device__ __forceinline__ uint32_t wt_hash(uint32_t key) {
    uint32_t x = key * 0x9E3779B1u;
    x ^= x >> 15;
    return x * 0x85EBCA77u;
}
__device__ __forceinline__ unsigned long long wt_rank(unsigned long long slot) {   // order of the arg-max: larger count, then smaller pair
    return (slot << 32) | (uint32_t)~(uint32_t)(slot >> 32);
}
__device__ __forceinline__ unsigned long long warp_max64(unsigned long long v) {
    const uint32_t hi = (uint32_t)(v >> 32);
    const uint32_t mh = __reduce_max_sync(0xFFFFFFFFu, hi);
    const uint32_t ml = __reduce_max_sync(0xFFFFFFFFu, hi == mh ? (uint32_t)v : 0u);
    return (unsigned long long)mh << 32 | ml;
}
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Puts a pair with its count into the table (set-up and growth; the pair is not there yet).  False: no room.
__device__ __forceinline__ bool wt_insert(unsigned long long* __restrict__ table, uint32_t log2, unsigned long long slot) {
    const uint32_t mask = (1u << log2) - 1u;
    uint32_t s = wt_hash((uint32_t)(slot >> 32)) >> (32u - log2);
    for (int p = 0; p < WM_MAX_PROBE; p++) {
        if (__ldcg(table + s) == 0ull && atomicCAS(table + s, 0ull, slot) == 0ull) return true;
        s = (s + 1u) & mask;
    }
    return false;
}
// The byte pairs of the corpus, and the control block of a fresh run.
__global__ void __launch_bounds__(256)
k_word_init(const unsigned long long* __restrict__ bins, const DictState* __restrict__ ds, unsigned long long* __restrict__ table, uint32_t log2,
            WordState* __restrict__ st, uint32_t first_id, uint32_t n, uint32_t front) {
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;      // 65,536 threads
    const unsigned long long v = bins[i];
    const uint32_t pair = (i >> 8) << 16 | (i & 0xFFu);
    if (v && !wt_insert(table, log2, (unsigned long long)pair << 32 | (uint32_t)v)) atomicOr(&st->status, (uint32_t)WS_FULL);
    if (i == 0) {
        st->tau = ~0ull;
        st->next_id = first_id;
        st->symbols = n;
        st->front = st->front_before = front;
        st->occupied = ds->pairs;
    }
}
// Copies the pairs that still occur into a larger table.
__global__ void __launch_bounds__(256)
k_word_rehash(const unsigned long long* __restrict__ from, uint32_t from_log2, unsigned long long* __restrict__ to, uint32_t to_log2, WordState* __restrict__ st) {
    uint32_t kept = 0;
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < 1u << from_log2; i += gridDim.x * 256) {
        const unsigned long long v = from[i];
        if ((uint32_t)v == 0u) continue;
        if (!wt_insert(to, to_log2, v)) atomicOr(&st->status, (uint32_t)WS_FULL);
        kept++;
    }
    if (kept) atomicAdd(&st->occupied, kept);
}
__global__ void k_word_regrown(WordState* st) { st->status = WS_OK; st->occupied = 0u; st->tau = ~0ull; st->best_valid = 0u; }
// Read-back of the pair counts.
__global__ void __launch_bounds__(256)
k_word_dump(const unsigned long long* __restrict__ table, uint32_t log2, unsigned long long* __restrict__ keys, uint32_t* __restrict__ counts, uint32_t cap,
            uint32_t* __restrict__ n) {
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < 1u << log2; i += gridDim.x * 256) {
        const unsigned long long v = table[i];
        if ((uint32_t)v == 0u) continue;
        const uint32_t k = atomicAdd(n, 1u), pair = (uint32_t)(v >> 32);
        if (k < cap) { keys[k] = (unsigned long long)(pair >> 16) << 32 | (pair & 0xFFFFu); counts[k] = (uint32_t)v; }
    }
}

struct WordTeam {
    WordShared& s;
    WordShared* lead;            // CTA 0's shared memory
    uint32_t rank, tid;
    cooperative_groups::cluster_group cluster;
};

// Count updates of up to N pairs by one thread, in step: their probes, insertions and adds are in flight together.  One after the other they
// were 6,000 of the 10,000 cycles of phase 1, and most of the wait at the barrier behind it: 64 MiB, 8,000 merges 85 -> 65 ms.
// wanted: bit k = pair[k] changes by w[k]; rise: bit k = upwards.  `tau` as in WordState; a rise across it makes the slot a candidate of
// this CTA.
template <int N>
__device__ __forceinline__ void wt_updates(const WordArgs& A, WordTeam& T, const uint32_t (&pair)[N], const uint32_t (&w)[N], uint32_t wanted, uint32_t rise,
                                           unsigned long long tau) {
    const uint32_t mask = (1u << A.table_log2) - 1u, sh = 32u - A.table_log2;
    uint32_t slot[N];
    unsigned long long seen[N];
#pragma unroll
    for (int k = 0; k < N; k++) {
        slot[k] = wt_hash(pair[k]) >> sh;
        seen[k] = (wanted >> k) & 1u ? __ldcg(A.table + slot[k]) : 0ull;
    }
    auto candidate = [&](uint32_t at) {
        const uint32_t i = atomicAdd(&T.s.ncand, 1u);
        if (i < WM_CAND) T.s.cand[i] = at; else atomicOr(&T.s.flags, (uint32_t)WS_CAND);
    };
    uint32_t open = wanted, found = 0u;
    for (int p = 0; open && p < WM_MAX_PROBE; p++) {
        uint32_t tried = 0u;
#pragma unroll
        for (int k = 0; k < N; k++) {
            if (((open >> k) & 1u) && seen[k] == 0ull) {
                if ((rise >> k) & 1u) { seen[k] = atomicCAS(A.table + slot[k], 0ull, (unsigned long long)pair[k] << 32 | w[k]); tried |= 1u << k; }
                else { atomicOr(&T.s.flags, (uint32_t)WS_FULL); open &= ~(1u << k); }       // a pair that occurs is in the table
            }
        }
#pragma unroll
        for (int k = 0; k < N; k++) {
            if (!((open >> k) & 1u)) continue;
            if (((tried >> k) & 1u) && seen[k] == 0ull) {                                   // inserted
                open &= ~(1u << k);
                atomicAdd(&T.s.inserted, 1u);
                if (wt_rank((unsigned long long)pair[k] << 32 | w[k]) >= tau) candidate(slot[k]);
            } else if ((uint32_t)(seen[k] >> 32) == pair[k]) {
                open &= ~(1u << k);
                found |= 1u << k;
            } else {
                slot[k] = (slot[k] + 1u) & mask;
                seen[k] = __ldcg(A.table + slot[k]);
            }
        }
    }
    if (open) atomicOr(&T.s.flags, (uint32_t)WS_FULL);
    int old[N];
#pragma unroll
    for (int k = 0; k < N; k++) {
        old[k] = 0;
        if (!((found >> k) & 1u)) continue;
        uint32_t* count = reinterpret_cast<uint32_t*>(A.table + slot[k]);   // the lower half
        if ((rise >> k) & 1u) old[k] = (int)atomicAdd(count, w[k]); else atomicSub(count, w[k]);
    }
#pragma unroll
    for (int k = 0; k < N; k++) {
        if (!((found & rise) >> k & 1u)) continue;
        // (in a "literal" run the rises and falls of a merge come in any order, so that a count can be below 0 on the way)
        const int now = old[k] + (int)w[k];
        const unsigned long long low = (uint32_t)~pair[k];
        if (now > 0 && ((unsigned long long)max(old[k], 0) << 32 | low) < tau && ((unsigned long long)now << 32 | low) >= tau) candidate(slot[k]);
    }
}
__device__ __forceinline__ void wt_update(const WordArgs& A, WordTeam& T, uint32_t pair, uint32_t w, bool rise, unsigned long long tau) {
    const uint32_t k[1] = {pair}, v[1] = {w};
    wt_updates<1>(A, T, k, v, 1u, rise ? 1u : 0u, tau);
}

// Best candidate of the cluster and the CTAs' flags; ends with the cluster barrier that also publishes phase 2's writes.
__device__ __forceinline__ void word_argmax(const WordArgs& A, WordTeam& T, unsigned long long& best, uint32_t& flags) {
    unsigned long long mine = 0ull;
    const uint32_t n = min(T.s.ncand, (uint32_t)WM_CAND);
    for (uint32_t i = T.tid; i < n; i += WM_THREADS) {
        const unsigned long long v = __ldcg(A.table + T.s.cand[i]);
        const unsigned long long r = (uint32_t)v ? wt_rank(v) : 0ull;
        mine = r > mine ? r : mine;
    }
    mine = warp_max64(mine);
    if ((T.tid & 31) == 0) T.s.wbest[T.tid >> 5] = mine;
    __syncthreads();
    if (T.tid < 32) {
        mine = warp_max64(T.tid < WM_THREADS / 32 ? T.s.wbest[T.tid] : 0ull);
        if (T.tid < WM_CLUSTER) {
            WordShared* to = T.cluster.map_shared_rank(&T.s, T.tid);
            to->xbest[T.rank] = mine;
            to->xflags[T.rank] = T.s.flags;
        }
        if (T.tid == 0) T.s.queued = 0u;
    }
    cluster_barrier();
    const uint32_t lane = T.tid & 31;
    best = warp_max64(lane < WM_CLUSTER ? T.s.xbest[lane] : 0ull);
    flags = __reduce_or_sync(0xFFFFFFFFu, lane < WM_CLUSTER ? T.s.xflags[lane] : 0u);
}

// Scan of the pair table: picks a threshold that about WM_CAND_GOAL pairs (of count 2 or more) reach and lists them.  A first
// pass bins the counts by their leading bits (8 bins per power of two); where a single bin holds more pairs than wanted (small
// counts: many ties) further passes split it, down to the single pair.  Every CTA takes the same decisions from CTA 0's bins.
__device__ __noinline__ void word_scan(const WordArgs& A, WordTeam& T, unsigned long long& tau) {
    const uint32_t slots = 1u << A.table_log2;
    const uint32_t first = T.tid * WM_CLUSTER + T.rank;
    unsigned long long lo = 2ull << 32, hi = ~0ull;      // ranks of the pairs still to be split: [lo, hi]
    uint32_t above = 0;                                   // pairs known to lie above hi
    for (int level = 0; level < 12; level++) {
        // bins of this pass: level 0 by leading bits of the count, then linear with 2^shift ranks each
        uint32_t shift = 0;
        if (level) while (((hi - lo) >> shift) >= WM_BINS) shift++;
        auto bin_of = [&](unsigned long long r) -> uint32_t {
            if (level) return (uint32_t)((r - lo) >> shift);
            const uint32_t c = (uint32_t)(r >> 32), e = 31u - (uint32_t)__clz((int)c);
            return e * 8u + (e >= 3u ? (c >> (e - 3u)) & 7u : (c << (3u - e)) & 7u);
        };
        for (uint32_t i = T.tid; i < WM_BINS; i += WM_THREADS) T.s.hist[i] = 0u;
        cluster_barrier();
        uint32_t* sums = T.lead->hist;
        for (uint32_t i = first; i < slots; i += WM_THREADS * WM_CLUSTER * 4) {
            unsigned long long v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) { const uint32_t j = i + k * WM_THREADS * WM_CLUSTER; v[k] = j < slots ? __ldcg(A.table + j) : 0ull; }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const unsigned long long r = wt_rank(v[k]);
                if ((uint32_t)v[k] >= 2u && r >= lo && r <= hi) atomicAdd(T.s.hist + bin_of(r), 1u);
            }
        }
        __syncthreads();
        // CTA 0's bins collect everybody's (its own are there already)
        if (T.rank != 0) for (uint32_t i = T.tid; i < WM_BINS; i += WM_THREADS) if (T.s.hist[i]) atomicAdd(sums + i, T.s.hist[i]);
        cluster_barrier();
        // from the top: the lowest bin down to which the list stays within the goal
        uint32_t total = above, bin = WM_BINS;
        __shared__ uint32_t s_bin, s_total;
        if (T.tid == 0) {
            while (bin > 0) {
                const uint32_t h = sums[bin - 1];
                if (total + h > WM_CAND_GOAL) break;
                total += h;
                bin--;
            }
            s_bin = bin;
            s_total = total;
        }
        __syncthreads();
        bin = s_bin;
        total = s_total;
        cluster_barrier();          // CTA 0's bins may be cleared again
        auto low_of = [&](uint32_t b) -> unsigned long long {
            if (level) return lo + ((unsigned long long)b << shift);
            const uint32_t e = b >> 3, m = b & 7u;
            return (unsigned long long)(e >= 3u ? (8u + m) << (e - 3u) : ((8u + m) >> (3u - e))) << 32;
        };
        if (bin == 0) { tau = lo; break; }
        const unsigned long long cut = low_of(bin);
        if (total >= WM_CAND_GOAL / 8 || (level && shift == 0)) { tau = cut < lo ? lo : cut; break; }
        // too few above the cut: split the bin below it
        above = total;
        const unsigned long long b_lo = low_of(bin - 1);
        if (cut - 1 < hi && bin < WM_BINS) hi = cut - 1;
        if (b_lo > lo) lo = b_lo;
        tau = lo;
    }
    if (T.tid == 0) { T.s.ncand = 0u; T.s.flags &= ~(uint32_t)WS_CAND; }
    __syncthreads();
    for (uint32_t i = first; i < slots; i += WM_THREADS * WM_CLUSTER * 4) {
        unsigned long long v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) { const uint32_t j = i + k * WM_THREADS * WM_CLUSTER; v[k] = j < slots ? __ldcg(A.table + j) : 0ull; }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if ((uint32_t)v[k] >= 2u && wt_rank(v[k]) >= tau) {
                const uint32_t c = atomicAdd(&T.s.ncand, 1u);
                if (c < WM_CAND) T.s.cand[c] = i + k * WM_THREADS * WM_CLUSTER; else atomicOr(&T.s.flags, (uint32_t)WS_CAND);
            }
        }
    }
    __syncthreads();
}

// ── the tail of a "literal" run ──
// "literal" compaction bounds its INPUT by the post-merge count (train.wgsl:698,727), so a merge of count c drops the last c symbols and
// leaves as many positions to what the destination held two merges ago.  Everything this ever touches lies near the end of the text:
// the dictionary takes the words of its front, where a merge does what it does in "fixed" mode, and the symbols behind them are kept one
// by one, in three buffers that take turns (this merge's source, the one before it, the destination).  `symbols` counts both parts; the
// tail's first symbol begins a word and is never dropped.  A merge that reaches past the tail ends the run here (WS_TAIL): the symbol
// buffers then take it from its start.
//
// A merge reads the tail twice: phase 1 counts what every warp's share keeps and updates the pairs that change; phase 2, with every
// offset known, writes the destination, rewrites the source in place as the reference does (train.wgsl:486-487: the next merge but one may see it),
// and copies the older symbols in.  The pairs' counts can rise here at any time, unlike the dictionary's.
// What bounds it: the round trip of a span's loads (the next span's are on their way meanwhile) and, where matches are many, the updates of
// the pairs around them.  Whole runs, us a merge: 64 KiB 15.5 -> 11.0, 1 MiB 17.3 -> 12.1 with the next span fetched ahead, shares dealt
// round the CTAs, and matches and single updates worked on beside the dictionary's occurrences; on the symbol buffers 36 and 31.
struct TailView {
    const uint32_t* cur;
    uint32_t n, limit;           // its symbols; the first `limit` are copied
    uint32_t a, b, fresh;
};
__device__ __forceinline__ bool tail_counted(uint32_t l, uint32_t r) { return !(r & WORD_START_BIT) && (l & TOKEN_MASK) && (r & TOKEN_MASK); }
// A source symbol as it was before this merge (the new id does not occur otherwise).
__device__ __forceinline__ uint32_t tail_before(const TailView& v, uint32_t s) { return (s & TOKEN_MASK) == v.fresh ? (s & WORD_START_BIT) | v.a : s; }
__device__ __forceinline__ bool tail_match(const TailView& v, uint32_t l, uint32_t r) {
    return (l & TOKEN_MASK) == v.a && (r & (TOKEN_MASK | WORD_START_BIT)) == v.b;
}
__device__ __forceinline__ uint32_t tail_at(const TailView& v, uint32_t i) {      // beyond the end: a word start, which ends everything
    return i < v.n ? tail_before(v, __ldcg(v.cur + i)) : WORD_START_BIT;
}
__device__ __forceinline__ void tail_pair(const WordArgs& A, WordTeam& T, uint32_t l, uint32_t r, bool rise, unsigned long long tau) {
    const uint32_t pair = (l & TOKEN_MASK) << 16 | (r & TOKEN_MASK);
    wt_update(A, T, pair, 1u, rise, tau);
}
// The changes at position i < limit: the pair that begins there goes unless it is copied as it is (from limit - 1 on all pairs go: tail_pairs);
// what the symbol there is copied next to comes.
__device__ __forceinline__ void tail_changes(const WordArgs& A, WordTeam& T, const TailView& v, uint32_t i, unsigned long long tau) {
    const uint32_t sm = i > 0u ? tail_at(v, i - 1u) : WORD_START_BIT, s0 = tail_at(v, i), s1 = tail_at(v, i + 1u), s2 = tail_at(v, i + 2u);
    const bool ml = i > 0u && tail_match(v, sm, s0), mi = tail_match(v, s0, s1), mr = tail_match(v, s1, s2);
    if (tail_counted(s0, s1) && i + 1u < v.limit && (ml || mi || mr)) tail_pair(A, T, s0, s1, false, tau);
    if (ml) return;
    uint32_t j = i + 1u, before = s0, s = s1;
    while (tail_match(v, before, s)) { before = s; s = tail_at(v, ++j); }
    if (j >= v.limit) return;              // (what the last copied symbol ends up next to is known in phase 2)
    const bool mj = tail_match(v, s, tail_at(v, j + 1u));
    if (!(mi || mj)) return;
    const uint32_t l = mi ? v.fresh : s0, r = mj ? (s & WORD_START_BIT) | v.fresh : s;
    if (tail_counted(l, r)) tail_pair(A, T, l, r, true, tau);
}
// The same for all positions around a match at m < limit that no earlier match sees to, with everything in flight together.
__device__ __forceinline__ void tail_match_changes(const WordArgs& A, WordTeam& T, const TailView& v, uint32_t m, unsigned long long tau) {
    uint32_t t[7];          // symbols m - 2 .. m + 4
#pragma unroll
    for (int k = 0; k < 7; k++) t[k] = m + k >= 2u ? tail_at(v, m + k - 2u) : WORD_START_BIT;
    const bool m2 = m >= 2u && tail_match(v, t[0], t[1]), m1 = m >= 1u && tail_match(v, t[1], t[2]);     // at m - 2, m - 1
    const bool n1 = tail_match(v, t[3], t[4]), n2 = tail_match(v, t[4], t[5]);                            // at m + 1, m + 2
    if (v.a == v.b) {       // runs of any length
        tail_changes(A, T, v, m, tau);
        if (!n1) { if (m + 1u < v.limit) tail_changes(A, T, v, m + 1u, tau); }
        if (m >= 1u && !m1 && !m2) tail_changes(A, T, v, m - 1u, tau);
        return;
    }
    // (a != b: a match is never next to another one; m + 2 may be the next)
    const bool before = m >= 1u && !m2;                     // position m - 1 is this match's to see to
    uint32_t pair[5], wanted = 0u;
    const uint32_t one[5] = {1u, 1u, 1u, 1u, 1u};
    auto put = [&](int k, uint32_t l, uint32_t r, bool yes) {
        pair[k] = (l & TOKEN_MASK) << 16 | (r & TOKEN_MASK);
        if (yes && tail_counted(l, r)) wanted |= 1u << k;
    };
    put(0, t[1], t[2], before && m < v.limit);              // falls
    put(1, t[2], t[3], m + 1u < v.limit);
    put(2, t[3], t[4], m + 2u < v.limit);
    put(3, t[1], (t[2] & WORD_START_BIT) | v.fresh, before);                                             // rises
    put(4, v.fresh, n2 ? (t[4] & WORD_START_BIT) | v.fresh : t[4], m + 2u < v.limit);
    wt_updates<5>(A, T, pair, one, wanted, 24u, tau);
}
// The tail goes by in spans of TAIL_SPAN symbols: four 16-byte loads per lane.  match: bit 4 u + k = a pair begins at symbol k of the lane's
// u-th four; left: one begins right before the span.
constexpr uint32_t TAIL_SPAN = 512;
constexpr uint32_t TAIL_QUEUE = 4096;
struct TailSpan { uint4 q[4]; uint32_t edge, match; bool left; };
__device__ __forceinline__ void tail_fetch(const TailView& v, uint32_t base, uint32_t lane, TailSpan& t) {
    if (base + TAIL_SPAN <= v.limit) {          // (behind the limit the rewrite is under way in phase 2)
        const uint4* __restrict__ p = reinterpret_cast<const uint4*>(v.cur + base) + lane;
#pragma unroll
        for (int u = 0; u < 4; u++) t.q[u] = __ldcg(p + u * 32);
    } else {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t i = base + u * 128u + lane * 4u;
            t.q[u] = make_uint4(tail_at(v, i), tail_at(v, i + 1u), tail_at(v, i + 2u), tail_at(v, i + 3u));
        }
    }
    t.edge = 0u;
    if (lane < 2u) t.edge = lane == 0u ? (base > 0u ? tail_at(v, base - 1u) : WORD_START_BIT) : tail_at(v, base + TAIL_SPAN);
}
__device__ __forceinline__ void tail_decide(const TailView& v, uint32_t lane, TailSpan& t) {
    const uint32_t before = __shfl_sync(0xFFFFFFFFu, t.edge, 0), behind = __shfl_sync(0xFFFFFFFFu, t.edge, 1);
    t.match = 0u;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        uint32_t nx = __shfl_down_sync(0xFFFFFFFFu, t.q[u].x, 1);
        const uint32_t far = u < 3 ? __shfl_sync(0xFFFFFFFFu, t.q[u < 3 ? u + 1 : u].x, 0) : behind;
        if (lane == 31) nx = far;
        t.match |= (tail_match(v, t.q[u].x, t.q[u].y) ? 1u : 0u) << (4 * u) | (tail_match(v, t.q[u].y, t.q[u].z) ? 2u : 0u) << (4 * u) |
                   (tail_match(v, t.q[u].z, t.q[u].w) ? 4u : 0u) << (4 * u) | (tail_match(v, t.q[u].w, nx) ? 8u : 0u) << (4 * u);
    }
    t.left = tail_match(v, before, __shfl_sync(0xFFFFFFFFu, t.q[0].x, 0));
}
// Phase 1 over [from, to), whole spans but for the last: queues the matches, and returns how many symbols are copied (the same in every lane).
__device__ __forceinline__ uint32_t tail_count(const WordArgs& A, WordTeam& T, const TailView& v, uint32_t from, uint32_t to, unsigned long long tau) {
    const uint32_t lane = T.tid & 31;
    uint32_t kept = to - from;
    TailSpan t, ahead;               // the next span is on its way while this one is worked on
    if (from < to) tail_fetch(v, from, lane, ahead);
    for (uint32_t span = from; span < to; span += TAIL_SPAN) {
        t = ahead;
        if (span + TAIL_SPAN < to) tail_fetch(v, span + TAIL_SPAN, lane, ahead);
        tail_decide(v, lane, t);
        const uint32_t end = to - span;           // symbols of the span that are in question
        uint32_t match = t.match, drops = 0u;
        if (end < TAIL_SPAN) {
#pragma unroll
            for (int k = 0; k < 16; k++) if ((uint32_t)(k / 4) * 128u + lane * 4u + k % 4 >= end) match &= ~(1u << k);
        }
        if (__any_sync(0xFFFFFFFFu, match != 0u)) {
            // what a match drops is the symbol behind it, if that is still in question
            const uint32_t last = span + TAIL_SPAN < to ? TAIL_SPAN : end;
            drops = __popc(match);
            const uint32_t at_end = last - 1u;    // (the position whose successor belongs to the next span or warp)
            if (at_end % 128u / 4u == lane && ((match >> (at_end / 128u * 4u + at_end % 4u)) & 1u)) drops--;
            drops = __reduce_add_sync(0xFFFFFFFFu, drops);
            while (match) {
                const uint32_t k = (uint32_t)__ffs((int)match) - 1u, m = span + k / 4u * 128u + lane * 4u + k % 4u;
                match &= match - 1u;
                const uint32_t i = atomicAdd(&T.s.tail_queued, 1u);
                if (i < TAIL_QUEUE) T.s.tail_queue[i] = m; else tail_match_changes(A, T, v, m, tau);
            }
            __syncwarp();
        }
        kept -= drops + (t.left ? 1u : 0u);
    }
    return kept;
}
// Pairs of neighbours among `n` symbols at s (with the one behind them): all of them go, or come; several in flight per thread.
__device__ __forceinline__ void tail_pairs(const WordArgs& A, WordTeam& T, const uint32_t* __restrict__ s, uint32_t n, uint32_t first, bool rise,
                                           unsigned long long tau, uint32_t* __restrict__ copy) {
    constexpr int U = 4;
    constexpr uint32_t STEP = WM_THREADS * WM_CLUSTER;
    for (uint32_t i0 = first; i0 < n; i0 += STEP * U) {
        uint32_t l[U], r[U], pair[U], wanted = 0u;
        const uint32_t one[U] = {1u, 1u, 1u, 1u};
#pragma unroll
        for (int k = 0; k < U; k++) {
            const uint32_t i = i0 + k * STEP;
            l[k] = i < n ? __ldcg(s + i) : 0u;
            r[k] = i + 1u < n ? __ldcg(s + i + 1u) : WORD_START_BIT;
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
            pair[k] = (l[k] & TOKEN_MASK) << 16 | (r[k] & TOKEN_MASK);
            if (tail_counted(l[k], r[k])) wanted |= 1u << k;
            if (copy && i0 + k * STEP < n) copy[i0 + k * STEP] = l[k];
        }
        wt_updates<U>(A, T, pair, one, wanted, rise ? 15u : 0u, tau);
    }
}
// Phase 2 over [from, to): what is copied goes to dst[out...], and the source gets this merge's rewrite.
__device__ __forceinline__ void tail_move(const TailView& v, uint32_t* src, uint32_t* __restrict__ dst, uint32_t from, uint32_t to, uint32_t out, uint32_t lane) {
    TailSpan t, ahead;
    if (from < to) tail_fetch(v, from, lane, ahead);
    for (uint32_t span = from; span < to; span += TAIL_SPAN) {
        t = ahead;
        if (span + TAIL_SPAN < to) tail_fetch(v, span + TAIL_SPAN, lane, ahead);
        tail_decide(v, lane, t);
        if (span + TAIL_SPAN <= to && !__any_sync(0xFFFFFFFFu, t.match != 0u || t.left)) {
            // nothing changes: whole 16-byte stores; element `shift` of every lane's four lies on a 16-byte boundary of the destination
            const uint32_t shift = (0u - out) & 3u;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint4 a = t.q[u];
                uint4 b;
                b.x = __shfl_down_sync(0xFFFFFFFFu, a.x, 1); b.y = __shfl_down_sync(0xFFFFFFFFu, a.y, 1); b.z = __shfl_down_sync(0xFFFFFFFFu, a.z, 1);
                const uint4 n0 = t.q[u < 3 ? u + 1 : u];
                const uint32_t fx = __shfl_sync(0xFFFFFFFFu, n0.x, 0), fy = __shfl_sync(0xFFFFFFFFu, n0.y, 0), fz = __shfl_sync(0xFFFFFFFFu, n0.z, 0);
                if (lane == 31) { b.x = fx; b.y = fy; b.z = fz; }
                uint32_t* o = dst + out + u * 128u + lane * 4u;
                if (u == 0 && lane == 0) { if (shift > 0u) o[0] = a.x; if (shift > 1u) o[1] = a.y; if (shift > 2u) o[2] = a.z; }
                if (u == 3 && lane == 31 && shift) {      // what does not fill a store
                    if (shift == 1u) o[1] = a.y;
                    if (shift <= 2u) o[2] = a.z;
                    o[3] = a.w;
                } else {
                    const uint4 w = shift == 0u ? a : shift == 1u ? make_uint4(a.y, a.z, a.w, b.x) : shift == 2u ? make_uint4(a.z, a.w, b.x, b.y)
                                                                                                               : make_uint4(a.w, b.x, b.y, b.z);
                    *reinterpret_cast<uint4*>(o + shift) = w;
                }
            }
            out += TAIL_SPAN;
            continue;
        }
        bool carry = t.left;          // the symbol before this lane's four is the first of a pair
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t i = span + u * 128u + lane * 4u, m = (t.match >> (4 * u)) & 15u;
            uint32_t before = __shfl_up_sync(0xFFFFFFFFu, m >> 3, 1);
            if (lane == 0) before = carry ? 1u : 0u;
            carry = __shfl_sync(0xFFFFFFFFu, m >> 3, 31) != 0u;
            const uint32_t sym[4] = {t.q[u].x, t.q[u].y, t.q[u].z, t.q[u].w};
            const uint32_t keep = ~(m << 1 | before) & 15u;
            const uint32_t there = i >= to ? 0u : to - i >= 4u ? 15u : (1u << (to - i)) - 1u;
            const uint32_t below = (1u << lane) - 1u, copied = keep & there;
            uint32_t at = out, row = 0u;
#pragma unroll
            for (int k = 0; k < 4; k++) { const uint32_t b = __ballot_sync(0xFFFFFFFFu, (copied >> k) & 1u); at += __popc(b & below); row += __popc(b); }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const bool mine = (m & there) >> k & 1u;
                const uint32_t x = mine ? (sym[k] & WORD_START_BIT) | v.fresh : sym[k];
                if (mine) src[i + k] = x;
                if ((copied >> k) & 1u) dst[at++] = x;
            }
            out += row;
        }
    }
}

template <bool LITERAL>
__global__ void __launch_bounds__(WM_THREADS, 1)
k_word_merges(WordArgs A, uint32_t target) {
    extern __shared__ __align__(16) unsigned char wm_smem[];
    WordShared& s = *reinterpret_cast<WordShared*>(wm_smem);
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), tid = threadIdx.x, lane = tid & 31;
    WordTeam T{s, cluster.map_shared_rank(&s, 0), rank, tid, cluster};
    constexpr uint32_t STEP = WM_THREADS * WM_CLUSTER;
    const uint32_t gtid = tid * WM_CLUSTER + rank;        // neighbours in a list go to different SMs
    const uint32_t gtid_mid = (tid ^ (WM_THREADS / 2)) * WM_CLUSTER + rank;   // the same from the middle: short lists side by side

    if (tid < sizeof(WordState) / 4) reinterpret_cast<uint32_t*>(&s.init)[tid] = __ldcg(reinterpret_cast<const uint32_t*>(A.st) + tid);
    uint32_t* my_cand = A.cand + (size_t)rank * (WM_CAND + 1);
    const uint32_t nc = min(__ldcg(my_cand), (uint32_t)WM_CAND);
    for (uint32_t i = tid; i < nc; i += WM_THREADS) s.cand[i] = __ldcg(my_cand + 1 + i);
    __syncthreads();
    if (tid == 0) {
        s.queued = 0u; s.flags = 0u; s.inserted = 0u; s.ncand = s.init.tau == ~0ull ? 0u : nc;
        s.c_entries = s.init.entries; s.c_inserted = 0u; s.c_merged = 0u; s.c_spilled = 0u; s.tail_queued = 0u;
    }
    cluster_barrier();           // also: everybody has read the control block before anybody writes it
    uint32_t done = s.init.merges_done, next_id = s.init.next_id, symbols = s.init.symbols, scans = s.init.scans;
    uint32_t early = s.init.early_stop, status = s.init.status;
    uint32_t front = s.init.front, front_before = s.init.front_before, turn = s.init.turn;
    unsigned long long tau = s.init.tau, best = s.init.best, touched = s.init.touched;
    bool valid = s.init.best_valid != 0u;
    uint32_t occ_most = s.init.occupied;     // upper bound of the occupied slots
    const uint32_t occ_start = s.init.occupied;
    const uint32_t room = (1u << A.table_log2) / 4u * 3u;
    uint32_t flags = 0u;
    uint32_t spilled_before = 0u;            // c_spilled after the merge before
    uint2* const spill_end = A.entries + 2u * (size_t)A.positions;
    if (early || status) return;             // the same in every CTA

    while (done < target) {
        if (!valid || best < tau || (flags & WS_CAND)) {
            word_scan(A, T, tau);
            scans++;
            word_argmax(A, T, best, flags);
            if (flags & WS_CAND) { status = WS_CAND; break; }
            valid = true;
        }
        const uint32_t count = (uint32_t)(best >> 32), pair = ~(uint32_t)best;
        if (count < 2u || next_id > TOKEN_MASK) { early = 1u; break; }
        const uint32_t a = pair >> 16, b = pair & 0xFFFFu, fresh = next_id;
        // the pair's occurrences
        uint32_t beg, end;
        const bool bytes = a < 256u && b < 256u;
        if (bytes) { beg = __ldcg(A.byte_off + (a << 8 | b)); end = __ldcg(A.byte_off + (a << 8 | b) + 1); }
        else { const uint2 g = __ldcg(A.segment + max(a, b)); beg = g.x; end = g.y; }
        const uint32_t len = end - beg;
        const uint32_t usual_a = a < 256u ? 1u : __ldcg(A.usual + a), usual_b = b < 256u ? 1u : __ldcg(A.usual + b);
        // a merge makes at most two new pairs per symbol in use, and per occurrence
        // (the tail: at most two per copied occurrence, with the new symbol, and what the older symbols bring back)
        const uint32_t grow = 2u * min(min(len, count), fresh + 1u) + (LITERAL ? 4u * min(count, fresh) + 4u : 0u);
        if (occ_most + grow > room) {
            occ_most = occ_start + T.lead->c_inserted;     // stable here: it changes between the two barriers of a merge
            if (occ_most + grow > room) { status = WS_GROW; break; }
        }
        occ_most += grow;
        touched += (unsigned long long)len * (bytes ? 4u : 8u) + (LITERAL ? 12ull * (symbols - front) : 0ull);
        TailView tail{};
        uint32_t* tail_src = nullptr;
        uint32_t tail_from = 0u, tail_to = 0u;
        if (LITERAL) {
            tail_src = A.tail[turn % 3u];
            const uint32_t n = symbols - front;
            if (count >= n) { status = WS_TAIL; break; }
            tail = TailView{tail_src, n, n - count, a, b, fresh};
            // a warp's share of what is copied, in whole spans
            const uint32_t share = (tail.limit + TAIL_SPAN * (STEP / 32u) - 1u) / (TAIL_SPAN * (STEP / 32u)) * TAIL_SPAN;
            tail_from = min(tail.limit, ((tid >> 5) * WM_CLUSTER + rank) * share);      // (neighbouring shares in different SMs)
            tail_to = min(tail.limit, tail_from + share);
        }
        uint32_t merged = 0u;        // LITERAL: symbols of the text's front that this thread's occurrences drop

        // ── phase 1: occurrences, counts, the new symbol's list ──
        auto apply = [&](uint32_t qi) {
            const uint32_t p = s.queue[qi].x;
            // every record that is usually needed, in one round trip: the second symbol and the one behind it where they usually are
            // (64 MiB, 8,000 merges: 65.4 -> 63.9 ms)
            const uint32_t q_usual = min(p + usual_a, A.positions), r_usual = min(p + usual_a + usual_b, A.positions);
            const uint32_t rp = A.rec[p], w = A.weight[p], rec_before = p > 0u ? A.rec[p - 1] : 0u;
            const uint32_t rec_q = A.rec[q_usual], rec_r = A.rec[r_usual];
            const uint32_t prev_end = (rp & WP_START) ? 0u : rec_before;
            bool ok = wp_sym(rp) == a;
            const uint32_t la = wp_span(rp), q = p + la;
            const uint32_t rq = !ok ? WP_START : q == q_usual ? rec_q : A.rec[q];
            ok = ok && !(rq & WP_START) && wp_sym(rq) == b;
            // the left neighbour: symbol x at l
            uint32_t l = 0u, x = 0u, rl = WP_START;
            if (ok && !(rp & WP_START)) { l = p - wp_span(prev_end); rl = A.rec[l]; x = wp_sym(rl); }
            if (a == b && x == a) ok = false;         // inside a run of equal symbols: its first position merges the whole run
            uint32_t r = q + wp_span(rq), rr = !ok ? WP_START : r == r_usual ? rec_r : A.rec[r];
            uint32_t drops = 1u;
            if (a == b) while (ok && !(rr & WP_START) && wp_sym(rr) == a) { r += wp_span(rr); rr = A.rec[r]; drops++; }
            if (LITERAL && ok) merged += drops * w;
            const uint32_t span = r - p;
            uint32_t y = (!ok || (rr & WP_START)) ? 0u : wp_sym(rr);
            uint32_t right_left = b;                   // symbol on the left of the right-hand neighbour before the merge
            uint32_t new_right = y;
            bool left = ok && x != 0u;
            if (a != b) {
                // an occurrence right behind this one: the pair in between is (b, a), and becomes (new, new); the left one sees to it
                if (y == a) {
                    const uint32_t rz = A.rec[r + wp_span(rr)];
                    if (!(rz & WP_START) && wp_sym(rz) == b) new_right = fresh;
                }
                if (left && x == b && !(rl & WP_START)) {
                    const uint32_t ll = l - wp_span(A.rec[l - 1]);
                    if (wp_sym(A.rec[ll]) == a) left = false;
                }
            }
            const bool right = y != 0u;
            s.queue[qi] = ok ? make_uint2(p, span | (a == b ? 0u : la << 16)) : make_uint2(~0u, 0u);
            // the four counts that change
            const uint32_t k0 = x << 16 | a, k1 = x << 16 | fresh, k2 = right_left << 16 | y, k3 = fresh << 16 | new_right;
            // room in the list of the new symbol: asked for now, needed last (the counter is in another SM)
            const uint32_t want = (left ? 1u : 0u) + (right ? 1u : 0u);
            const uint32_t active = __activemask();
            const uint32_t one = __ballot_sync(active, want & 1u), two = __ballot_sync(active, want & 2u);
            const int leader = __ffs((int)active) - 1;
            uint32_t at = 0u;
            if ((int)lane == leader && (one | two)) at = atomicAdd(&T.lead->c_entries, __popc(one) + 2u * __popc(two));
            const uint32_t keys[4] = {k0, k1, k2, k3}, by[4] = {w, w, w, w};
            wt_updates<4>(A, T, keys, by, (left ? 3u : 0u) | (right ? 12u : 0u), 10u, tau);
            const uint32_t below = (1u << lane) - 1u;
            at = __shfl_sync(active, at, leader) + __popc(one & below) + 2u * __popc(two & below);
            if (left) A.entries[at++] = make_uint2(l, k1);
            if (right) A.entries[at] = make_uint2(p, k3);
        };
        // Phase 2 of one occurrence.
        auto rewrite = [&](uint2 o) {
            if (o.x == ~0u) return;
            const uint32_t p = o.x, span = o.y & 0x7FFFu, e = p + span - 1u;
            const uint32_t rp = A.rec[p];
            if (a != b) {
                const uint32_t q = p + (o.y >> 16);
                if (q != e) A.rec[q] = 0u;
            } else {
                for (uint32_t q = p + wp_span(rp); q <= e;) {
                    const uint32_t rq = A.rec[q];
                    A.rec[q] = 0u;
                    q += max(wp_span(rq), 1u);
                }
            }
            A.rec[e] = span << 16;
            A.rec[p] = fresh | span << 16 | (rp & WP_START);
        };
        // The queue's first n occurrences, with what phase 1 found out about them, to the end of the entries' buffer, downwards.  Phase 2 takes
        // them from there and looks at no neighbour again: in a run of equal symbols the neighbours are another thread's to rewrite, and
        // may be gone.  There is room: an occurrence writes two entries at most and ends a position, so with L symbols left after
        // this merge the lists hold 2 (positions - L) entries at most; and every occurrence leaves a symbol, so L are spilled at most.
        auto spill = [&](uint32_t n) {
            uint32_t mine = 0u;
            for (uint32_t i0 = 0; i0 < n; i0 += WM_THREADS) {
                const uint32_t i = i0 + tid;                 // (the thread that has looked at it)
                mine += __popc(__ballot_sync(0xFFFFFFFFu, i < n && s.queue[i].x != ~0u));
            }
            uint32_t at = 0u;
            if (lane == 0 && mine) at = atomicAdd(&T.lead->c_spilled, mine) - spilled_before;
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
            for (uint32_t i0 = 0; i0 < n; i0 += WM_THREADS) {
                const uint32_t i = i0 + tid;
                const uint2 o = i < n ? s.queue[i] : make_uint2(~0u, 0u);
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, o.x != ~0u);
                if (o.x != ~0u) *(spill_end - 1u - (at + __popc(m & ((1u << lane) - 1u)))) = o;
                at += __popc(m);
            }
        };
        // The list in rounds of WM_UNROLL entries per thread; the queued occurrences are taken whenever the queue could overflow
        // (only a list of more than one round can), and at the end.
        const bool spills = len > STEP * WM_UNROLL;          // the same in every CTA
        auto walk = [&]() {
            for (uint32_t base = 0; base < len; base += STEP * WM_UNROLL) {
                uint32_t pos[WM_UNROLL];
                bool hit[WM_UNROLL];
#pragma unroll
                for (int k = 0; k < WM_UNROLL; k++) {
                    const uint32_t i = base + k * STEP + gtid;
                    hit[k] = i < len;
                    pos[k] = 0u;
                    if (hit[k]) {
                        if (bytes) pos[k] = __ldcg(A.byte_list + beg + i);
                        else { const uint2 g = __ldcg(A.entries + beg + i); pos[k] = g.x; hit[k] = g.y == pair; }
                    }
                }
#pragma unroll
                for (int k = 0; k < WM_UNROLL; k++) {
                    const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit[k]);
                    if (m) {
                        uint32_t at = 0u;
                        if (lane == 0) at = atomicAdd(&s.queued, (uint32_t)__popc(m));
                        at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(m & ((1u << lane) - 1u));
                        if (hit[k]) s.queue[at].x = pos[k];
                    }
                }
                __syncthreads();
                const uint32_t n = s.queued;
                const bool last = base + STEP * WM_UNROLL >= len;
                if (!last) __syncthreads();          // everybody has read the fill before the next round adds to it
                if (last || n + WM_THREADS * WM_UNROLL > WM_QUEUE) {
                    for (uint32_t i = tid; i < n; i += WM_THREADS) apply(i);
                    __syncwarp();
                    if (!last) {
                        spill(n);
                        __syncthreads();
                        if (tid == 0) s.queued = 0u;
                        __syncthreads();
                    }
                }
            }
        };
        static_assert(WM_THREADS * WM_UNROLL <= WM_QUEUE, "a round fits the queue");
        if (LITERAL) {
            const uint32_t kept = tail_count(A, T, tail, tail_from, tail_to, tau);
            if (lane < WM_CLUSTER) cluster.map_shared_rank(&s, lane)->kept[(tid >> 5) * WM_CLUSTER + rank] = kept;
            __syncthreads();
        }
        walk();
        if (LITERAL) {
            // the tail's matches from the last thread down: where both are few, other warps than those with the dictionary's occurrences
            for (uint32_t i = WM_THREADS - 1u - tid; i < min(s.tail_queued, TAIL_QUEUE); i += WM_THREADS) tail_match_changes(A, T, tail, s.tail_queue[i], tau);
            tail_pairs(A, T, tail_src + (tail.limit - 1u), tail.n - (tail.limit - 1u), gtid_mid, false, tau, nullptr);
            __syncwarp();
            merged = __reduce_add_sync(0xFFFFFFFFu, merged);
            if (lane == 0 && merged) atomicAdd(&T.lead->c_merged, merged);
        } else if (rank == WM_CLUSTER - 1 && tid == WM_THREADS - 1) {
            // every occurrence of the pair itself goes (a thread that seldom has an occurrence: this is a chain of round trips of its own)
            wt_update(A, T, pair, count, false, tau);
        }
        __syncwarp();
        cluster_barrier();

        uint32_t dropped = 0u, kept_all = 0u, stale = 0u;      // LITERAL: see below
        if (LITERAL) {
            dropped = T.lead->c_merged;                        // by the front; the rest of `count` by the tail
            uint32_t out = 0u;                                 // what the warps with earlier shares copy
#pragma unroll
            for (uint32_t k = 0; k < WM_CLUSTER * WM_THREADS / 32; k += 32) {
                const uint32_t kept = s.kept[k + lane];
                kept_all += kept;
                if (k + lane < (tid >> 5) * WM_CLUSTER + rank) out += kept;
            }
            kept_all = __reduce_add_sync(0xFFFFFFFFu, kept_all);
            out = __reduce_add_sync(0xFFFFFFFFu, out);
            const uint32_t n1 = tail.n - (count - dropped);    // tail symbols after this merge, kept_all of them copied
            stale = n1 - kept_all;
            const uint32_t from = front - dropped + kept_all;  // position of the first that keeps its older contents
            if (stale && from < front_before) { status = WS_TAIL; break; }
            uint32_t* dst = A.tail[(turn + 1u) % 3u];
            const uint32_t* older = A.tail[(turn + 2u) % 3u] + (from - front_before);
            tail_move(tail, tail_src, dst, tail_from, tail_to, out, lane);
            for (uint32_t i = tail.limit + gtid; i < tail.n; i += STEP) {       // the rewrite where nothing is copied
                const uint32_t l = tail_at(tail, i);
                if (tail_match(tail, l, tail_at(tail, i + 1u))) tail_src[i] = (l & WORD_START_BIT) | fresh;
            }
            tail_pairs(A, T, older, stale, gtid_mid, true, tau, dst + kept_all);
            // single updates, each a chain of round trips, by threads of different SMs
            if (tid == WM_THREADS - 1) {
                if (rank == 0 && stale) {      // the last copied symbol and the first older one
                    uint32_t i = tail.limit - 1u, l = tail_at(tail, i);
                    const uint32_t behind = tail_at(tail, i + 1u), r = __ldcg(older);
                    uint32_t prev = i > 0u ? tail_at(tail, i - 1u) : WORD_START_BIT, next = behind;
                    while (i > 0u && tail_match(tail, prev, l)) { next = l; l = prev; i--; prev = i > 0u ? tail_at(tail, i - 1u) : WORD_START_BIT; }
                    if (tail_match(tail, l, next)) l = fresh;
                    if (tail_counted(l, r)) tail_pair(A, T, l, r, true, tau);
                }
                if (rank == 1 && dropped)      // the front's occurrences of the pair itself go (the tail's went one by one)
                    wt_update(A, T, pair, dropped, false, tau);
            }
            __syncwarp();
        }
        // ── phase 2: the records; the next merge's pair ──
        {
            const uint32_t n = s.queued;
            for (uint32_t i = tid; i < n; i += WM_THREADS) rewrite(s.queue[i]);
        }
        if (spills) {
            const uint32_t all = T.lead->c_spilled, n = all - spilled_before;     // (nobody spills before the next cluster barrier)
            for (uint32_t i = gtid; i < n; i += STEP) rewrite(__ldcg(spill_end - 1 - i));
            spilled_before = all;
        }
        if (gtid == 0) {
            const uint32_t e1 = s.c_entries;
            A.segment[fresh] = make_uint2(s.init.entries, e1);
            A.usual[fresh] = usual_a + usual_b;
            s.init.entries = e1;
            A.log[done] = make_uint4(a, b, fresh, count);
        }
        if (LITERAL) cluster_barrier();      // counts change in phase 2 too: all of them before the arg-max looks
        if (tid == 0 && s.inserted) {
            atomicAdd(&T.lead->c_inserted, s.inserted);
            s.inserted = 0u;
        }
        done++;
        next_id++;
        symbols -= count;
        if (LITERAL) {
            front_before = front;
            front -= dropped;
            turn++;
            if (gtid == 0) s.c_merged = 0u;
            if (tid == 0) s.tail_queued = 0u;
        }
        word_argmax(A, T, best, flags);
        if (flags & WS_FULL) { status = WS_FULL; break; }
    }
    // control block and candidates for the next launch
    cluster_barrier();
    const uint32_t n = min(s.ncand, (uint32_t)WM_CAND);
    for (uint32_t i = tid; i < n; i += WM_THREADS) my_cand[1 + i] = s.cand[i];
    if (tid == 0) my_cand[0] = n;
    if (gtid == 0) {
        WordState o = s.init;
        o.tau = (flags & WS_CAND) ? ~0ull : tau;
        o.best = best;
        o.best_valid = (valid && !(flags & WS_CAND)) ? 1u : 0u;
        o.merges_done = done;
        o.next_id = next_id;
        o.early_stop = early;
        o.status = status;
        o.occupied = occ_start + s.c_inserted;
        o.symbols = symbols;
        o.scans = scans;
        o.touched = touched;
        o.front = front;
        o.front_before = front_before;
        o.turn = turn;
        *A.st = o;
    }
    cluster_barrier();           // no CTA ends while its shared memory may still be read
}

}  // namespace b200bpe
