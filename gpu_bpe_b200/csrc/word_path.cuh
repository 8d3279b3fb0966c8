// Host side of training on the dictionary of distinct words (word_dict.cuh, word_merge.cuh): buffers, set-up, the batch loop.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ctx.cuh"
#include "word_merge.cuh"

namespace b200bpe {

constexpr uint32_t WORD_MAX_TABLE_LOG2 = 28;

struct WordPath {
    Ctx* ctx = nullptr;
    const uint8_t* bytes = nullptr;      // the corpus and its word starts, on the device
    const uint8_t* mask = nullptr;
    uint64_t n = 0;
    DictTables dict{};
    WordArgs args{};
    uint32_t* cursor = nullptr;
    unsigned long long* bins = nullptr;
    uint64_t cap_positions = 0;
    uint32_t positions = 0;
    WordState* h_state = nullptr;        // pinned: one per batch in flight
    DictState* h_dict = nullptr;         // pinned
    size_t pinned = 0;                   // bytes of the pinned block
    uint8_t* own_mask = nullptr;         // heuristic word starts, or those of tagged symbols
    uint8_t* own_bytes = nullptr;
    uint4* h_log = nullptr;              // pinned
    uint32_t goal = 0;                   // merges the log has room for
    bool given_log2 = false;             // the caller chose the pair table's size
    bool literal = false;
    uint64_t n_front = 0;                // bytes that the dictionary takes: all, or what is before the tail of a "literal" run
    uint64_t cap_tail = 0;
    static constexpr uint32_t TAIL_SHORT = 3, TAIL_LONG = 8;
    uint32_t tail_share = TAIL_SHORT;    // 32nds of the text
    WordState seen{};                    // control block after the last batch
    uint64_t launches = 0;
    std::vector<cudaEvent_t> ev;

    static constexpr int IN_FLIGHT = 4;  // batches enqueued ahead of the host

    ~WordPath() { release(); }
    void release() {
        if (!ctx) return;
        for (void* p : {(void*)dict.short_key, (void*)dict.short_cnt, (void*)dict.short_base, (void*)dict.long_key, (void*)dict.long_cnt,
                        (void*)dict.long_base, (void*)dict.st, (void*)args.rec, (void*)args.weight, (void*)args.byte_list, (void*)args.byte_off,
                        (void*)args.entries, (void*)args.segment, (void*)args.usual, (void*)args.table, (void*)args.cand, (void*)args.st, (void*)args.log,
                        (void*)cursor, (void*)bins, (void*)own_mask, (void*)own_bytes, (void*)args.tail[0], (void*)args.tail[1], (void*)args.tail[2]})
            ctx->free(p);
        ctx->free_pinned(h_state, pinned);
        for (auto e : ev) cudaEventDestroy(e);
        ctx = nullptr;
    }

    // Buffers whose size does not depend on the text.
    b200bpe_status create(Ctx* c, uint64_t n_bytes, uint32_t merges_goal, uint32_t table_log2, bool literal_mode) {
        ctx = c;
        n = n_bytes;
        literal = literal_mode;
        goal = std::max<uint32_t>(1, merges_goal);
        auto log2_of = [](uint64_t x) { uint32_t l = 0; while ((1ull << l) < x) l++; return l; };
        // slots for one distinct short word per 8 bytes and one distinct long word per 32
        dict.short_log2 = std::min<uint32_t>(27, std::max<uint32_t>(10, log2_of(n / 8)));
        dict.long_log2 = std::min<uint32_t>(26, std::max<uint32_t>(8, log2_of(n / 32)));
        args.table_log2 = table_log2;
        given_log2 = table_log2 != 0;
        B2_CUDA(ctx->alloc(&dict.short_key, sizeof(WordKey) << dict.short_log2));
        B2_CUDA(ctx->alloc(&dict.short_cnt, sizeof(uint32_t) << dict.short_log2));
        B2_CUDA(ctx->alloc(&dict.short_base, sizeof(uint32_t) << dict.short_log2));
        B2_CUDA(ctx->alloc(&dict.long_key, sizeof(unsigned long long) << dict.long_log2));
        B2_CUDA(ctx->alloc(&dict.long_cnt, sizeof(uint32_t) << dict.long_log2));
        B2_CUDA(ctx->alloc(&dict.long_base, sizeof(uint32_t) << dict.long_log2));
        B2_CUDA(ctx->alloc(&dict.st, sizeof(DictState)));
        B2_CUDA(ctx->alloc(&args.byte_off, sizeof(uint32_t) * 65537));
        B2_CUDA(ctx->alloc(&cursor, sizeof(uint32_t) * 65536));
        B2_CUDA(ctx->alloc(&bins, sizeof(unsigned long long) * 65536));
        B2_CUDA(ctx->alloc(&args.segment, sizeof(uint2) * 65536));
        B2_CUDA(ctx->alloc(&args.usual, sizeof(uint32_t) * 65536));
        B2_CUDA(ctx->alloc(&args.cand, sizeof(uint32_t) * WM_CLUSTER * (WM_CAND + 1)));
        B2_CUDA(ctx->alloc(&args.st, sizeof(WordState)));
        B2_CUDA(ctx->alloc(&args.log, sizeof(uint4) * (size_t)goal));
        pinned = sizeof(WordState) * IN_FLIGHT + sizeof(DictState) + sizeof(uint4) * (size_t)goal;
        B2_CUDA(ctx->alloc_pinned(reinterpret_cast<void**>(&h_state), &pinned));
        h_log = reinterpret_cast<uint4*>(h_state + IN_FLIGHT);
        h_dict = reinterpret_cast<DictState*>(h_log + goal);
        for (int i = 0; i < IN_FLIGHT; i++) {
            cudaEvent_t e;
            B2_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            ev.push_back(e);
        }
        B2_CUDA(cudaFuncSetAttribute(k_dict_words, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WD_SMEM_BYTES));
        B2_CUDA(cudaFuncSetAttribute(kernel(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WordShared)));
        B2_CUDA(cudaFuncSetAttribute(kernel(), cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        return B200BPE_OK;
    }

    int blocks(uint64_t items, int per_block, int per_sm) const {
        return (int)std::max<uint64_t>(1, std::min<uint64_t>((items + per_block - 1) / per_block, (uint64_t)ctx->sm_count * per_sm));
    }
    void (*kernel() const)(WordArgs, uint32_t) { return literal ? k_word_merges<true> : k_word_merges<false>; }
    // The tail has to hold about three times a merge's count: what is dropped, and what came in its place two merges ago.  The first
    // merges count most, some 2.5 % of a text each; a run that they end starts again with a longer tail.
    uint64_t tail_goal() const { return n / 32 * tail_share; }
    int aligned() const { return (((uintptr_t)bytes | (uintptr_t)mask) & 15u) == 0 ? 1 : 0; }

    // Texts of few letters whose words are mostly distinct (DNA, digits) are the symbol buffers': a merge then has millions of occurrences in
    // the dictionary too, on 16 SMs and with their counts on a few hot slots.  With P positions for n bytes and E byte pairs in use (the
    // inverse of the chance that two pairs are the same), merges with the dictionary took 10 P / (n sqrt E) times as long as on the symbol
    // buffers where these merges are most of a run, and what later merges save pays for 3,500 of P / sqrt E each; in "literal" runs an
    // explicit symbol of the tail costs as much as two positions, and a later merge saves a quarter of that.  Create + run, dictionary / symbol
    // buffers, ms, 128 MiB of distinct words of 65 letters, 64 merges: 2 letters 324 / 61, 4 letters 231 / 90, 8 letters 135 / 97, 12 letters
    // 103 / 102, 64 letters 47 / 61; 4 letters, 4,000 merges 568 / 480, every word four times 170 / 466.  Up to 4 MiB the dictionary was never
    // slower.  A text that goes to the symbol buffers by this rule pays 1 ms per 128 MiB for having its words looked up.
    static constexpr uint64_t FEW_LETTERS_FROM = 8ull << 20;
    bool few_letters() const {
        if (h_dict->squares == 0) return false;
        const double e = (double)h_dict->sampled * (double)h_dict->sampled / (double)h_dict->squares;
        // (a first merge of more than a 32nd of the text needs the long tail)
        const double tail = literal ? (double)n / 32 * (e < 32 ? TAIL_LONG : tail_share) : 0.0;
        return ((double)h_dict->positions + 2 * tail) / std::sqrt(e) > (double)n / 10 + (literal ? 900.0 : 3500.0) * goal;
    }

    // Builds the dictionary of the text and the state of a fresh run.  *fits is false (and nothing else is set up) when the text is
    // not one of words that a dictionary pays for: the symbol buffers of the other path then take it.
    b200bpe_status build(const uint8_t* d_bytes, const uint8_t* d_mask, const uint32_t* d_symbols, uint32_t first_id, bool* fits) {
        cudaStream_t s = ctx->stream;
        *fits = false;
        B2_CUDA(cudaMemsetAsync(dict.st, 0, sizeof(DictState), s));
        bytes = d_bytes;
        mask = d_mask;
        if (d_symbols) {
            if (!own_bytes) B2_CUDA(ctx->alloc(&own_bytes, n));
            if (!own_mask) B2_CUDA(ctx->alloc(&own_mask, n));
            k_dict_split<<<blocks(n, 256, 16), 256, 0, s>>>(d_symbols, n, own_bytes, own_mask, dict.st);
            bytes = own_bytes;
            mask = own_mask;
            launches++;
        } else if (!mask) {
            if (!own_mask) B2_CUDA(ctx->alloc(&own_mask, n));
            k_dict_heuristic<<<blocks(n, 256, 16), 256, 0, s>>>(bytes, n, own_mask);
            mask = own_mask;
            launches++;
        }
        B2_CUDA(cudaMemsetAsync(dict.short_key, 0, sizeof(WordKey) << dict.short_log2, s));
        B2_CUDA(cudaMemsetAsync(dict.short_cnt, 0, sizeof(uint32_t) << dict.short_log2, s));
        B2_CUDA(cudaMemsetAsync(dict.long_key, 0, sizeof(unsigned long long) << dict.long_log2, s));
        B2_CUDA(cudaMemsetAsync(dict.long_cnt, 0, sizeof(uint32_t) << dict.long_log2, s));
        n_front = n;
        if (literal) {
            k_dict_split_at<<<1, 256, 0, s>>>(mask, n, n - tail_goal(), dict.st);
            launches++;
            B2_CUDA(cudaMemcpyAsync(h_dict, dict.st, sizeof(DictState), cudaMemcpyDeviceToHost, s));
            B2_CUDA(cudaStreamSynchronize(s));
            n_front = h_dict->split;
            if (n_front == 0 || n_front >= n) return B200BPE_OK;
        }
        const bool large = n_front >= FEW_LETTERS_FROM;
        if (large) {
            B2_CUDA(cudaMemsetAsync(bins, 0, sizeof(unsigned long long) * 65536, s));
            k_dict_sample<<<1, 1024, 0, s>>>(bytes, mask, n_front, bins, dict.st);
            launches++;
        }
        k_dict_words<<<blocks(n_front, WD_TILE, 3), WD_THREADS, WD_SMEM_BYTES, s>>>(bytes, mask, n_front, dict, aligned());
        const uint64_t slots = (1ull << dict.short_log2) + (1ull << dict.long_log2);
        k_dict_places<<<blocks(slots, 1024, 8), 256, 0, s>>>(mask, n_front, dict);
        launches += 2;
        B2_CUDA(cudaMemcpyAsync(h_dict, dict.st, sizeof(DictState), cudaMemcpyDeviceToHost, s));
        B2_CUDA(cudaStreamSynchronize(s));
        B2_CUDA(cudaGetLastError());
        if (h_dict->status || (large && few_letters())) return B200BPE_OK;
        positions = h_dict->positions;
        args.positions = positions;
        if (positions > cap_positions || !args.rec) {
            for (void* p : {(void*)args.rec, (void*)args.weight, (void*)args.byte_list, (void*)args.entries}) ctx->free(p);
            args.rec = nullptr; args.weight = nullptr; args.byte_list = nullptr; args.entries = nullptr;
            cap_positions = positions;
            B2_CUDA(ctx->alloc(&args.rec, sizeof(uint32_t) * (cap_positions + 4)));
            B2_CUDA(ctx->alloc(&args.weight, sizeof(uint32_t) * cap_positions));
            B2_CUDA(ctx->alloc(&args.byte_list, sizeof(uint32_t) * cap_positions));
            B2_CUDA(ctx->alloc(&args.entries, sizeof(uint2) * 2 * cap_positions));   // a merge of one occurrence makes two pairs and ends a position
        }
        uint32_t* weight = const_cast<uint32_t*>(args.weight);
        uint32_t* list = const_cast<uint32_t*>(args.byte_list);
        uint32_t* off = const_cast<uint32_t*>(args.byte_off);
        B2_CUDA(cudaMemsetAsync(bins, 0, sizeof(unsigned long long) * 65536, s));
        B2_CUDA(cudaMemsetAsync(args.st, 0, sizeof(WordState), s));
        k_dict_fill<<<blocks(slots, 256, 16), 256, 0, s>>>(bytes, mask, n_front, dict, args.rec, weight);
        k_dict_count<<<blocks(positions, 256, 8), 256, 0, s>>>(args.rec, weight, positions, bins);
        if (literal) {
            const uint64_t tail = n - n_front;
            if (tail > cap_tail) {
                for (auto& t : args.tail) { ctx->free(t); t = nullptr; }
                for (auto& t : args.tail) B2_CUDA(ctx->alloc(&t, sizeof(uint32_t) * (tail + 4)));
                cap_tail = tail;
            }
            // (the destination of the first merge starts zeroed, as a fresh WebGPU buffer does: it is what the older symbols come from)
            B2_CUDA(cudaMemsetAsync(args.tail[2], 0, sizeof(uint32_t) * tail, s));
            k_dict_tail<<<blocks(tail, 256, 16), 256, 0, s>>>(bytes, mask, n_front, n, args.tail[0], bins);
            launches++;
        }
        k_dict_offsets<<<1, 1024, 0, s>>>(bins, off, cursor, dict.st);
        k_dict_lists<<<blocks(positions, 256, 8), 256, 0, s>>>(args.rec, positions, cursor, list);
        launches += 4;
        // The table has room for twice the byte pairs there can be at most; it grows when merges fill it.  It is sparse (two slots a position
        // at most): a probe that collides is another round trip, and the scans that pay for its size are a few in a run.
        if (args.table_log2 == 0) {
            uint32_t l = 13;
            while (l < 23 && (2ull << l) < positions + (n - n_front)) l++;
            args.table_log2 = l;
        }
        uint64_t most = std::min<uint64_t>((uint64_t)positions + (n - n_front), 65536);
        if (given_log2) {   // a size from the caller holds what there is, and no more
            B2_CUDA(cudaMemcpyAsync(h_dict, dict.st, sizeof(DictState), cudaMemcpyDeviceToHost, s));
            B2_CUDA(cudaStreamSynchronize(s));
            most = (h_dict->pairs + 1) / 2;
        }
        while ((3ull << (args.table_log2 - 2)) < 2 * most) {
            if (args.table) { ctx->free(args.table); args.table = nullptr; }
            args.table_log2++;
        }
        if (!args.table) B2_CUDA(ctx->alloc(&args.table, sizeof(unsigned long long) << args.table_log2));
        B2_CUDA(cudaMemsetAsync(args.table, 0, sizeof(unsigned long long) << args.table_log2, s));
        k_word_init<<<256, 256, 0, s>>>(bins, dict.st, args.table, args.table_log2, args.st, first_id, (uint32_t)n, (uint32_t)n_front);
        seen = WordState{};
        seen.symbols = (uint32_t)n;
        seen.front = (uint32_t)n_front;
        launches++;
        B2_CUDA(cudaGetLastError());
        *fits = true;
        return B200BPE_OK;
    }

    b200bpe_status enqueue_batch(uint32_t target) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(WM_CLUSTER);
        cfg.blockDim = dim3(WM_THREADS);
        cfg.dynamicSmemBytes = sizeof(WordShared);
        cfg.stream = ctx->stream;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = WM_CLUSTER;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        B2_CUDA(cudaLaunchKernelEx(&cfg, kernel(), args, target));
        launches++;
        return B200BPE_OK;
    }

    b200bpe_status grow() {
        if (args.table_log2 >= WORD_MAX_TABLE_LOG2) return B200BPE_ERR_TABLE_FULL;
        cudaStream_t s = ctx->stream;
        unsigned long long* to = nullptr;
        B2_CUDA(ctx->alloc(&to, sizeof(unsigned long long) << (args.table_log2 + 1)));
        B2_CUDA(cudaMemsetAsync(to, 0, sizeof(unsigned long long) << (args.table_log2 + 1), s));
        k_word_regrown<<<1, 1, 0, s>>>(args.st);
        k_word_rehash<<<blocks(1ull << args.table_log2, 256, 8), 256, 0, s>>>(args.table, args.table_log2, to, args.table_log2 + 1, args.st);
        launches += 2;
        B2_CUDA(cudaGetLastError());
        ctx->free(args.table);
        args.table = to;
        args.table_log2++;
        return B200BPE_OK;
    }

    // The live symbols into d_out (device, room for the count in `symbols`).
    b200bpe_status expand(uint32_t* d_out) {
        cudaStream_t s = ctx->stream;
        const uint64_t tiles = (n_front + WD_TILE - 1) / WD_TILE;
        uint32_t* counts = nullptr;
        B2_CUDA(ctx->alloc(&counts, sizeof(uint32_t) * (tiles + 1)));
        k_dict_expand<false><<<blocks(tiles, 1, 4), WD_THREADS, 0, s>>>(bytes, mask, n_front, dict, args.rec, counts, nullptr, aligned());
        k_dict_scan<<<1, 1024, 0, s>>>(counts, tiles);
        k_dict_expand<true><<<blocks(tiles, 1, 4), WD_THREADS, 0, s>>>(bytes, mask, n_front, dict, args.rec, counts, d_out, aligned());
        launches += 3;
        if (n_front < n)
            B2_CUDA(cudaMemcpyAsync(d_out + seen.front, args.tail[seen.turn % 3], sizeof(uint32_t) * (size_t)(seen.symbols - seen.front), cudaMemcpyDeviceToDevice, s));
        cudaError_t e = cudaGetLastError();
        ctx->free(counts);
        B2_CUDA(e);
        return B200BPE_OK;
    }
};

}  // namespace b200bpe
