// Token ids back to bytes: TrieTokenizer.decode (src/bpe/tokenizer/tokenizer.js of toprakdeviren/gpu-bpe), which appends the vocabulary's
// bytes token by token and U+FFFD for an id that the vocabulary does not have.
//
// The vocabulary lies on the device as one run of bytes with offsets.  k_decode_places gives every token the place of its bytes (lengths,
// scan, look-back over the tiles), k_decode_copy copies them.  Both are bound by the gathers from the vocabulary, which L2 holds; at
// the sizes of a call that is little against the two copies over the bus.
// 85,000 tokens of a 32,256-entry vocabulary from and to host memory: 7.86 ms token by token on the host, 0.147 ms here.
//
// Detokenising is what a server's worker threads do at any time, so a handle does not change once it is made: what a call needs belongs
// to the call, and the work goes through the context's stream for decoders, apart from a graph that its other stream may be recording.  (A stream
// per handle makes a block of the pool change streams from call to call when several handles take turns: 158 us a call, with this one 146.)
#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "ctx.cuh"
#include "look_back.cuh"

namespace b200bpe {

constexpr int DC_THREADS = 256;
constexpr int DC_PER = 4;
constexpr int DC_TILE = DC_THREADS * DC_PER;      // tokens per tile

// ctl: {total bytes, tile ticket | error flag << 32}, then the look-back descriptors.
__global__ void __launch_bounds__(DC_THREADS)
k_decode_places(const uint32_t* __restrict__ tokens, uint64_t n, const uint64_t* __restrict__ off, uint32_t entries, uint64_t* __restrict__ place,
                unsigned long long* __restrict__ ctl) {
    __shared__ uint64_t s_warp[DC_THREADS / 32], s_base;
    __shared__ uint32_t s_tile;
    uint32_t* ticket = reinterpret_cast<uint32_t*>(ctl + 1);
    const uint64_t tiles = (n + DC_TILE - 1) / DC_TILE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
        __syncthreads();
        const uint64_t tile = s_tile;
        if (tile >= tiles) return;
        uint64_t len[DC_PER], sum = 0;
#pragma unroll
        for (int k = 0; k < DC_PER; k++) {
            const uint64_t i = tile * DC_TILE + threadIdx.x * DC_PER + k;
            const uint32_t t = i < n ? min(tokens[i], entries) : 0u;        // entry `entries` is the replacement character
            len[k] = i < n ? off[t + 1] - off[t] : 0ull;
            sum += len[k];
        }
        uint64_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += x;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        uint64_t at = inc - sum, total = 0;
#pragma unroll
        for (int w = 0; w < DC_THREADS / 32; w++) { const uint64_t v = s_warp[w]; if (w < warp) at += v; total += v; }
        if (warp == 0) {
            const unsigned long long base = sc_look_back(ctl + 2, tile, total, lane, SC_MAX_SPINS, ticket);
            if (lane == 0) {
                s_base = base;
                if (tile == tiles - 1) ctl[0] = base + total;
            }
        }
        __syncthreads();
        at += s_base;
#pragma unroll
        for (int k = 0; k < DC_PER; k++) {
            const uint64_t i = tile * DC_TILE + threadIdx.x * DC_PER + k;
            if (i < n) place[i] = at;
            at += len[k];
        }
    }
}
// Copies every token's bytes to its place, if all of them fit `cap` (and every tile learned its place).
__global__ void __launch_bounds__(DC_THREADS)
k_decode_copy(const uint32_t* __restrict__ tokens, uint64_t n, const uint64_t* __restrict__ off, const uint8_t* __restrict__ bytes, uint32_t entries,
              const uint64_t* __restrict__ place, const unsigned long long* __restrict__ ctl, uint8_t* __restrict__ out, uint64_t cap) {
    if (ctl[0] > cap || (ctl[1] >> 32) != 0ull) return;
    for (uint64_t i = (uint64_t)blockIdx.x * DC_THREADS + threadIdx.x; i < n; i += (uint64_t)gridDim.x * DC_THREADS) {
        const uint32_t t = min(tokens[i], entries);
        const uint64_t from = off[t], len = off[t + 1] - from, to = place[i];
        for (uint64_t k = 0; k < len; k++) out[to + k] = bytes[from + k];
    }
}

struct Decoder {
    CtxHold hold;
    Ctx* ctx = nullptr;
    cudaStream_t stream = nullptr;
    uint32_t entries = 0;
    uint64_t* d_off = nullptr;
    uint8_t* d_bytes = nullptr;
    // the text of the last b200bpe_decoder_run
    std::mutex mutex;
    uint8_t* d_text = nullptr;
    uint64_t n_text = 0;

    ~Decoder() {
        if (!ctx) return;
        cudaSetDevice(ctx->device);
        for (void* p : {(void*)d_off, (void*)d_bytes, (void*)d_text}) ctx->free(p, stream);
    }

    // Host tokens to bytes on the device: *text, the caller's to free (null without bytes), and their number.
    b200bpe_status run(const uint32_t* tokens, uint64_t n, uint8_t** text, uint64_t* n_bytes) {
        cudaStream_t s = stream;
        *text = nullptr;
        *n_bytes = 0;
        if (n == 0) return B200BPE_OK;
        const uint64_t tiles = (n + DC_TILE - 1) / DC_TILE;
        uint32_t* d_tok = nullptr;
        uint64_t* place = nullptr;
        unsigned long long* ctl = nullptr;
        uint8_t* d_out = nullptr;
        void* pinned = nullptr;
        size_t pinned_bytes = 16;
        uint64_t cap = n * 8;       // a guess; an output that needs more is copied again
        auto work = [&]() -> b200bpe_status {
            B2_CUDA(ctx->alloc_pinned(&pinned, &pinned_bytes));
            uint64_t* h_ctl = static_cast<uint64_t*>(pinned);
            B2_CUDA(ctx->alloc(&d_tok, n * 4, s));
            B2_CUDA(ctx->alloc(&place, n * 8, s));
            B2_CUDA(ctx->alloc(&ctl, (tiles + 2) * 8, s));
            B2_CUDA(ctx->alloc(&d_out, cap, s));
            B2_CUDA(cudaMemcpyAsync(d_tok, tokens, n * 4, cudaMemcpyHostToDevice, s));
            B2_CUDA(cudaMemsetAsync(ctl, 0, (tiles + 2) * 8, s));
            const int most = ctx->sm_count * 8;
            k_decode_places<<<(int)std::min<uint64_t>(most, tiles), DC_THREADS, 0, s>>>(d_tok, n, d_off, entries, place, ctl);
            const int grid = (int)std::min<uint64_t>(most, (n + DC_THREADS - 1) / DC_THREADS);
            k_decode_copy<<<grid, DC_THREADS, 0, s>>>(d_tok, n, d_off, d_bytes, entries, place, ctl, d_out, cap);
            B2_CUDA(cudaGetLastError());
            B2_CUDA(cudaMemcpyAsync(h_ctl, ctl, 16, cudaMemcpyDeviceToHost, s));
            B2_CUDA(cudaStreamSynchronize(s));
            if ((uint32_t)(h_ctl[1] >> 32) != 0u) return B200BPE_ERR_LOOKBACK_TIMEOUT;
            if (h_ctl[0] > cap) {
                ctx->free(d_out, s);
                d_out = nullptr;
                cap = h_ctl[0];
                B2_CUDA(ctx->alloc(&d_out, cap, s));
                k_decode_copy<<<grid, DC_THREADS, 0, s>>>(d_tok, n, d_off, d_bytes, entries, place, ctl, d_out, cap);
                B2_CUDA(cudaGetLastError());
            }
            *text = d_out;
            *n_bytes = h_ctl[0];
            d_out = nullptr;
            return B200BPE_OK;
        };
        const b200bpe_status r = work();
        if (r != B200BPE_OK) {
            cudaGetLastError();              // (an allocation that failed is nobody else's error)
            cudaStreamSynchronize(s);        // nothing is on its way to the pinned block
        }
        for (void* p : {(void*)d_tok, (void*)place, (void*)ctl, (void*)d_out}) ctx->free(p, s);
        ctx->free_pinned(pinned, pinned_bytes);
        return r;
    }

    b200bpe_status read(const uint8_t* text, uint8_t* out, uint64_t n) {
        if (n == 0) return B200BPE_OK;
        B2_CUDA(cudaMemcpyAsync(out, text, n, cudaMemcpyDeviceToHost, stream));
        B2_CUDA(cudaStreamSynchronize(stream));
        return B200BPE_OK;
    }
};

}  // namespace b200bpe

struct b200bpe_decoder { b200bpe::Decoder d; };

using namespace b200bpe;

extern "C" {

b200bpe_status b200bpe_decoder_create(b200bpe_ctx* c, const uint8_t* bytes, const uint64_t* offsets, uint32_t n_entries, b200bpe_decoder** out) {
    if (!c || !offsets || !out || n_entries == 0xFFFFFFFFu || offsets[0] != 0) return B200BPE_ERR_BAD_ARG;
    for (uint32_t i = 0; i < n_entries; i++) if (offsets[i + 1] < offsets[i]) return B200BPE_ERR_BAD_ARG;
    const uint64_t n = offsets[n_entries];
    if (!bytes && n) return B200BPE_ERR_BAD_ARG;
    B2_CUDA(cudaSetDevice(c->c.device));
    b200bpe_decoder* h = new b200bpe_decoder();
    Decoder& d = h->d;
    d.ctx = &c->c;
    d.hold.take(c);
    d.entries = n_entries;
    static const uint8_t replacement[3] = {0xEF, 0xBF, 0xBD};
    const uint64_t end = n + 3;
    cudaStream_t s = d.stream = c->c.decode_stream;
    cudaError_t e = c->c.alloc(&d.d_off, ((uint64_t)n_entries + 2) * 8, s);
    if (e == cudaSuccess) e = c->c.alloc(&d.d_bytes, end, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.d_off, offsets, ((uint64_t)n_entries + 1) * 8, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.d_off + n_entries + 1, &end, 8, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && n) e = cudaMemcpyAsync(d.d_bytes, bytes, n, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.d_bytes + n, replacement, 3, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { delete h; set_last_error(std::string("b200bpe_decoder_create: ") + cudaGetErrorString(e)); return e == cudaErrorMemoryAllocation ? B200BPE_ERR_OOM : B200BPE_ERR_CUDA; }
    *out = h;
    return B200BPE_OK;
}

b200bpe_status b200bpe_decoder_decode(b200bpe_decoder* h, const uint32_t* tokens, uint64_t n, uint8_t* out, uint64_t cap, uint64_t* n_bytes_out) {
    if (!h || (!tokens && n) || (!out && cap) || !n_bytes_out) return B200BPE_ERR_BAD_ARG;
    Decoder& d = h->d;
    B2_CUDA(cudaSetDevice(d.ctx->device));
    uint8_t* text = nullptr;
    b200bpe_status r = d.run(tokens, n, &text, n_bytes_out);
    if (r == B200BPE_OK) r = *n_bytes_out > cap ? B200BPE_ERR_CAPACITY : d.read(text, out, *n_bytes_out);
    d.ctx->free(text, d.stream);
    return r;
}

b200bpe_status b200bpe_decoder_run(b200bpe_decoder* h, const uint32_t* tokens, uint64_t n, uint64_t* n_bytes_out) {
    if (!h || (!tokens && n) || !n_bytes_out) return B200BPE_ERR_BAD_ARG;
    Decoder& d = h->d;
    B2_CUDA(cudaSetDevice(d.ctx->device));
    std::lock_guard<std::mutex> lock(d.mutex);
    d.ctx->free(d.d_text, d.stream);
    const b200bpe_status r = d.run(tokens, n, &d.d_text, &d.n_text);
    *n_bytes_out = d.n_text;
    return r;
}

b200bpe_status b200bpe_decoder_read(b200bpe_decoder* h, uint8_t* out, uint64_t cap) {
    if (!h) return B200BPE_ERR_BAD_ARG;
    Decoder& d = h->d;
    std::lock_guard<std::mutex> lock(d.mutex);
    if (!out && d.n_text) return B200BPE_ERR_BAD_ARG;
    if (cap < d.n_text) return B200BPE_ERR_CAPACITY;
    B2_CUDA(cudaSetDevice(d.ctx->device));
    return d.read(d.d_text, out, d.n_text);
}

void b200bpe_decoder_destroy(b200bpe_decoder* h) { delete h; }

}  // extern "C"
