// Small kernels that sit between the two hot paths in a batch-1 decode step of a
// Llama/Mistral-style block: embedding fetch, RMSNorm, rotary embedding, greedy argmax and
// the on-device bookkeeping of the sequence position / page table, so that a whole decode
// step can be replayed as one CUDA graph without the host touching per-step values.
// Rounding points follow the HF eager modules the reference runs around its kernels
// (transformers modeling_mistral.py: MistralRMSNorm, apply_rotary_pos_emb).

#include <algorithm>

#include "decode_frame.cuh"

namespace leankv {
namespace {

// Optional residual update h += delta (fp16 add, as the decoder block does), then
// y = w * fp16( h * rsqrt(mean(h^2) + eps) ), statistics in fp32.
// One CTA per row; 16-byte accesses; the (updated) row stays in registers between the two phases
// (n % 8 == 0, n <= kNormThreads * 8 * kNormVecs).
constexpr int kNormThreads = 512;
constexpr int kNormVecs = 4;
__global__ void __launch_bounds__(kNormThreads) rmsnorm_kernel(__half* x, const __half* delta,
                                                               const __half* w, __half* y, int n, float eps) {
    __shared__ float s_tmp[32];
    pdl_begin();
    const int nvec = n >> 3;
    x += (size_t)blockIdx.x * n;
    y += (size_t)blockIdx.x * n;
    if (delta != nullptr) delta += (size_t)blockIdx.x * n;
    uint4 v[kNormVecs];
    float ss = 0.f;
#pragma unroll
    for (int it = 0; it < kNormVecs; ++it) {
        const int i = threadIdx.x + it * kNormThreads;
        if (i < nvec) {
            uint4 a = reinterpret_cast<const uint4*>(x)[i];
            if (delta != nullptr) {
                const uint4 d = __ldg(reinterpret_cast<const uint4*>(delta) + i);
                __half2* ah = reinterpret_cast<__half2*>(&a);
                const __half2* dh = reinterpret_cast<const __half2*>(&d);
#pragma unroll
                for (int q = 0; q < 4; ++q) ah[q] = __hadd2(ah[q], dh[q]);
                reinterpret_cast<uint4*>(x)[i] = a;
            }
            v[it] = a;
            const __half2* ah = reinterpret_cast<const __half2*>(&a);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 f = __half22float2(ah[q]);
                ss = fmaf(f.x, f.x, ss);
                ss = fmaf(f.y, f.y, ss);
            }
        }
    }
    const float tot = cta_sum(ss, s_tmp);
    const float r = rsqrtf(tot / (float)n + eps);
#pragma unroll
    for (int it = 0; it < kNormVecs; ++it) {
        const int i = threadIdx.x + it * kNormThreads;
        if (i < nvec) {
            const uint4 wv = __ldg(reinterpret_cast<const uint4*>(w) + i);
            const __half2* ah = reinterpret_cast<const __half2*>(&v[it]);
            const __half2* wh = reinterpret_cast<const __half2*>(&wv);
            uint4 o;
            __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 f = __half22float2(ah[q]);
                oh[q] = __hmul2(wh[q], __floats2half2_rn(f.x * r, f.y * r));
            }
            reinterpret_cast<uint4*>(y)[i] = o;
        }
    }
}

// Rotary embedding (rotate_half form) on the q and k parts of a fused qkv row.
// cos/sin are rounded to fp16 and the products/sum are fp16, as in the HF module.
__global__ void __launch_bounds__(64) rope_kernel(const __half* qkv, const float* inv_freq,
                                                  const int* state, __half* q_out, __half* k_out,
                                                  int n_q_heads, int n_kv_heads) {
    pdl_begin();
    const int head = blockIdx.x;                 // q heads first, then k heads
    const int i = threadIdx.x;                   // 0..63
    const float ang = (float)state[kPos] * inv_freq[i];
    const __half c = __float2half_rn(cosf(ang)), s = __float2half_rn(sinf(ang));
    const __half* src = qkv + (size_t)head * 128;
    __half* dst = head < n_q_heads ? q_out + (size_t)head * 128
                                   : k_out + (size_t)(head - n_q_heads) * 128;
    const __half a = src[i], b = src[i + 64];
    dst[i] = __hadd(__hmul(a, c), __hmul(__hneg(b), s));
    dst[i + 64] = __hadd(__hmul(b, c), __hmul(a, s));
}

// Greedy next token (as decode_end_kernel) for an output head that is split over the vocabulary among tensor-parallel ranks: every
// rank finds the best of its own slice, sends {value, index} (two 64-bit words, each tagged with the
// step's epoch like the partial sums of the row-parallel GEMV) to every rank's receive area, waits
// (bounded) for all ranks' words, and takes the largest value, lowest index on ties: every rank
// arrives at the same token. As the last exchange of a step it also moves the epoch on.
struct ShardedEndParams {
    const __half* logits;      // this rank's slice [vocab_local]
    int vocab_local, vocab_offset;
    long long* token;
    long long* history;
    int history_cap;
    int* pos;
    int* step_ptr;
    int world, rank, limit;
    unsigned long long* recv[LEANKV_MAX_RANKS];   // slot base in every rank's area: [world][2] words
    int* epoch;
    int* status;
};

__global__ void __launch_bounds__(1024) decode_end_sharded_kernel(const ShardedEndParams p) {
    __shared__ float s_v[32];
    __shared__ int s_i[32];
    pdl_begin();
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    const int nvec = p.vocab_local >> 3;      // vocab_local % 8 == 0 (checked on the host)
    for (int vi = threadIdx.x; vi < nvec; vi += blockDim.x) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(p.logits) + vi);
        const __half* hp = reinterpret_cast<const __half*>(&a);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float v = __half2float(hp[q]);
            if (v > best) { best = v; best_i = vi * 8 + q; }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { s_v[warp] = best; s_i[warp] = best_i; }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
        if (s_v[w] > best || (s_v[w] == best && s_i[w] < best_i)) { best = s_v[w]; best_i = s_i[w]; }
    if (best_i != 0x7fffffff) best_i += p.vocab_offset;

    const unsigned int ep = (unsigned int)*reinterpret_cast<volatile int*>(p.epoch);
    const unsigned long long tag = (unsigned long long)ep << 32;
    for (int i = 0; i < p.world; ++i) {
        int r = p.rank + i;
        r = r >= p.world ? r - p.world : r;
        unsigned long long* dst = p.recv[r] + 2 * p.rank;
        asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(dst), "l"(tag | __float_as_uint(best)) : "memory");
        asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(dst + 1), "l"(tag | (unsigned int)best_i) : "memory");
    }
    const bool live = *reinterpret_cast<volatile int*>(p.status) == 0;
    bool ok = live;
    float top = -INFINITY;
    int top_i = 0x7fffffff;
    const unsigned long long* src = p.recv[p.rank];
    for (int r = 0; r < p.world && live; ++r) {
        unsigned long long wv = 0, wi = 0;
        int it = 0;
        for (;;) {
            asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(wv) : "l"(src + 2 * r) : "memory");
            asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(wi) : "l"(src + 2 * r + 1) : "memory");
            if (((unsigned int)(wv >> 32) == ep && (unsigned int)(wi >> 32) == ep) || it >= p.limit) break;
            __nanosleep(20);
            ++it;
        }
        if ((unsigned int)(wv >> 32) != ep || (unsigned int)(wi >> 32) != ep) {
            ok = false;
            continue;
        }
        const float v = __uint_as_float((unsigned int)wv);
        const int idx = (int)(unsigned int)wi;
        if (v > top || (v == top && idx < top_i)) { top = v; top_i = idx; }
    }
    if (!ok && live) atomicOr(p.status, 1);
    if (top_i == 0x7fffffff) top_i = 0;      // all-NaN rows, or a dead exchange
    *p.token = top_i;
    const int step = *p.step_ptr;
    if (step < p.history_cap) p.history[step] = top_i;
    *p.step_ptr = step + 1;
    *p.pos = *p.pos + 1;
    *p.epoch = (int)(ep + 1u);
}

// Batched step prologue: embedding rows of B tokens, and the flat page table of this step built from
// a per-sequence block table. Sequence b caches pos[b] tokens and appends one: it uses
// pos[b] / 16 + 1 pages, the first entries of block_table[b][0..max_pps). One CTA per sequence; each
// derives its own offset from the positions of the sequences before it, so no CTA waits on another.
__global__ void __launch_bounds__(256) batch_begin_kernel(const __half* table, const long long* tokens,
                                                          __half* h, int hidden, int vocab, int B,
                                                          const int* pos, const int* block_table, int max_pps,
                                                          int* kv_indptr, int* kv_page_indices,
                                                          int* kv_last_page_len) {
    __shared__ int s_part[8];
    pdl_begin();
    const int b = blockIdx.x;
    long long tok = tokens[b];
    if (tok < 0 || tok >= vocab) tok = 0;
    const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)tok * hidden);
    uint4* dst = reinterpret_cast<uint4*>(h + (size_t)b * hidden);
    for (int i = threadIdx.x; i < hidden / 8; i += blockDim.x) dst[i] = __ldg(src + i);

    int before = 0;
    for (int i = threadIdx.x; i < b; i += blockDim.x) before += min(pos[i] / 16 + 1, max_pps);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = before;
    __syncthreads();
    int start = 0;
    for (int w = 0; w < 8; ++w) start += s_part[w];
    const int mine = min(pos[b] / 16 + 1, max_pps);
    for (int i = threadIdx.x; i < mine; i += blockDim.x)
        kv_page_indices[start + i] = block_table[(size_t)b * max_pps + i];
    if (threadIdx.x == 0) {
        kv_indptr[b] = start;
        if (b == B - 1) kv_indptr[B] = start + mine;
        kv_last_page_len[b] = pos[b] % 16 + 1;
    }
}

__device__ __forceinline__ uint4 silu_mul8(const uint4& g, const uint4& u) {
    const __half2* gh = reinterpret_cast<const __half2*>(&g);
    const __half2* uh = reinterpret_cast<const __half2*>(&u);
    uint4 o;
    __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 f = __half22float2(gh[q]);
        const __half2 act = __floats2half2_rn(f.x / (1.f + expf(-f.x)), f.y / (1.f + expf(-f.y)));
        oh[q] = __hmul2(act, uh[q]);
    }
    return o;
}

// out = fp16(silu(gate)) * up, the rounding points of the HF MLP (act_fn output is an fp16 tensor).
// gate, up: rows of `inter`, `ld` apart; out: [rows][inter]. The exponential and the division are the work, not the 44 MB of 512 x
// 14336, which stay in L2: 9.1 us with as many blocks as fit at once, whose last round was nearly empty, and a 64-bit division for
// the row of every eight columns; 7.5 with a block for every 2048 columns of a row.
__global__ void __launch_bounds__(256) silu_mul_kernel(const __half* gate, const __half* up, size_t ld, __half* out, int inter, int rows) {
    pdl_begin();
    const int nvec = inter >> 3, c = blockIdx.x * 256 + threadIdx.x;
    if (c >= nvec) return;
    for (int r = blockIdx.y; r < rows; r += gridDim.y) {
        const uint4 g = reinterpret_cast<const uint4*>(gate + (size_t)r * ld)[c];        // out may be gate or up
        const uint4 u = reinterpret_cast<const uint4*>(up + (size_t)r * ld)[c];
        reinterpret_cast<uint4*>(out + (size_t)r * inter)[c] = silu_mul8(g, u);
    }
}

// The same for many short rows, whose blocks would be mostly idle: over all pieces in one walk. us by rows / so: 4096 x 256 4.6 / 2.5, 4096 x
// 512 4.6 / 3.7, 65536 x 64 68 / 6.3 (the rate at which blocks start), but 2048 x 768 3.1 / 3.5 and 512 x 256 1.6 / 1.6.
constexpr int kShortRow = 768, kManyRows = 1024;
__global__ void __launch_bounds__(256) silu_mul_short_kernel(const __half* gate, const __half* up, size_t ld, __half* out, int inter, int rows) {
    pdl_begin();
    const int nvec = inter >> 3;
    const long long total = (long long)rows * nvec;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / nvec;
        const int c = (int)(i - r * nvec);
        const uint4 g = reinterpret_cast<const uint4*>(gate + (size_t)r * ld)[c], u = reinterpret_cast<const uint4*>(up + (size_t)r * ld)[c];
        reinterpret_cast<uint4*>(out + (size_t)r * inter)[c] = silu_mul8(g, u);
    }
}

// A prompt chunk's projections [T][(n_q + 2 n_kv) heads][128] into what the cache and attention read: queries [T][n_q][128]
// and keys [n_kv][T][128] turned by their position (cos, sin: fp16 [T][128], halves equal; fp16 products and sum, as in
// rope_kernel), values [n_kv][T][128] as they are. Eight lanes a (token, head), 32 bytes each, whole rows of 256 bytes on both
// sides. As tensor operations (negate, concatenate, two products, sum, two transposes) the same took 45 us of a layer with
// 512 tokens; here 3.
__global__ void __launch_bounds__(256) rope_split_kernel(const __half* qkv, const __half* cos_t, const __half* sin_t, __half* q,
                                                         __half* k, __half* v, int T, int n_q, int n_kv) {
    pdl_begin();
    const int heads = n_q + 2 * n_kv;
    const long long i = (long long)blockIdx.x * 32 + (threadIdx.x >> 3);
    if (i >= (long long)T * heads) return;
    const int t = (int)(i / heads), head = (int)(i - (long long)t * heads), c = threadIdx.x & 7;
    const uint4* src = reinterpret_cast<const uint4*>(qkv + i * 128) + c;
    uint4 lo = __ldg(src), hi = __ldg(src + 8);
    __half* dst = head < n_q ? q + ((size_t)t * n_q + head) * 128
                : head < n_q + n_kv ? k + ((size_t)(head - n_q) * T + t) * 128 : v + ((size_t)(head - n_q - n_kv) * T + t) * 128;
    if (head < n_q + n_kv) {
        const uint4 cv = __ldg(reinterpret_cast<const uint4*>(cos_t + (size_t)t * 128) + c);
        const uint4 sv = __ldg(reinterpret_cast<const uint4*>(sin_t + (size_t)t * 128) + c);
        const __half2* ch = reinterpret_cast<const __half2*>(&cv);
        const __half2* sh = reinterpret_cast<const __half2*>(&sv);
        __half2* a = reinterpret_cast<__half2*>(&lo);
        __half2* b = reinterpret_cast<__half2*>(&hi);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __half2 x = a[j], y = b[j];
            a[j] = __hadd2_rn(__hmul2_rn(x, ch[j]), __hmul2_rn(__hneg2(y), sh[j]));
            b[j] = __hadd2_rn(__hmul2_rn(y, ch[j]), __hmul2_rn(x, sh[j]));
        }
    }
    reinterpret_cast<uint4*>(dst)[c] = lo;
    reinterpret_cast<uint4*>(dst)[c + 8] = hi;
}

// What the layers of a prompt chunk share: the rotary tables fp16 [T][128] of positions start .. start + T - 1 (halves equal; angles,
// cosines and sines in fp32, as in rope_kernel), and the two small vectors that the append reads. As tensor operations and two uploads
// this was eleven launches and a wait of the host for the device in front of every chunk. Here one launch: 40 tokens through two
// layers of width 1024, where the launches are the time, 677 -> 586 us; 600 in three chunks through four of 2048, 2485 -> 2222.
__global__ void __launch_bounds__(256) prompt_begin_kernel(const float* inv_freq, int T, int start, int n_pages, __half* cos_t,
                                                           __half* sin_t, int32_t* indptr, int32_t* start_out) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    const int t = (int)(i >> 5), j = (int)(i & 31);                      // two neighbouring angles of a token
    const float pos = (float)(start + min(t, T - 1));
    const float2 rate = __ldg(reinterpret_cast<const float2*>(inv_freq) + j);
    const float a = pos * rate.x, b = pos * rate.y;
    const __half2 c = __floats2half2_rn(cosf(a), cosf(b)), s = __floats2half2_rn(sinf(a), sinf(b));
    pdl_begin();
    if (i == 0) {
        indptr[0] = 0;
        indptr[1] = n_pages;
        *start_out = start;
    }
    if (t >= T) return;
    __half2* ct = reinterpret_cast<__half2*>(cos_t + (size_t)t * 128) + j;
    __half2* st = reinterpret_cast<__half2*>(sin_t + (size_t)t * 128) + j;
    ct[0] = c; ct[32] = c;
    st[0] = s; st[32] = s;
}

}  // namespace
}  // namespace leankv

using namespace leankv;

extern "C" int leankv_rmsnorm_f16(void* x, const void* delta, const void* weight, void* y, int n,
                                  float eps, void* stream) {
    if (!x || !weight || !y || n <= 0) return LEANKV_EINVAL;
    if (n % 8 != 0 || !aligned16(x) || !aligned16(weight) || !aligned16(y) || (delta && !aligned16(delta)))
        return LEANKV_EALIGN;
    if (n > kNormThreads * 8 * kNormVecs) return LEANKV_ELIMIT;
    LEANKV_CUDA_TRY(launch_early(rmsnorm_kernel, dim3(1), dim3(kNormThreads), 0, static_cast<cudaStream_t>(stream),
                                  static_cast<__half*>(x), static_cast<const __half*>(delta),
                                  static_cast<const __half*>(weight), static_cast<__half*>(y), n, eps));
    return LEANKV_OK;
}

extern "C" int leankv_decode_begin(const void* embed_table, const long long* token, void* h,
                                   int hidden, int vocab, int32_t* state, void* stream) {
    if (!embed_table || !token || !h || !state || hidden <= 0 || vocab <= 0) return LEANKV_EINVAL;
    if (hidden % 8 != 0 || !aligned16(embed_table) || !aligned16(h)) return LEANKV_EALIGN;
    LEANKV_CUDA_TRY(launch_early(decode_begin_kernel<__half, __half>, dim3(1), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                  static_cast<const __half*>(embed_table), token, static_cast<__half*>(h),
                                  hidden, vocab, state));
    return LEANKV_OK;
}

extern "C" int leankv_rope_f16(const void* qkv, const float* inv_freq, const int32_t* state,
                               void* q_out, void* k_out, int n_q_heads, int n_kv_heads,
                               int head_dim, void* stream) {
    if (!qkv || !inv_freq || !state || !q_out || !k_out || n_q_heads <= 0 || n_kv_heads <= 0)
        return LEANKV_EINVAL;
    if (head_dim != 128) return LEANKV_EUNSUPPORTED;
    LEANKV_CUDA_TRY(launch_early(rope_kernel, dim3(n_q_heads + n_kv_heads), dim3(64), 0,
                                  static_cast<cudaStream_t>(stream), static_cast<const __half*>(qkv), inv_freq,
                                  state, static_cast<__half*>(q_out), static_cast<__half*>(k_out), n_q_heads,
                                  n_kv_heads));
    return LEANKV_OK;
}

extern "C" int leankv_decode_end(const void* logits, int vocab, long long* token, long long* history,
                                 int history_cap, int32_t* state, void* stream) {
    if (!logits || !token || !history || !state || vocab <= 0 || history_cap < 0) return LEANKV_EINVAL;
    if (!aligned16(logits)) return LEANKV_EALIGN;
    LEANKV_CUDA_TRY(launch_early(decode_end_kernel<__half, 8>, dim3(8), dim3(end_threads(8)), 0, static_cast<cudaStream_t>(stream),
                                  static_cast<const __half*>(logits), vocab, token, history, history_cap,
                                  state + kPos, state + kStep, static_cast<int*>(nullptr)));
    return LEANKV_OK;
}

extern "C" int leankv_decode_end_sharded(const void* logits_local, int vocab_local, int vocab_offset,
                                         long long* token, long long* history, int history_cap, int32_t* state,
                                         const leankv_xchg_t* xchg, int slot, void* stream) {
    if (!logits_local || !token || !history || !state || !xchg || vocab_local <= 0 || vocab_offset < 0 ||
        history_cap < 0)
        return LEANKV_EINVAL;
    if (vocab_local % 8 != 0 || !aligned16(logits_local)) return LEANKV_EALIGN;
    if (xchg->world < 1 || xchg->world > LEANKV_MAX_RANKS || xchg->rank < 0 || xchg->rank >= xchg->world ||
        slot < 0 || slot >= xchg->n_slots || 2 * xchg->world > xchg->world * xchg->max_cols || !xchg->epoch ||
        !xchg->status || xchg->max_wait_iters < 1)
        return LEANKV_EINVAL;
    ShardedEndParams p{};
    p.logits = static_cast<const __half*>(logits_local);
    p.vocab_local = vocab_local;
    p.vocab_offset = vocab_offset;
    p.token = token;
    p.history = history;
    p.history_cap = history_cap;
    p.pos = state + kPos;
    p.step_ptr = state + kStep;
    p.world = xchg->world;
    p.rank = xchg->rank;
    p.limit = xchg->max_wait_iters;
    for (int r = 0; r < xchg->world; ++r) {
        if (!xchg->recv[r] || (reinterpret_cast<uintptr_t>(xchg->recv[r]) & 7u) != 0) return LEANKV_EINVAL;
        p.recv[r] = static_cast<unsigned long long*>(xchg->recv[r]) + (size_t)slot * xchg->world * xchg->max_cols;
    }
    p.epoch = const_cast<int*>(xchg->epoch);
    p.status = xchg->status;
    LEANKV_CUDA_TRY(launch_kernel(decode_end_sharded_kernel, dim3(1), dim3(1024), 0,
                                  static_cast<cudaStream_t>(stream), p));
    return LEANKV_OK;
}

extern "C" int leankv_rmsnorm_rows_f16(void* x, const void* delta, const void* weight, void* y, int rows, int n,
                                       float eps, void* stream) {
    if (!x || !weight || !y || n <= 0 || rows <= 0) return LEANKV_EINVAL;
    if (n % 8 != 0 || !aligned16(x) || !aligned16(weight) || !aligned16(y) || (delta && !aligned16(delta)))
        return LEANKV_EALIGN;
    if (n > kNormThreads * 8 * kNormVecs) return LEANKV_ELIMIT;
    LEANKV_CUDA_TRY(launch_early(rmsnorm_kernel, dim3(rows), dim3(kNormThreads), 0,
                                  static_cast<cudaStream_t>(stream), static_cast<__half*>(x),
                                  static_cast<const __half*>(delta), static_cast<const __half*>(weight),
                                  static_cast<__half*>(y), n, eps));
    return LEANKV_OK;
}

extern "C" int leankv_batch_decode_begin(const void* embed_table, const long long* tokens, void* h, int hidden,
                                         int vocab, int B, const int32_t* pos, const int32_t* block_table,
                                         int max_pages_per_seq, int32_t* kv_indptr, int32_t* kv_page_indices,
                                         int32_t* kv_last_page_len, void* stream) {
    if (!embed_table || !tokens || !h || !pos || !block_table || !kv_indptr || !kv_page_indices ||
        !kv_last_page_len || hidden <= 0 || vocab <= 0 || B <= 0 || max_pages_per_seq <= 0)
        return LEANKV_EINVAL;
    if (hidden % 8 != 0 || !aligned16(embed_table) || !aligned16(h)) return LEANKV_EALIGN;
    LEANKV_CUDA_TRY(launch_early(batch_begin_kernel, dim3(B), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                  static_cast<const __half*>(embed_table), tokens, static_cast<__half*>(h), hidden,
                                  vocab, B, pos, block_table, max_pages_per_seq, kv_indptr, kv_page_indices,
                                  kv_last_page_len));
    return LEANKV_OK;
}

static int launch_silu_mul(const void* gate, const void* up, size_t ld, void* out, int rows, int inter, void* stream) {
    const long long blocks = ((long long)rows * (inter / 8) + 255) / 256;
    const bool is_short = inter < kShortRow && rows > kManyRows;
    const dim3 grid = is_short ? dim3((unsigned)std::min<long long>(blocks, sm_count() * 8LL))
                               : dim3((inter / 8 + 255) / 256, std::min(rows, 65535));
    LEANKV_CUDA_TRY(launch_early(is_short ? silu_mul_short_kernel : silu_mul_kernel, grid, dim3(256), 0, static_cast<cudaStream_t>(stream),
                                  static_cast<const __half*>(gate), static_cast<const __half*>(up), ld,
                                  static_cast<__half*>(out), inter, rows));
    return LEANKV_OK;
}

extern "C" int leankv_silu_mul_f16(const void* gate_up, void* out, int rows, int inter, void* stream) {
    if (!gate_up || !out || rows <= 0 || inter <= 0) return LEANKV_EINVAL;
    if (inter % 8 != 0 || !aligned16(gate_up) || !aligned16(out)) return LEANKV_EALIGN;
    return launch_silu_mul(gate_up, static_cast<const __half*>(gate_up) + inter, 2 * (size_t)inter, out, rows, inter, stream);
}

extern "C" int leankv_silu_mul_pair_f16(const void* gate, const void* up, void* out, int rows, int inter, void* stream) {
    if (!gate || !up || !out || rows <= 0 || inter <= 0) return LEANKV_EINVAL;
    if (inter % 8 != 0 || !aligned16(gate) || !aligned16(up) || !aligned16(out)) return LEANKV_EALIGN;
    return launch_silu_mul(gate, up, (size_t)inter, out, rows, inter, stream);
}

extern "C" int leankv_prompt_begin_f16(const float* inv_freq, int T, int start, void* cos, void* sin, int32_t* indptr,
                                       int32_t* start_out, void* stream) {
    if (!inv_freq || !cos || !sin || !indptr || !start_out || T <= 0 || start < 0) return LEANKV_EINVAL;
    if (start > 0x7fffffff - 15 - T) return LEANKV_ELIMIT;
    if (!aligned16(inv_freq) || !aligned16(cos) || !aligned16(sin)) return LEANKV_EALIGN;
    const long long blocks = ((long long)T * 32 + 255) / 256;
    LEANKV_CUDA_TRY(launch_early(prompt_begin_kernel, dim3((unsigned)blocks), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                 inv_freq, T, start, (start + T + 15) / 16, static_cast<__half*>(cos), static_cast<__half*>(sin),
                                 indptr, start_out));
    return LEANKV_OK;
}

extern "C" int leankv_rope_split_f16(const void* qkv, const void* cos, const void* sin, void* q, void* k, void* v, int T,
                                     int n_q_heads, int n_kv_heads, void* stream) {
    if (!qkv || !cos || !sin || !q || !k || !v || T <= 0 || n_q_heads <= 0 || n_kv_heads <= 0) return LEANKV_EINVAL;
    if (!aligned16(qkv) || !aligned16(cos) || !aligned16(sin) || !aligned16(q) || !aligned16(k) || !aligned16(v))
        return LEANKV_EALIGN;
    const long long blocks = ((long long)T * ((long long)n_q_heads + 2ll * n_kv_heads) + 31) / 32;
    if (blocks > 0x7fffffffll) return LEANKV_ELIMIT;
    LEANKV_CUDA_TRY(launch_early(rope_split_kernel, dim3((unsigned)blocks), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                  static_cast<const __half*>(qkv), static_cast<const __half*>(cos),
                                  static_cast<const __half*>(sin), static_cast<__half*>(q), static_cast<__half*>(k),
                                  static_cast<__half*>(v), T, n_q_heads, n_kv_heads));
    return LEANKV_OK;
}

extern "C" int leankv_batch_decode_end(const void* logits, int vocab, int B, long long* tokens,
                                       long long* history, int history_cap, int32_t* pos, int32_t* steps,
                                       void* stream) {
    if (!logits || !tokens || !history || !pos || !steps || vocab <= 0 || B <= 0 || history_cap < 0)
        return LEANKV_EINVAL;
    if (!aligned16(logits) || vocab % 8 != 0) return LEANKV_EALIGN;
    const int ctas = end_ctas(B, vocab);
    LEANKV_CUDA_TRY(launch_early(ctas == 1 ? decode_end_kernel<__half, 1> : decode_end_kernel<__half, 8>, dim3(B * ctas), dim3(end_threads(ctas)), 0, static_cast<cudaStream_t>(stream),
                                  static_cast<const __half*>(logits), vocab, tokens, history, history_cap, pos,
                                  steps, static_cast<int*>(nullptr)));
    return LEANKV_OK;
}

// ---------------------------------------------------------------------------------------------
// Page table of a paged cache kept on the device (replaces the host loops of
// leankv/turboquant/paged_cache.py:96-103 (_allocate_page), :147-164 (page assignment in update) and
// :215-233 (flat metadata for the attention call)).
// ---------------------------------------------------------------------------------------------
namespace leankv {
namespace {

constexpr int kTableThreads = 1024;

// A new page table in one launch: `zeros` words of zero in front of the stack of free pages 0, 1, .., n - 1 and its height. As three
// tensor operations: clearing a cache took the host 45 - 59 us, so 38 - 41; a prompt of 2048 tokens in four chunks 305 -> 291.
__global__ void __launch_bounds__(256) paged_table_begin_kernel(int32_t* words, int zeros, int n, int top) {
    pdl_begin();
    for (long long i = blockIdx.x * 256 + threadIdx.x; i <= top; i += gridDim.x * 256)
        words[i] = i < zeros ? 0 : i < top ? (int)i - zeros : n;
}

// One CTA. Sequence b grows by t_new tokens: it takes the pages it lacks from the top of the free
// stack (sequence 0 first, as the reference's loop does), its length advances, and the flat
// (kv_indptr, kv_page_indices, kv_last_page_len, start_pos) arrays of the append / attention calls are
// rebuilt. If the stack does not hold enough pages nothing changes and status bit 0 is set.
// The time is barriers and round trips to L2: the scans take log2(B) steps, not log2 of the CTA, and a warp moves a
// sequence's page ids (one thread a sequence walked 125 ids one after another: 8.4 us for a 2000-token sequence, now 2.7).
__global__ void __launch_bounds__(kTableThreads) paged_table_step_kernel(
    int t_new, int B, int32_t* seq_len, int32_t* block_table, int pps_cap, int32_t* free_stack, int32_t* free_top,
    int32_t* kv_indptr, int32_t* kv_page_indices, int32_t* kv_last_page_len, int32_t* start_pos, int32_t* status) {
    __shared__ int s_scan[kTableThreads];
    __shared__ int s_have[kTableThreads], s_need[kTableThreads], s_first[kTableThreads], s_off[kTableThreads];
    __shared__ int s_fail, s_top;
    pdl_begin();
    const int b = threadIdx.x, warp = b >> 5, lane = b & 31;
    const int len = b < B ? seq_len[b] : 0;
    const int have = (len + 15) / 16;
    const int want = b < B ? (len + t_new + 15) / 16 : 0;
    const int need = max(want - have, 0);
    // inclusive scans (Hillis-Steele over the first B threads) of the pages needed and of the pages held afterwards
    auto scan = [&](int v) -> int {
        s_scan[b] = v;
        __syncthreads();
        for (int o = 1; o < B; o <<= 1) {
            const int add = b >= o ? s_scan[b - o] : 0;
            __syncthreads();
            s_scan[b] += add;
            __syncthreads();
        }
        const int incl = s_scan[b];
        __syncthreads();
        return incl;
    };
    const int need_incl = scan(need);
    const int overflow = __syncthreads_or(b < B && want > pps_cap);   // a row of the block table would not hold it
    if (b == B - 1) {
        const int total = need_incl, top = *free_top;                 // the last sequence's inclusive sum is the total
        const bool fail = total > top || overflow != 0;
        if (total > top) atomicOr(status, 1);
        if (overflow) atomicOr(status, 2);
        if (!fail) *free_top = top - total;
        s_fail = fail ? 1 : 0;
        s_top = top;
    }
    __syncthreads();
    const int top = s_top;
    const bool grows = s_fail == 0 && b < B;
    const int new_len = grows ? len + t_new : len;
    if (grows) seq_len[b] = new_len;
    const int pages_now = b < B ? (new_len + 15) / 16 : 0;
    const int pages_incl = scan(pages_now);
    if (b < B) {
        start_pos[b] = len;
        kv_indptr[b + 1] = pages_incl;
        if (b == 0) kv_indptr[0] = 0;
        const int rem = new_len % 16;
        kv_last_page_len[b] = rem > 0 ? rem : 16;        // 0 -> page_size, the reference's convention (:225-226)
    }
    s_have[b] = grows ? have : pages_now;                // pages that the block table holds already; the rest come off the stack
    s_need[b] = grows ? need : 0;
    s_first[b] = need_incl - need;                       // pages popped by sequences before this one
    s_off[b] = pages_incl - pages_now;
    __syncthreads();
    for (int s = warp; s < B; s += kTableThreads / 32) {
        int32_t* row = block_table + (size_t)s * pps_cap;
        int32_t* flat = kv_page_indices + s_off[s];
        const int held = s_have[s], more = s_need[s], first = s_first[s];
        for (int i = lane; i < held; i += 32) flat[i] = row[i];
        for (int i = lane; i < more; i += 32) {
            const int page = free_stack[top - 1 - first - i];
            row[held + i] = page;
            flat[held + i] = page;
        }
    }
}

}  // namespace
}  // namespace leankv

extern "C" int leankv_paged_table_begin(int32_t* words, int zeros, int max_pages, int top, void* stream) {
    if (!words || zeros < 0 || max_pages <= 0 || top < zeros || top - zeros < max_pages) return LEANKV_EINVAL;
    const int grid = std::min(top / 256 + 1, sm_count() * 8);
    LEANKV_CUDA_TRY(launch_early(paged_table_begin_kernel, dim3(grid), dim3(256), 0, static_cast<cudaStream_t>(stream), words, zeros,
                                 max_pages, top));
    return LEANKV_OK;
}

extern "C" int leankv_paged_table_step(int t_new, int B, int32_t* seq_len, int32_t* block_table,
                                       int max_pages_per_seq, int32_t* free_stack, int32_t* free_top,
                                       int32_t* kv_indptr, int32_t* kv_page_indices, int32_t* kv_last_page_len,
                                       int32_t* start_pos, int32_t* status, void* stream) {
    if (t_new < 0 || B <= 0 || max_pages_per_seq <= 0 || !seq_len || !block_table || !free_stack || !free_top ||
        !kv_indptr || !kv_page_indices || !kv_last_page_len || !start_pos || !status)
        return LEANKV_EINVAL;
    if (B > kTableThreads) return LEANKV_ELIMIT;
    LEANKV_CUDA_TRY(launch_early(paged_table_step_kernel, dim3(1), dim3(kTableThreads), 0,
                                  static_cast<cudaStream_t>(stream), t_new, B, seq_len, block_table, max_pages_per_seq,
                                  free_stack, free_top, kv_indptr, kv_page_indices, kv_last_page_len, start_pos,
                                  status));
    return LEANKV_OK;
}
