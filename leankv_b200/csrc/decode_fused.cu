// One launch for everything between the fused q/k/v projection and attention in a decode step
// (one new token per sequence): rotary embedding of q and k, rotation of q into the key codebook's space, and
// rotate + Lloyd-Max quantize + 3-bit pack of the new k and v into their page.
//
// It produces bit for bit what leankv_rope_f16 + leankv_tq_pool_append (T_new = 1) +
// the query rotation of leankv_tq_decode_attn produce as three launches: same fp16 rounding
// points for the rotary step, same norm / division / ascending-k fma order for the rotations
// (the arithmetic contract stated at the top of tq_quantize.cu).

#include <algorithm>

#include "common.cuh"
#include "tq_layout.cuh"

namespace leankv {
namespace {

constexpr int kDim = LEANKV_TQ_DIM;

struct PostParams {
    const __half* qkv;        // [B][(nq + 2 nkv) * 128]
    const float* inv_freq;
    const int* pos;           // [B] position of the token being decoded
    const int* kv_indptr;     // [B + 1] offsets into page_indices, or nullptr (one sequence at offset 0)
    int B;
    const float* Pi_k_t;   // transposes of the rotations: Pi_k_t[k][j] = Pi_k[j][k]
    const float* Pi_v_t;
    const float* bounds;
    uint8_t* pool;
    int n_pages;
    const int32_t* page_indices;
    int nq, nkv;
    float* q_rot;             // [B][nq][128]
};

// A CTA serves one head for kSeqs sequences at a time, its rotation column in registers. What bounds it is the chain of
// one vector (the fp64 sum of 64 squares alone is 64 dependent steps), not any unit, so a batch takes four sequences
// through the chain together: 32 sequences, 48 heads: 21.9 -> 12.6 us. With kEarly position, page, shared word and rotary angles
// are there when the projections are: four steps of 32 layers of one sequence 8577 -> 8215 us; alone one sequence 3.5 -> 2.3, a
// batch of 32 10.3 -> 9.5 without and 8.7 with kEarly, of 80 24.4 -> 22.5 and 23.5 (hence without where a CTA walks several groups).
template <int kSeqs, bool kEarly>
__global__ void __launch_bounds__(kDim, kSeqs > 1 ? 3 : 1) decode_qkv_post_kernel(const PostParams p) {
    __shared__ float s_x[kSeqs][kDim];       // the head vectors (after rotary embedding, fp16 values)
    __shared__ __align__(16) float s_u[kSeqs][kDim];   // what gets rotated: x for q, x / (norm + 1e-10) for k and v
    __shared__ double s_ss[kSeqs][2];
    __shared__ float s_bounds[8];
    __shared__ __align__(4) uint8_t s_code[kSeqs][kDim];

    const int j = threadIdx.x;
    const int head = blockIdx.x;
    const int kind = head < p.nq ? 0 : (head < p.nq + p.nkv ? 1 : 2);   // 0 q, 1 k, 2 v
    // The rotation matrix is a constant of the cache, not an output of the previous kernel: fetch this
    // thread's column of it right away (128 independent loads, one memory round trip) so that it
    // is in registers by the time the vector has been prepared.
    const float* PiT = kind == 2 ? p.Pi_v_t : p.Pi_k_t;
    float pi_col[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) pi_col[k] = __ldg(PiT + k * kDim + j);
    const int row = (p.nq + 2 * p.nkv) * kDim;
    const int which = kind - 1;
    const int h = which == 0 ? head - p.nq : head - p.nq - p.nkv;
    // Where the new tokens go, the word of V shared with the pair token, and the rotary angles: with kEarly the first sequences' are there
    // when the projections are, else they are fetched beside the row, so that nothing trails the arithmetic.
    int slot[kSeqs];
    uint32_t* words[kSeqs];
    uint32_t old_word[kSeqs];
    __half2 turn[kSeqs];                                 // cosine, sine
    auto locate = [&](int b0) {
#pragma unroll
        for (int q = 0; q < kSeqs; ++q) {
            const int b = min(b0 + q, p.B - 1);          // a sequence beyond the batch is computed and not stored
            const int pos = p.pos[b];
            slot[q] = pos & 15;
            words[q] = nullptr;
            old_word[q] = 0;
            if (kind != 0 && b0 + q < p.B) {
                const int base = p.kv_indptr != nullptr ? p.kv_indptr[b] : 0;
                const int page = p.page_indices[base + (pos >> 4)];
                if (page >= 0 && page < p.n_pages) {
                    words[q] = reinterpret_cast<uint32_t*>(p.pool + (((size_t)page * 2 + which) * p.nkv + h) * kChunkBytes);
                    if (which == 1 && j < 24) {
                        const int g = j & 7, kk = j >> 3, pr = slot[q] >> 1;
                        old_word[q] = words[q][kk * 64 + (pr < 4 ? 4 * g + pr : 32 + 4 * g + (pr - 4))];
                    }
                }
            }
            if (kind != 2) {
                // cos/sin rounded to fp16 (HF apply_rotary_pos_emb)
                const float ang = (float)pos * p.inv_freq[j & 63];
                turn[q] = __halves2half2(__float2half_rn(cosf(ang)), __float2half_rn(sinf(ang)));
            }
        }
    };
    // one sequence: the code of `locate` once, around the wait; a batch: ahead of it and in the loop
    const int first = blockIdx.y * kSeqs;
    bool waited = kSeqs > 1 || !kEarly;
    if (kSeqs > 1 && kEarly) locate(first);
    if (waited) pdl_begin();
    for (int b0 = first; b0 < p.B; b0 += gridDim.y * kSeqs) {
        __half xr[kSeqs], other[kSeqs];
        auto load_rows = [&]() {
#pragma unroll
            for (int q = 0; q < kSeqs; ++q) {
                const __half* src = p.qkv + (size_t)min(b0 + q, p.B - 1) * row + (size_t)head * kDim;
                xr[q] = src[j];
                if (kind != 2) other[q] = src[j ^ 64];
            }
        };
        if (waited) load_rows();
        if (kSeqs == 1 || !kEarly || b0 != first) locate(b0);
        if (!waited) {
            pdl_begin();
            waited = true;
            load_rows();
        }
        if (j < 8) s_bounds[j] = j < 7 ? p.bounds[j] : __int_as_float(0x7f800000);
        float xf[kSeqs];
#pragma unroll
        for (int q = 0; q < kSeqs; ++q) {
            // rotate_half form: out[i] = x[i] cos - x[i+64] sin ; out[i+64] = x[i+64] cos + x[i] sin, products and sum in fp16
            const __half c = __low2half(turn[q]), s = __high2half(turn[q]);
            const __half xv = kind == 2 ? xr[q]
                              : j < 64  ? __hadd(__hmul(xr[q], c), __hmul(__hneg(other[q]), s))
                                        : __hadd(__hmul(xr[q], c), __hmul(other[q], s));
            xf[q] = __half2float(xv);
        }
        __syncthreads();                       // the previous sequences' readers of s_x / s_u / s_code are done
#pragma unroll
        for (int q = 0; q < kSeqs; ++q) s_x[q][j] = xf[q];
        __syncthreads();

        float norm[kSeqs];
        if (kind != 0) {
            // fp64 sums of squares of coordinates 0..63 and 64..127, ascending (one thread each)
            if ((j & 63) < kSeqs) {
                double ss = 0.0;
#pragma unroll 8
                for (int k = 0; k < 64; ++k) {
                    const double v = (double)s_x[j & 63][(j & 64) + k];
                    ss = fma(v, v, ss);
                }
                s_ss[j & 63][j >> 6] = ss;
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kSeqs; ++q) {
                norm[q] = (float)sqrt(s_ss[q][0] + s_ss[q][1]);
                s_u[q][j] = xf[q] / (norm[q] + 1e-10f);
            }
        } else {
#pragma unroll
            for (int q = 0; q < kSeqs; ++q) {
                norm[q] = 0.f;
                s_u[q][j] = xf[q];
            }
        }
        __syncthreads();

        // y_j = sum_k Pi[j][k] u[k], k ascending
        float y[kSeqs];
#pragma unroll
        for (int q = 0; q < kSeqs; ++q) y[q] = 0.f;
#pragma unroll
        for (int k = 0; k < kDim; k += 4) {
#pragma unroll
            for (int q = 0; q < kSeqs; ++q) {
                const float4 u = *reinterpret_cast<const float4*>(&s_u[q][k]);
                y[q] = fmaf(pi_col[k], u.x, y[q]);
                y[q] = fmaf(pi_col[k + 1], u.y, y[q]);
                y[q] = fmaf(pi_col[k + 2], u.z, y[q]);
                y[q] = fmaf(pi_col[k + 3], u.w, y[q]);
            }
        }
        if (kind == 0) {
#pragma unroll
            for (int q = 0; q < kSeqs; ++q)
                if (b0 + q < p.B) p.q_rot[((size_t)(b0 + q) * p.nq + head) * kDim + j] = y[q];
            continue;
        }
#pragma unroll
        for (int q = 0; q < kSeqs; ++q) {
            int code = 0;
#pragma unroll
            for (int i = 0; i < 7; ++i) code += (y[q] > s_bounds[i]) ? 1 : 0;
            s_code[q][j] = (uint8_t)code;
        }
        __syncthreads();

#pragma unroll
        for (int q = 0; q < kSeqs; ++q) {
            if (words[q] == nullptr) continue;
            uint8_t* chunk = reinterpret_cast<uint8_t*>(words[q]);
            if (j == 0) reinterpret_cast<__half*>(chunk + kNormOffsetBytes)[slot[q]] = __float2half_rn(norm[q]);

            // four codes per 32-bit shared-memory load; pack4 squeezes the low nibbles of 4 bytes into 16 bits
            auto pack4 = [](uint32_t v) -> uint32_t {
                const uint32_t t2 = (v | (v >> 4)) & 0x00FF00FFu;
                return (t2 | (t2 >> 8)) & 0xFFFFu;
            };
            if (which == 0) {
                if (j < 12) {                      // 4 units (quarters of the vector) x 3 words, this token only
                    const int t4 = j & 3, kk = j >> 2;
                    const uint32_t* c4 = reinterpret_cast<const uint32_t*>(&s_code[q][32 * t4]);
                    const uint32_t lo = c4[2 * kk] & 0x07070707u, hi = c4[2 * kk + 1] & 0x07070707u;
                    const uint32_t s_lo = ((c4[6] >> kk) & 0x01010101u) << 3, s_hi = ((c4[7] >> kk) & 0x01010101u) << 3;
                    words[q][kk * 64 + slot[q] * 4 + t4] = pack4(lo) | (pack4(hi) << 16) | pack4(s_lo) | (pack4(s_hi) << 16);
                }
            } else {
                if (j < 24) {                      // 8 units (16-coordinate groups) x 3 words, shared with the pair token
                    const int g = j & 7, kk = j >> 3;
                    const int pr = slot[q] >> 1, par = slot[q] & 1;
                    const int ui = pr < 4 ? 4 * g + pr : 32 + 4 * g + (pr - 4);
                    const uint32_t* ca = reinterpret_cast<const uint32_t*>(&s_code[q][16 * g]);
                    const uint32_t a4 = ca[kk] & 0x07070707u, as4 = (ca[3] >> kk) & 0x01010101u;
                    const uint32_t bits = par ? ((a4 << 4) | (as4 << 7)) : (a4 | (as4 << 3));
                    const uint32_t keep = par ? 0x0F0F0F0Fu : 0xF0F0F0F0u;   // the other token's nibbles
                    words[q][kk * 64 + ui] = bits | (old_word[q] & keep);
                }
            }
        }
    }
}

}  // namespace
}  // namespace leankv

using namespace leankv;

static int post_launch(const void* qkv, int B, const float* inv_freq, const int32_t* pos,
                       const int32_t* kv_indptr, const float* Pi_k_t, const float* Pi_v_t,
                       const float* decision_boundaries, void* pool, int n_pages, const int32_t* page_indices,
                       int n_q_heads, int n_kv_heads, float* q_rot, int flags, void* stream) {
    if (!qkv || !inv_freq || !pos || !Pi_k_t || !Pi_v_t || !decision_boundaries || !pool || !page_indices ||
        !q_rot || n_pages <= 0 || n_q_heads <= 0 || n_kv_heads <= 0 || B <= 0)
        return LEANKV_EINVAL;
    if (!aligned16(pool)) return LEANKV_EALIGN;
    PostParams p{};
    p.qkv = static_cast<const __half*>(qkv);
    p.inv_freq = inv_freq;
    p.pos = pos;
    p.kv_indptr = kv_indptr;
    p.B = B;
    p.Pi_k_t = Pi_k_t;
    p.Pi_v_t = Pi_v_t;
    p.bounds = decision_boundaries;
    p.pool = static_cast<uint8_t*>(pool);
    p.n_pages = n_pages;
    p.page_indices = page_indices;
    p.nq = n_q_heads;
    p.nkv = n_kv_heads;
    p.q_rot = q_rot;
    // One sequence alone keeps the kernel whose chain is its only work; a batch goes four at a time, over as many CTAs as are
    // resident at once (two or three an SM), each of which walks the rest of its head's sequences with the same column.
    const int heads = n_q_heads + 2 * n_kv_heads;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    bool early = (flags & LEANKV_POST_EARLY) != 0;
    if (B == 1) {
        LEANKV_CUDA_TRY(launch_kernel_ex(true, early ? decode_qkv_post_kernel<1, true> : decode_qkv_post_kernel<1, false>, dim3(heads, 1),
                                         dim3(kDim), 0, st, p));
    } else {
        constexpr int kSeqs = 4;
        const int groups = (B + kSeqs - 1) / kSeqs, gy = std::max(1, std::min(groups, 3 * sm_count() / heads));
        early = early && gy == groups;       // CTAs that walk several groups gain on the first only and pay on the others: 23.5 against 22.5
        LEANKV_CUDA_TRY(launch_kernel_ex(true, early ? decode_qkv_post_kernel<kSeqs, true> : decode_qkv_post_kernel<kSeqs, false>,
                                         dim3(heads, gy), dim3(kDim), 0, st, p));
    }
    return LEANKV_OK;
}

extern "C" int leankv_decode_qkv_post_flags(const void* qkv, const float* inv_freq, const int32_t* state,
                                            const float* Pi_k_t, const float* Pi_v_t, const float* decision_boundaries,
                                            void* pool, int n_pages, const int32_t* page_indices, int n_q_heads,
                                            int n_kv_heads, float* q_rot, int flags, void* stream) {
    return post_launch(qkv, 1, inv_freq, state /* state[0] = position */, nullptr, Pi_k_t, Pi_v_t,
                       decision_boundaries, pool, n_pages, page_indices, n_q_heads, n_kv_heads, q_rot, flags, stream);
}

extern "C" int leankv_decode_qkv_post(const void* qkv, const float* inv_freq, const int32_t* state,
                                      const float* Pi_k_t, const float* Pi_v_t,
                                      const float* decision_boundaries, void* pool, int n_pages,
                                      const int32_t* page_indices, int n_q_heads, int n_kv_heads,
                                      float* q_rot, void* stream) {
    return leankv_decode_qkv_post_flags(qkv, inv_freq, state, Pi_k_t, Pi_v_t, decision_boundaries, pool, n_pages, page_indices,
                                        n_q_heads, n_kv_heads, q_rot, 0, stream);
}

extern "C" int leankv_batch_qkv_post_flags(const void* qkv, int B, const float* inv_freq, const int32_t* pos,
                                           const int32_t* kv_indptr, const float* Pi_k_t, const float* Pi_v_t,
                                           const float* decision_boundaries, void* pool, int n_pages,
                                           const int32_t* kv_page_indices, int n_q_heads, int n_kv_heads,
                                           float* q_rot, int flags, void* stream) {
    if (!kv_indptr) return LEANKV_EINVAL;
    return post_launch(qkv, B, inv_freq, pos, kv_indptr, Pi_k_t, Pi_v_t, decision_boundaries, pool, n_pages,
                       kv_page_indices, n_q_heads, n_kv_heads, q_rot, flags, stream);
}

extern "C" int leankv_batch_qkv_post(const void* qkv, int B, const float* inv_freq, const int32_t* pos,
                                     const int32_t* kv_indptr, const float* Pi_k_t, const float* Pi_v_t,
                                     const float* decision_boundaries, void* pool, int n_pages,
                                     const int32_t* kv_page_indices, int n_q_heads, int n_kv_heads,
                                     float* q_rot, void* stream) {
    return leankv_batch_qkv_post_flags(qkv, B, inv_freq, pos, kv_indptr, Pi_k_t, Pi_v_t, decision_boundaries, pool, n_pages,
                                       kv_page_indices, n_q_heads, n_kv_heads, q_rot, 0, stream);
}
