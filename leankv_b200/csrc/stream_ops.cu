// Row-wise kernels around the projections of a prompt portion (residual sum, norm, token shift, gating) and
// the two frame kernels of a decode step whose residual stream is fp32.

#include <algorithm>

#include "decode_frame.cuh"
#include "leankv_mixers.h"

namespace leankv {
namespace {

constexpr int kRowThreads = 256;

// One CTA per row. With token shift the row above is normed a second time here (two rows of L2 reads)
// rather than handed over through memory, so rows stay independent and one launch does the whole chain.
template <typename T, typename D>
__global__ void __launch_bounds__(kRowThreads) stream_norm_kernel(const leankv_stream_norm_t a) {
    __shared__ float s_tmp[32];
    pdl_begin();
    const int t = blockIdx.x, W = a.width;
    const D* delta = static_cast<const D*>(a.delta);
    const float* scale = a.post_gain != nullptr ? a.post_gain : a.scale;
    const bool shift = a.n_mix > 0;
    auto branch_factor = [&](int row) {         // of a branch that is normed before it joins the stream
        if (a.post_gain == nullptr) return 1.f;
        float ss = 0.f;
        for (int i = threadIdx.x; i < W; i += kRowThreads) {
            const float d = to_f32(delta[(size_t)row * W + i]);
            ss = fmaf(d, d, ss);
        }
        return a.post_mult / sqrtf(cta_sum(ss, s_tmp) / (float)W + a.eps);
    };
    const float f_here = branch_factor(t), f_above = shift && t > 0 ? branch_factor(t - 1) : 1.f;
    auto value = [&](int row, int i) {
        float x = a.x_in[(size_t)row * W + i];
        if (delta != nullptr)
            x = fmaf(to_f32(delta[(size_t)row * W + i]) * (row == t ? f_here : f_above), __ldg(scale + i), x);
        return x;
    };
    float ss = 0.f, ss_above = 0.f;
    for (int i = threadIdx.x; i < W; i += kRowThreads) {
        const float x = value(t, i);
        ss = fmaf(x, x, ss);
        if (delta != nullptr) a.x_out[(size_t)t * W + i] = x;
        if (shift && t > 0) {
            const float y = value(t - 1, i);
            ss_above = fmaf(y, y, ss_above);
        }
    }
    if (a.gain == nullptr) return;
    const float gain = a.gain_per_col ? 1.f : __ldg(a.gain);
    const float rs = gain / sqrtf(cta_sum(ss, s_tmp) / (float)W + a.eps);
    float rs_above = 0.f;
    if (shift && t > 0) rs_above = gain / sqrtf(cta_sum(ss_above, s_tmp) / (float)W + a.eps);
    T* h = static_cast<T*>(a.h);
    T* mixed = static_cast<T*>(a.mixed);
    for (int i = threadIdx.x; i < W; i += kRowThreads) {
        const float ci = a.gain_per_col ? __ldg(a.gain + i) : 1.f;
        const float hv = value(t, i) * rs * ci;
        if (h != nullptr) h[(size_t)t * W + i] = from_f32<T>(hv);
        if (shift) {
            const float d = (t > 0 ? value(t - 1, i) * rs_above * ci : a.prev_in[i]) - hv;
            for (int m = 0; m < a.n_mix; ++m)
                mixed[((size_t)m * a.rows + t) * W + i] = from_f32<T>(fmaf(d, __ldg(a.mu[m] + i), hv));
        }
        if (a.prev_out != nullptr && t == a.rows - 1) a.prev_out[i] = hv;
    }
}

template <typename T>
__device__ __forceinline__ void store4(T* p, const float (&v)[4]) { leankv::store4(p, make_float4(v[0], v[1], v[2], v[3])); }
__device__ __forceinline__ void fetch4(const float* p, float (&v)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void fetch4(const bf16* p, float (&v)[4]) {
    const uint2 a = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(a.x << 16); v[1] = __uint_as_float(a.x & 0xffff0000u);
    v[2] = __uint_as_float(a.y << 16); v[3] = __uint_as_float(a.y & 0xffff0000u);
}

// The same with 4-element accesses and rows in registers (width % 4 == 0, width <= kRowThreads * 4 * NV). A CTA
// walks `per_cta` consecutive rows and keeps the row above, so only its first row is normed twice. With a normed branch (kPost) a
// row's stream and branch are asked for together, and a sum costs one barrier: 2048 x 2048 13.2 us when the branch was read twice, now 12.0
// (59 MB). A branch that joins as it is needs no sum of its own, so piece by piece takes fewer registers: with five shifted mixes
// 1024 / 2048 / 4096 columns 9.6 / 24.8 / 47.5 us, in one trip 13.3 / 23.0 / 65.2; hence one trip at two pieces.
template <typename T, typename D, int NV, bool kPost>
__global__ void __launch_bounds__(kRowThreads) stream_norm_vec_kernel(const leankv_stream_norm_t a, int per_cta) {
    __shared__ float s_tmp[2][32];
    pdl_begin();
    const int W = a.width, r0 = blockIdx.x * per_cta, r1 = min(a.rows, r0 + per_cta), tid = threadIdx.x;
    const D* delta = static_cast<const D*>(a.delta);
    T* h = static_cast<T*>(a.h);
    T* mixed = static_cast<T*>(a.mixed);
    const bool shift = a.n_mix > 0, per_col = a.gain_per_col != 0;
    const float gain = a.gain == nullptr || per_col ? 1.f : __ldg(a.gain);
    const float* scale = kPost ? a.post_gain : a.scale;
    float cur[NV][4], above[NV][4];
    int turn = 0;                 // sums take two buffers in turn, so that one barrier each is enough
    auto sum = [&](float v) { return cta_sum_once(v, s_tmp[turn ^= 1]); };
    auto load = [&](int row, bool store) -> float {       // the updated stream of `row` into cur; its norm factor
        constexpr bool kTrip = kPost || NV == 2;          // everything of the row in one trip
        float dv[kTrip ? NV : 1][4], ss = 0.f, f = 1.f;
        if constexpr (kTrip) {
#pragma unroll
            for (int n = 0; n < NV; ++n) {
                const int i = (tid + n * kRowThreads) * 4;
                if (i >= W) continue;
                fetch4(a.x_in + (size_t)row * W + i, cur[n]);
                if (kPost || delta != nullptr) fetch4(delta + (size_t)row * W + i, dv[n]);
            }
        }
        if constexpr (kPost) {                            // the branch is normed before it joins
#pragma unroll
            for (int n = 0; n < NV; ++n)
                if ((tid + n * kRowThreads) * 4 < W)
#pragma unroll
                    for (int q = 0; q < 4; ++q) ss = fmaf(dv[n][q], dv[n][q], ss);
            f = a.post_mult / sqrtf(sum(ss) / (float)W + a.eps);
            ss = 0.f;
        }
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const int i = (tid + n * kRowThreads) * 4;
            if (i < W) {
                if constexpr (!kTrip) fetch4(a.x_in + (size_t)row * W + i, cur[n]);
                if (kPost || delta != nullptr) {
                    float sv[4];
                    if constexpr (!kTrip) fetch4(delta + (size_t)row * W + i, dv[0]);
                    fetch4(scale + i, sv);
#pragma unroll
                    for (int q = 0; q < 4; ++q) cur[n][q] = fmaf(dv[kTrip ? n : 0][q] * f, sv[q], cur[n][q]);
                    if (store) store4(a.x_out + (size_t)row * W + i, cur[n]);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) ss = fmaf(cur[n][q], cur[n][q], ss);
            }
        }
        return a.gain == nullptr ? 1.f : gain / sqrtf(sum(ss) / (float)W + a.eps);
    };
    auto norm = [&](int n, float rs) {
        const int i = (tid + n * kRowThreads) * 4;
        float g[4] = {1.f, 1.f, 1.f, 1.f};
        if (per_col && i < W) fetch4(a.gain + i, g);
#pragma unroll
        for (int q = 0; q < 4; ++q) cur[n][q] *= rs * g[q];
    };
    if (shift) {
        if (r0 > 0) {
            const float rs = load(r0 - 1, false);
#pragma unroll
            for (int n = 0; n < NV; ++n) {
                norm(n, rs);
#pragma unroll
                for (int q = 0; q < 4; ++q) above[n][q] = cur[n][q];
            }
        } else {
#pragma unroll
            for (int n = 0; n < NV; ++n) {
                const int i = (tid + n * kRowThreads) * 4;
                if (i < W) fetch4(a.prev_in + i, above[n]);
            }
        }
    }
    for (int row = r0; row < r1; ++row) {
        const float rs = load(row, true);
        if (a.gain == nullptr) continue;
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const int i = (tid + n * kRowThreads) * 4;
            if (i >= W) continue;
            norm(n, rs);
            if (h != nullptr) store4(h + (size_t)row * W + i, cur[n]);
            if (shift) {
                for (int m = 0; m < a.n_mix; ++m) {
                    float mv[4];
                    fetch4(a.mu[m] + i, mv);
#pragma unroll
                    for (int q = 0; q < 4; ++q) mv[q] = fmaf(above[n][q] - cur[n][q], mv[q], cur[n][q]);
                    store4(mixed + ((size_t)m * a.rows + row) * W + i, mv);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) above[n][q] = cur[n][q];
                if (row == a.rows - 1) store4(a.prev_out + i, cur[n]);
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) silu_mul_rows_kernel(const T* gate_up, T* out, int inter, long long total) {
    pdl_begin();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / inter, c = i - r * inter;
        const float g = to_f32(gate_up[r * 2 * inter + c]), u = to_f32(gate_up[r * 2 * inter + inter + c]);
        out[i] = from_f32<T>(g * sigmoid_f32(g) * u);
    }
}

// Eight elements per thread (inter % 8 == 0, aligned), a block for every 2048 columns of a row: with as many blocks as fit twice the
// last round was nearly empty (2048 x 7168 in bf16: 17.9 us, so 15.9). Blocks of short rows would be mostly idle: kShort walks over all pieces
// (us by rows / so, bf16: 4096 x 256 4.6 / 3.0, 65536 x 64 68 / 5.8, 65536 x 768 69 / 62, but 4096 x 1792 8.2 / 8.9 and 512 x 256 1.7 / 1.8;
// fp32: 4096 x 512 4.8 / 3.9, 65536 x 768 87 / 91).
template <typename T>
bool short_rows(int rows, int inter) { return rows > 1024 && inter < (sizeof(T) == 2 ? 1024 : 768); }
template <typename T, bool kShort>
__global__ void __launch_bounds__(256) silu_mul_vec_kernel(const T* gate_up, T* out, int inter, int rows) {
    pdl_begin();
    const auto piece = [&](long long r, int c) {
        Raw8<T> rg, ru;
        load8(gate_up + r * 2 * inter + c, rg);
        load8(gate_up + r * 2 * inter + inter + c, ru);
        float g[8], u[8];
        unpack8(rg, g);
        unpack8(ru, u);
        T o[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) o[q] = from_f32<T>(g[q] * sigmoid_f32(g[q]) * u[q]);
        memcpy(&rg, o, sizeof(rg));
        *reinterpret_cast<Raw8<T>*>(out + r * inter + c) = rg;
    };
    if constexpr (kShort) {
        const int n8 = inter >> 3;
        const long long total = (long long)rows * n8;
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
            piece(i / n8, (int)(i % n8) * 8);
    } else {
        const int c = (blockIdx.x * 256 + threadIdx.x) * 8;
        if (c >= inter) return;
        for (long long r = blockIdx.y; r < rows; r += gridDim.y) piece(r, c);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) tanh_split_kernel(const float* in, T* out, int n, long long total) {
    pdl_begin();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const float v = tanhf(in[i]);
        if constexpr (sizeof(T) == 4) {
            out[i] = v;
        } else {
            const long long r = i / n, c = i - r * n;
            const T hi = from_f32<T>(v);
            out[r * 2 * n + c] = hi;
            out[r * 2 * n + n + c] = from_f32<T>(v - to_f32(hi));
        }
    }
}

// The rows of a portion's tokens out of the embedding table, as the fp32 stream: one CTA a row, eight columns a thread. Bound by
// memory: 2048 rows x 2048 in bf16, gather and conversion 14.2 us as two tensor operations, 6.4 us here.
template <typename T, bool kVec>
__global__ void __launch_bounds__(kRowThreads) embed_rows_kernel(const T* table, const long long* ids, float* x, int width, int vocab) {
    pdl_begin();
    long long tok = __ldg(ids + blockIdx.x);
    if (tok < 0 || tok >= vocab) tok = 0;
    const T* src = table + (size_t)tok * width;
    float* dst = x + (size_t)blockIdx.x * width;
    if constexpr (kVec) {
        for (int i = threadIdx.x * 8; i < width; i += kRowThreads * 8) {
            Raw8<T> r;
            float v[8];
            load8(src + i, r);
            unpack8(r, v);
            *reinterpret_cast<float4*>(dst + i) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(dst + i + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
    } else {
        for (int i = threadIdx.x; i < width; i += kRowThreads) dst[i] = to_f32(src[i]);
    }
}

__global__ void __launch_bounds__(256) softcap_kernel(float* x, long long n, float cap) {
    pdl_begin();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        x[i] = cap * tanhf(x[i] / cap);
}

template <typename T, typename D>
int launch_stream_norm(const leankv_stream_norm_t* a, cudaStream_t st) {
    bool vec = a->width % 4 == 0 && a->width <= kRowThreads * 4 * 8 && aligned16(a->x_in) && aligned16(a->x_out) &&
               aligned16(a->delta) && aligned16(a->scale) && aligned16(a->h) && aligned16(a->mixed) &&
               aligned16(a->prev_in) && aligned16(a->prev_out) && aligned16(a->post_gain) &&
               (!a->gain_per_col || aligned16(a->gain));
    for (int i = 0; i < a->n_mix; ++i) vec = vec && aligned16(a->mu[i]);
    if (!vec) {
        LEANKV_CUDA_TRY(launch_early(stream_norm_kernel<T, D>, dim3(a->rows), dim3(kRowThreads), 0, st, *a));
        return LEANKV_OK;
    }
    // Rows of a CTA with a shift: more than one spares norming the row above, but leaves fewer CTAs. us, five mixes in bf16: 1200 x 1536 with
    // four rows a CTA 10.3, with two 8.2, 2048 x 2048 16.3 and 14.2, 4000 x 2048 with a branch 41.4 and 35.8; one piece a thread, 600 x 1024 with
    // one row 5.9, with two 4.9, 900 x 1024 6.0 and 5.4 (but 600 x 2048 6.1 and 7.1, and in fp32 900 x 1024 7.7 and 7.9).
    const int nv = (a->width + kRowThreads * 4 - 1) / (kRowThreads * 4);
    const bool pairs = sizeof(T) == 2 && nv == 1 && a->rows >= sm_count() * 4;
    const int per = a->n_mix == 0 ? 1 : a->rows >= sm_count() * 8 ? (nv == 2 ? 2 : 4) : pairs ? 2 : 1;
    const dim3 grid((a->rows + per - 1) / per), block(kRowThreads);
    const bool post = a->post_gain != nullptr;
    const auto go = [&](auto pieces) -> int {
        constexpr int NV = decltype(pieces)::value;
        LEANKV_CUDA_TRY(launch_early(post ? stream_norm_vec_kernel<T, D, NV, true> : stream_norm_vec_kernel<T, D, NV, false>, grid, block, 0,
                                     st, *a, per));
        return LEANKV_OK;
    };
    return nv <= 1   ? go(std::integral_constant<int, 1>{})
           : nv <= 2 ? go(std::integral_constant<int, 2>{})
           : nv <= 4 ? go(std::integral_constant<int, 4>{})
                     : go(std::integral_constant<int, 8>{});
}

bool known(int dtype) { return dtype == LEANKV_DT_BF16 || dtype == LEANKV_DT_F32; }

}  // namespace
}  // namespace leankv

using namespace leankv;

extern "C" int leankv_embed_begin(const void* table, int dtype, const long long* token, float* x, int width,
                                  int vocab, int32_t* state, void* stream) {
    if (!table || !token || !x || !state || width <= 0 || vocab <= 0) return LEANKV_EINVAL;
    if (!known(dtype)) return LEANKV_EUNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == LEANKV_DT_BF16)
        LEANKV_CUDA_TRY(launch_early(decode_begin_kernel<bf16, float>, dim3(1), dim3(256), 0, st,
                                      static_cast<const bf16*>(table), token, x, width, vocab, state));
    else
        LEANKV_CUDA_TRY(launch_early(decode_begin_kernel<float, float>, dim3(1), dim3(256), 0, st,
                                      static_cast<const float*>(table), token, x, width, vocab, state));
    return LEANKV_OK;
}

extern "C" int leankv_embed_rows(const void* table, int dtype, const long long* ids, int rows, int width, int vocab, float* x,
                                 void* stream) {
    if (!table || !ids || !x || rows <= 0 || width <= 0 || vocab <= 0) return LEANKV_EINVAL;
    if (!known(dtype)) return LEANKV_EUNSUPPORTED;
    const bool vec = width % 8 == 0 && aligned16(table) && aligned16(x);
    const auto go = [&](auto tag) -> int {
        using T = decltype(tag);
        LEANKV_CUDA_TRY(launch_early(vec ? embed_rows_kernel<T, true> : embed_rows_kernel<T, false>, dim3(rows), dim3(kRowThreads), 0,
                                     static_cast<cudaStream_t>(stream), static_cast<const T*>(table), ids, x, width, vocab));
        return LEANKV_OK;
    };
    return dtype == LEANKV_DT_BF16 ? go(bf16{}) : go(float{});
}

extern "C" int leankv_greedy_end(const float* logits, int vocab, long long* token, long long* history,
                                 int history_cap, int32_t* state, void* stream) {
    if (!logits || !token || !history || !state || vocab <= 0 || history_cap < 0) return LEANKV_EINVAL;
    if (!aligned16(logits)) return LEANKV_EALIGN;
    LEANKV_CUDA_TRY(launch_early(decode_end_kernel<float, 8>, dim3(8), dim3(end_threads(8)), 0, static_cast<cudaStream_t>(stream),
                                  logits, vocab, token, history, history_cap, state + kPos, state + kStep,
                                  state + kParity));
    return LEANKV_OK;
}

extern "C" int leankv_stream_norm(const leankv_stream_norm_t* a, void* stream) {
    if (!a || !a->x_in || a->rows <= 0 || a->width <= 0 || a->n_mix < 0 || a->n_mix > LEANKV_MAX_MIX) return LEANKV_EINVAL;
    if (!a->gain && (a->h || a->n_mix > 0 || !a->delta)) return LEANKV_EINVAL;
    if (a->delta && (!a->x_out || (!a->scale && !a->post_gain) || a->x_out == a->x_in)) return LEANKV_EINVAL;
    if (a->post_gain && !a->delta) return LEANKV_EINVAL;
    if (a->n_mix > 0) {
        if (!a->mixed || !a->prev_in || !a->prev_out || a->prev_in == a->prev_out) return LEANKV_EINVAL;
        for (int i = 0; i < a->n_mix; ++i)
            if (!a->mu[i]) return LEANKV_EINVAL;
    }
    if (!known(a->dtype) || (a->delta && !known(a->delta_dtype))) return LEANKV_EUNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool d16 = a->delta && a->delta_dtype == LEANKV_DT_BF16;
    if (a->dtype == LEANKV_DT_BF16)
        return d16 ? launch_stream_norm<bf16, bf16>(a, st) : launch_stream_norm<bf16, float>(a, st);
    return d16 ? launch_stream_norm<float, bf16>(a, st) : launch_stream_norm<float, float>(a, st);
}

extern "C" int leankv_silu_mul(const void* gate_up, void* out, int dtype, int rows, int inter, void* stream) {
    if (!gate_up || !out || rows <= 0 || inter <= 0) return LEANKV_EINVAL;
    if (!known(dtype)) return LEANKV_EUNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool vec = inter % 8 == 0 && aligned16(gate_up) && aligned16(out);
    const long long total = (long long)rows * inter;
    const int grid = (int)std::min<long long>(((vec ? total / 8 : total) + 255) / 256, (long long)sm_count() * 16);
    auto go = [&](auto tag) -> int {
        using T = decltype(tag);
        if (vec && short_rows<T>(rows, inter))
            LEANKV_CUDA_TRY(launch_early(silu_mul_vec_kernel<T, true>, dim3(grid), dim3(256), 0, st, static_cast<const T*>(gate_up),
                                         static_cast<T*>(out), inter, rows));
        else if (vec)
            LEANKV_CUDA_TRY(launch_early(silu_mul_vec_kernel<T, false>, dim3((inter / 8 + 255) / 256, std::min(rows, 65535)), dim3(256), 0, st,
                                         static_cast<const T*>(gate_up), static_cast<T*>(out), inter, rows));
        else
            LEANKV_CUDA_TRY(launch_early(silu_mul_rows_kernel<T>, dim3(grid), dim3(256), 0, st, static_cast<const T*>(gate_up),
                                         static_cast<T*>(out), inter, total));
        return LEANKV_OK;
    };
    return dtype == LEANKV_DT_BF16 ? go(bf16{}) : go(float{});
}

extern "C" int leankv_tanh_split(const float* in, void* out, int dtype, int rows, int n, void* stream) {
    if (!in || !out || rows <= 0 || n <= 0) return LEANKV_EINVAL;
    if (!known(dtype)) return LEANKV_EUNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long total = (long long)rows * n;
    const int grid = (int)std::min<long long>((total + 255) / 256, (long long)sm_count() * 8);
    auto go = [&](auto tag) -> int {
        using T = decltype(tag);
        LEANKV_CUDA_TRY(launch_early(tanh_split_kernel<T>, dim3(grid), dim3(256), 0, st, in, static_cast<T*>(out), n,
                                      total));
        return LEANKV_OK;
    };
    return dtype == LEANKV_DT_BF16 ? go(bf16{}) : go(float{});
}

extern "C" int leankv_softcap(float* x, long long n, float cap, void* stream) {
    if (!x || n <= 0 || !(cap > 0.f)) return LEANKV_EINVAL;
    const int grid = (int)std::min<long long>((n + 255) / 256, (long long)sm_count() * 8);
    LEANKV_CUDA_TRY(launch_early(softcap_kernel, dim3(grid), dim3(256), 0, static_cast<cudaStream_t>(stream), x, n, cap));
    return LEANKV_OK;
}
