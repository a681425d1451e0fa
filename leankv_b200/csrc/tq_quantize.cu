// TurboQuant (MSE variant) quantize / dequantize and the paged-pool append for B200.
//
// Arithmetic contract shared by every kernel in this file (and restated on the CPU by
// the test oracle), chosen so that a vector's codes never depend on how vectors are
// batched, tiled or appended:
//   norm   = float( sqrt( S_lo + S_hi ) ),  S_lo / S_hi = fp64 sums of squares of
//            coordinates 0..63 / 64..127 taken in ascending order
//   u[k]   = x[k] / (norm + 1e-10f)                       (fp32, IEEE division)
//   y[j]   = fma(Pi[j][127], u[127], ... fma(Pi[j][0], u[0], 0))   (fp32, ascending k)
//   code_j = #{ i : boundary[i] < y[j] }
// This is leankv/turboquant/quantizer.py:119-129; the reference leaves the summation
// order to its BLAS, so a code can differ from it only where y lies within rounding
// distance of a decision boundary.

#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "tq_layout.cuh"
#include "umma.cuh"

namespace leankv {
namespace {

constexpr int kDim = LEANKV_TQ_DIM;

// Sum of squares of 64 values in fp64, ascending order.
__device__ __forceinline__ double sumsq64(const float (&x)[64]) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 64; ++i) s = fma((double)x[i], (double)x[i], s);
    return s;
}

// ---------------------------------------------------------------------------
// Pool append: one CTA quantizes the new tokens that fall into one page of one
// (sequence, head, K|V) and writes them in the chunk layout of tq_layout.cuh.
// ---------------------------------------------------------------------------
struct AppendParams {
    const __half* k;
    const __half* v;
    int B, H, T_new;
    long long k_seq, k_head, v_seq, v_head;      // elements from a sequence / a head to the next; tokens are 128 apart
    const float* Pi_k;
    const float* Pi_v;
    const float* bounds;
    uint8_t* pool;
    int n_pages;
    const int32_t* kv_indptr;
    const int32_t* kv_page_indices;
    const int32_t* start_pos;
};
__device__ __forceinline__ const __half* append_source(const AppendParams& p, int which, int b, int h) {
    return which == 0 ? p.k + b * p.k_seq + h * p.k_head : p.v + b * p.v_seq + h * p.v_head;
}

template <int kTok>   // register accumulators per thread: 1 (single-token decode) or 16
__global__ void __launch_bounds__(128) tq_pool_append_kernel(const AppendParams p) {
    __shared__ __align__(16) float s_u[kDim][kTok];      // [k][token slot in this CTA]
    __shared__ uint8_t s_code[kTok][kDim];
    __shared__ float s_norm[kTok];
    __shared__ float s_bounds[8];

    pdl_begin();
    const int tid = threadIdx.x;
    const int b = blockIdx.x / p.H, h = blockIdx.x % p.H;
    const int which = blockIdx.z;                         // 0 = K, 1 = V
    const int pos0 = p.start_pos[b];
    const int page_ord = pos0 / 16 + blockIdx.y;          // page ordinal inside the sequence
    const int first = max(pos0, page_ord * 16);           // first / last+1 absolute positions handled here
    const int last = min(pos0 + p.T_new, page_ord * 16 + 16);
    const int nt = last - first;
    if (nt <= 0) return;
    const int slot0 = first - page_ord * 16;
    const int page = p.kv_page_indices[p.kv_indptr[b] + page_ord];
    if (page < 0 || page >= p.n_pages) return;            // invalid table entry: write nothing

    if (tid < 8) s_bounds[tid] = tid < 7 ? p.bounds[tid] : __int_as_float(0x7f800000);

    const __half* src = append_source(p, which, b, h) + (size_t)(first - pos0) * kDim;
    const float* Pi = which == 0 ? p.Pi_k : p.Pi_v;

    // norms and unit vectors: two threads per token, 64 coordinates each
    if (tid < 2 * kTok) {
        const int t = tid >> 1, hf = tid & 1;
        float xr[64];
        if (t < nt) {
            const uint4* s4 = reinterpret_cast<const uint4*>(src + (size_t)t * kDim + hf * 64);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint4 w = __ldg(s4 + i);
                const float2 a = h2_to_f2(w.x), bb = h2_to_f2(w.y), c = h2_to_f2(w.z), d = h2_to_f2(w.w);
                xr[8 * i + 0] = a.x; xr[8 * i + 1] = a.y; xr[8 * i + 2] = bb.x; xr[8 * i + 3] = bb.y;
                xr[8 * i + 4] = c.x; xr[8 * i + 5] = c.y; xr[8 * i + 6] = d.x; xr[8 * i + 7] = d.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 64; ++i) xr[i] = 0.f;
        }
        const double mine = sumsq64(xr);
        // only the 2 * kTok lanes inside this branch take part in the exchange
        constexpr unsigned kPairMask = kTok >= 16 ? 0xffffffffu : ((1u << (2 * kTok)) - 1u);
        const double other = __shfl_xor_sync(kPairMask, mine, 1);
        const double tot = hf == 0 ? mine + other : other + mine;
        const float norm = (float)sqrt(tot);
        const float denom = norm + 1e-10f;
        if (hf == 0) s_norm[t] = norm;
#pragma unroll
        for (int i = 0; i < 64; ++i) s_u[hf * 64 + i][t] = xr[i] / denom;
    }
    __syncthreads();

    // rotation: thread j owns output coordinate j for every token of the CTA
    {
        const int j = tid;
        float acc[kTok];
#pragma unroll
        for (int t = 0; t < kTok; ++t) acc[t] = 0.f;
        const float4* row = reinterpret_cast<const float4*>(Pi + (size_t)j * kDim);
#pragma unroll 2
        for (int k4 = 0; k4 < kDim / 4; ++k4) {
            const float4 pv = __ldg(row + k4);
            const float pk[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = 4 * k4 + q;
#pragma unroll
                for (int t = 0; t < kTok; ++t) acc[t] = fmaf(pk[q], s_u[k][t], acc[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < kTok; ++t) {
            int c = 0;
#pragma unroll
            for (int q = 0; q < 7; ++q) c += (acc[t] > s_bounds[q]) ? 1 : 0;
            s_code[t][j] = (uint8_t)c;
        }
    }
    __syncthreads();

    uint8_t* chunk = p.pool + (((size_t)page * 2 + which) * p.H + h) * kChunkBytes;
    uint32_t* words = reinterpret_cast<uint32_t*>(chunk);
    __half* norms = reinterpret_cast<__half*>(chunk + kNormOffsetBytes);

    if (tid < nt) norms[slot0 + tid] = __float2half_rn(s_norm[tid]);

    for (int w = tid; w < kChunkWords; w += 128) {
        const int kk = w >> 6, ui = w & 63;
        if (which == 0) {
            const int slot = ui >> 2, t4 = ui & 3;
            const int t = slot - slot0;
            if (t < 0 || t >= nt) continue;
            uint32_t bits = 0;
#pragma unroll 8
            for (int e = 0; e < 32; ++e) bits |= unit_word_bits(e, kk, s_code[t][32 * t4 + e]);
            words[w] = bits;
        } else {
            const int pr = ui < 32 ? (ui & 3) : 4 + (ui & 3);
            const int g = (ui & 31) >> 2;
            const int ta = 2 * pr - slot0, tb = ta + 1;           // CTA-local token indices of the pair
            const bool has_a = ta >= 0 && ta < nt, has_b = tb >= 0 && tb < nt;
            if (!has_a && !has_b) continue;
            uint32_t bits = 0;
#pragma unroll 8
            for (int c = 0; c < 16; ++c) {
                if (has_a) bits |= unit_word_bits(2 * c, kk, s_code[ta][16 * g + c]);
                if (has_b) bits |= unit_word_bits(2 * c + 1, kk, s_code[tb][16 * g + c]);
            }
            if (!(has_a && has_b)) {
                // the other token of the pair was (or will be) written by another launch
                const uint32_t keep = has_a ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
                bits |= words[w] & keep;
            }
            words[w] = bits;
        }
    }
}

#include "tq_append_tc.cuh"
#include "tq_append_t5.cuh"
#include "tq_rows.cuh"

// Coordinates decided by the exact chain / coordinates quantized by the tensor-core append, per device,
// since the last reset (read by leankv_tq_band_stats).
__device__ unsigned long long g_band_stats[2];
// Non-zero once a bounded wait inside the quantize kernel or the tcgen05 append has run out (per device, sticky; read by
// leankv_tq_append_status).
__device__ int g_append_status;

struct UnpackParams {
    const uint8_t* pool;
    int n_pages, H;
    const int32_t* page_indices;
    int n_tokens, which;
    uint8_t* indices;
    float* norms;
};

__global__ void tq_pool_unpack_kernel(const UnpackParams p) {
    const long long total = (long long)p.H * p.n_tokens * 64;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int byte = (int)(i & 63);
        const long long ht = i >> 6;
        const int tok = (int)(ht % p.n_tokens), h = (int)(ht / p.n_tokens);
        const int page = p.page_indices[tok >> 4], slot = tok & 15;
        if (page < 0 || page >= p.n_pages) {
            // a stale or foreign page id: nothing is read from the pool; the token reads as code 0, norm 0
            p.indices[i] = 0;
            if (byte == 0) p.norms[ht] = 0.f;
            continue;
        }
        const uint8_t* chunk = p.pool + (((size_t)page * 2 + p.which) * p.H + h) * kChunkBytes;
        const uint32_t* words = reinterpret_cast<const uint32_t*>(chunk);
        const int c0 = 2 * byte, c1 = c0 + 1;
        const int lo = chunk_get_code(words, p.which == 0 ? k_code_slot(slot, c0) : v_code_slot(slot, c0));
        const int hi = chunk_get_code(words, p.which == 0 ? k_code_slot(slot, c1) : v_code_slot(slot, c1));
        p.indices[i] = (uint8_t)(lo | (hi << 4));
        if (byte == 0)
            p.norms[ht] = __half2float(reinterpret_cast<const __half*>(chunk + kNormOffsetBytes)[slot]);
    }
}

// LEANKV_TQ_APPEND selects the kernel of multi-token appends: "fp32" = the fp32 kernel (the definition the
// tensor-core paths are tested against), default / "mma" = fast rotation on mma.sync (64-token tiles, two CTAs
// per SM), "t5" = fast rotation on tcgen05 (128-token tiles, one CTA per SM: measured slower, 1.49 ms
// for a million vectors against 0.64 ms, because its norm / code / pack phases have no second CTA to overlap with).
// All three write the same bits.
int tc_append_mode() {
    static int state = -1;
    if (state < 0) {
        const char* e = std::getenv("LEANKV_TQ_APPEND");
        state = e == nullptr ? 1 : (e[0] == 'f' ? 0 : (e[0] == 't' && e[1] == '5' ? 2 : 1));
    }
    return state;
}
bool tc_append_enabled() { return tc_append_mode() != 0; }

int check_tq_common(long long n_vec, int dim, int bits) {
    if (n_vec < 0) return LEANKV_EINVAL;
    if (dim != kDim) return LEANKV_EUNSUPPORTED;
    if (bits < 1 || bits > 4) return LEANKV_EUNSUPPORTED;
    return LEANKV_OK;
}

// What a device is asked once: the kernel's opt-in to large shared memory, the status word's address. Racing first
// calls store the same values.
template <auto kKernel, typename... More>
int launch_rows(RowsParams p, int per_cta, int threads, size_t smem, void* stream, More... more) {      // per_cta: vectors at least
    constexpr int kMaxDevices = 64;
    static int* status[kMaxDevices] = {};
    int dev = 0;
    LEANKV_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return LEANKV_ELIMIT;
    if (status[dev] == nullptr) {
        void* word = nullptr;
        LEANKV_CUDA_TRY(cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        LEANKV_CUDA_TRY(cudaGetSymbolAddress(&word, g_append_status));
        status[dev] = static_cast<int*>(word);
    }
    p.wide = aligned16(p.indices) ? 1 : 0;
    p.status = status[dev];
    const long long want = (p.n_vec + per_cta - 1) / per_cta;
    const int grid = (int)(want < sm_count() ? want : sm_count());
    kKernel<<<grid, threads, smem, static_cast<cudaStream_t>(stream)>>>(p, more...);
    LEANKV_CUDA_TRY(cudaGetLastError());
    return LEANKV_OK;
}
template <typename Raw>
int launch_quantize(const RowsParams& p, int bits, void* stream) {
    switch (bits) {
        case 1: return launch_rows<tq_quantize_rows_kernel<1, Raw>>(p, kRowsTile, kRowsThreads, kRowsSmemBytes, stream);
        case 2: return launch_rows<tq_quantize_rows_kernel<2, Raw>>(p, kRowsTile, kRowsThreads, kRowsSmemBytes, stream);
        case 3: return launch_rows<tq_quantize_rows_kernel<3, Raw>>(p, kRowsTile, kRowsThreads, kRowsSmemBytes, stream);
        default: return launch_rows<tq_quantize_rows_kernel<4, Raw>>(p, kRowsTile, kRowsThreads, kRowsSmemBytes, stream);
    }
}

}  // namespace
}  // namespace leankv

using namespace leankv;

extern "C" int leankv_tq_packed_len(int dim, int bits) {
    if (dim <= 0 || bits < 1) return LEANKV_EINVAL;
    const int vpb = bits == 1 ? 8 : bits == 2 ? 4 : bits <= 4 ? 2 : 1;
    return (dim + vpb - 1) / vpb;
}

extern "C" int leankv_tq_quantize(const void* x, int x_dtype, long long n_vec, int dim, int bits,
                                  const float* Pi, const float* decision_boundaries,
                                  uint8_t* indices, float* norms, void* stream) {
    int rc = check_tq_common(n_vec, dim, bits);
    if (rc != LEANKV_OK) return rc;
    if (n_vec == 0) return LEANKV_OK;
    if (!x || !Pi || !decision_boundaries || !indices || !norms) return LEANKV_EINVAL;
    if (x_dtype != 0 && x_dtype != 1) return LEANKV_EINVAL;
    if (!aligned16(x) || !aligned16(Pi)) return LEANKV_EALIGN;
    RowsParams p{};
    p.x = x;
    p.n_vec = n_vec;
    p.Pi = Pi;
    p.table = decision_boundaries;
    p.indices = indices;
    p.norms = norms;
    return x_dtype == 0 ? launch_quantize<__half>(p, bits, stream) : launch_quantize<float>(p, bits, stream);
}

extern "C" int leankv_tq_dequantize(const uint8_t* indices, const float* norms, long long n_vec,
                                    int dim, int bits, const float* Pi, const float* centroids,
                                    void* x_hat, int out_dtype, void* stream) {
    int rc = check_tq_common(n_vec, dim, bits);
    if (rc != LEANKV_OK) return rc;
    if (n_vec == 0) return LEANKV_OK;
    if (!indices || !norms || !Pi || !centroids || !x_hat) return LEANKV_EINVAL;
    if (out_dtype != 0 && out_dtype != 1) return LEANKV_EINVAL;
    if (!aligned16(x_hat) || !aligned16(Pi)) return LEANKV_EALIGN;
    RowsParams p{};
    p.n_vec = n_vec;
    p.Pi = Pi;
    p.table = centroids;
    p.indices = const_cast<uint8_t*>(indices);
    p.norms = const_cast<float*>(norms);
    p.out = x_hat;
    p.out_dtype = out_dtype;
    return launch_rows<tq_dequantize_rows_kernel>(p, 16, kDequantThreads, kDequantSmemBytes, stream, bits);
}

extern "C" size_t leankv_tq_pool_bytes(int n_pages, int n_kv_heads) {
    if (n_pages <= 0 || n_kv_heads <= 0) return 0;
    return (size_t)n_pages * 2 * n_kv_heads * kChunkBytes;
}

extern "C" int leankv_tq_pool_append_strided(const void* k, const void* v, int B, int n_kv_heads, int T_new, long long k_seq,
                                             long long k_head, long long v_seq, long long v_head,
                                     const float* Pi_k, const float* Pi_v,
                                     const float* decision_boundaries, void* pool, int n_pages,
                                     const int32_t* kv_indptr, const int32_t* kv_page_indices,
                                     const int32_t* start_pos, void* stream) {
    if (B < 0 || n_kv_heads <= 0 || T_new < 0 || n_pages <= 0) return LEANKV_EINVAL;
    if (B == 0 || T_new == 0) return LEANKV_OK;
    if (!k || !v || !Pi_k || !Pi_v || !decision_boundaries || !pool || !kv_indptr ||
        !kv_page_indices || !start_pos)
        return LEANKV_EINVAL;
    if (!aligned16(k) || !aligned16(v) || !aligned16(Pi_k) || !aligned16(Pi_v) || !aligned16(pool))
        return LEANKV_EALIGN;
    if (k_seq % 8 != 0 || k_head % 8 != 0 || v_seq % 8 != 0 || v_head % 8 != 0) return LEANKV_EALIGN;
    if ((long long)B * n_kv_heads > 0x7fffffffLL) return LEANKV_ELIMIT;
    AppendParams p{};
    p.k_seq = k_seq; p.k_head = k_head; p.v_seq = v_seq; p.v_head = v_head;
    p.k = static_cast<const __half*>(k);
    p.v = static_cast<const __half*>(v);
    p.B = B;
    p.H = n_kv_heads;
    p.T_new = T_new;
    p.Pi_k = Pi_k;
    p.Pi_v = Pi_v;
    p.bounds = decision_boundaries;
    p.pool = static_cast<uint8_t*>(pool);
    p.n_pages = n_pages;
    p.kv_indptr = kv_indptr;
    p.kv_page_indices = kv_page_indices;
    p.start_pos = start_pos;
    // T_new tokens starting anywhere inside a page touch at most (T_new + 14) / 16 + 1 pages.
    const int groups = (T_new + 14) / 16 + 1;
    if (T_new >= 16 && tc_append_enabled()) {
        // prompt-sized appends: rotation on tensor cores, codes identical to the fp32 kernels
        AppendTcParams tp{};
        tp.a = p;
        const bool t5 = tc_append_mode() == 2;
        const int pages_per_tile = t5 ? kT5Pages : 4;
        tp.groups = (groups + pages_per_tile - 1) / pages_per_tile;
        tp.n_tiles = 2LL * B * n_kv_heads * tp.groups;
        void* stats = nullptr;
        LEANKV_CUDA_TRY(cudaGetSymbolAddress(&stats, g_band_stats));
        tp.stats = static_cast<unsigned long long*>(stats);
        int dev = 0;
        LEANKV_CUDA_TRY(cudaGetDevice(&dev));
        constexpr int kMaxDevices = 64;
        static bool attr_done[kMaxDevices] = {};
        if (dev < 0 || dev >= kMaxDevices || !attr_done[dev]) {
            LEANKV_CUDA_TRY(cudaFuncSetAttribute(tq_pool_append_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)kTcSmemBytes));
            LEANKV_CUDA_TRY(cudaFuncSetAttribute(tq_pool_append_t5_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)kT5SmemBytes));
            if (dev >= 0 && dev < kMaxDevices) attr_done[dev] = true;
        }
        if (t5) {
            void* st_word = nullptr;
            LEANKV_CUDA_TRY(cudaGetSymbolAddress(&st_word, g_append_status));
            const long long slots1 = sm_count();            // 148 KB of shared memory: one CTA per SM
            const int grid_t5 = (int)(tp.n_tiles < slots1 ? tp.n_tiles : slots1);
            LEANKV_CUDA_TRY(launch_plain(tq_pool_append_t5_kernel, dim3(grid_t5), dim3(kT5Threads), kT5SmemBytes,
                                          static_cast<cudaStream_t>(stream), tp, static_cast<int*>(st_word)));
            return LEANKV_OK;
        }
        const long long slots = 2LL * sm_count();
        const int grid_tc = (int)(tp.n_tiles < slots ? tp.n_tiles : slots);
        LEANKV_CUDA_TRY(launch_early(tq_pool_append_tc_kernel, dim3(grid_tc), dim3(kTcThreads), kTcSmemBytes,
                                      static_cast<cudaStream_t>(stream), tp));
        return LEANKV_OK;
    }
    if (groups > 65535) return LEANKV_ELIMIT;
    dim3 grid(B * n_kv_heads, groups, 2);
    if (T_new == 1)
        LEANKV_CUDA_TRY(launch_early(tq_pool_append_kernel<1>, grid, dim3(128), 0, static_cast<cudaStream_t>(stream), p));
    else
        LEANKV_CUDA_TRY(launch_early(tq_pool_append_kernel<16>, grid, dim3(128), 0, static_cast<cudaStream_t>(stream), p));
    return LEANKV_OK;
}

extern "C" int leankv_tq_pool_append(const void* k, const void* v, int B, int n_kv_heads, int T_new,
                                     const float* Pi_k, const float* Pi_v,
                                     const float* decision_boundaries, void* pool, int n_pages,
                                     const int32_t* kv_indptr, const int32_t* kv_page_indices,
                                     const int32_t* start_pos, void* stream) {
    const long long head = (long long)T_new * kDim, seq = head * n_kv_heads;
    return leankv_tq_pool_append_strided(k, v, B, n_kv_heads, T_new, seq, head, seq, head, Pi_k, Pi_v, decision_boundaries, pool,
                                         n_pages, kv_indptr, kv_page_indices, start_pos, stream);
}

extern "C" int leankv_tq_pool_unpack(const void* pool, int n_pages, int n_kv_heads,
                                     const int32_t* page_indices, int n_tokens, int which,
                                     uint8_t* indices, float* norms, void* stream) {
    if (n_pages <= 0 || n_kv_heads <= 0 || n_tokens < 0 || (which != 0 && which != 1))
        return LEANKV_EINVAL;
    if (n_tokens == 0) return LEANKV_OK;
    if (!pool || !page_indices || !indices || !norms) return LEANKV_EINVAL;
    UnpackParams p{};
    p.pool = static_cast<const uint8_t*>(pool);
    p.n_pages = n_pages;
    p.H = n_kv_heads;
    p.page_indices = page_indices;
    p.n_tokens = n_tokens;
    p.which = which;
    p.indices = indices;
    p.norms = norms;
    const long long total = (long long)n_kv_heads * n_tokens * 64;
    long long blocks = (total + 255) / 256;
    if (blocks > sm_count() * 16LL) blocks = sm_count() * 16LL;
    tq_pool_unpack_kernel<<<(int)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
    LEANKV_CUDA_TRY(cudaGetLastError());
    return LEANKV_OK;
}

extern "C" int leankv_tq_append_status(int* status /* host */) {
    if (!status) return LEANKV_EINVAL;
    LEANKV_CUDA_TRY(cudaMemcpyFromSymbol(status, g_append_status, sizeof(int)));
    return LEANKV_OK;
}

extern "C" int leankv_tq_band_stats(unsigned long long* stats /* host, 2 */, int reset) {
    if (!stats) return LEANKV_EINVAL;
    LEANKV_CUDA_TRY(cudaMemcpyFromSymbol(stats, g_band_stats, sizeof(unsigned long long) * 2));
    if (reset) {
        const unsigned long long zero[2] = {0ull, 0ull};
        LEANKV_CUDA_TRY(cudaMemcpyToSymbol(g_band_stats, zero, sizeof(zero)));
    }
    return LEANKV_OK;
}
