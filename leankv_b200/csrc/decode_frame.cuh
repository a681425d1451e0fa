// First and last kernel of a decode step: embedding fetch and greedy next token. Templated on the storage
// type of the table / the logits, so that every decode loop of the library frames its step the same way.
#pragma once

#include "typed.cuh"

namespace leankv {

// Decode state words (int32[8], device), as the header describes them beside leankv_decode_begin: position,
// step count, the one-sequence page table (kv_indptr[0..1], kv_last_page_len, start position), and the half
// of a double-buffered per-sequence vector that the current step reads.
enum { kPos = 0, kStep = 1, kIndptr0 = 2, kIndptr1 = 3, kLastLen = 4, kStartPos = 5, kParity = 6 };

// Fetch the embedding row of the current token and derive this step's page-table words.
template <typename In, typename Out>
__global__ void __launch_bounds__(256) decode_begin_kernel(const In* table, const long long* token, Out* h,
                                                           int hidden, int vocab, int* state) {
    pdl_begin();
    long long tok = *token;
    if (tok < 0 || tok >= vocab) tok = 0;
    if constexpr (sizeof(In) == 2 && sizeof(Out) == 2) {      // same type, hidden % 8 == 0 (checked on the host)
        const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)tok * hidden);
        uint4* dst = reinterpret_cast<uint4*>(h);
        for (int i = threadIdx.x; i < hidden / 8; i += blockDim.x) dst[i] = __ldg(src + i);
    } else if (hidden % 8 == 0 && ((reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(h)) & 15) == 0) {
        const In* src = table + (size_t)tok * hidden;      // one trip to memory for rows of up to 2048 columns
        for (int i = threadIdx.x * 8; i < hidden; i += blockDim.x * 8) {
            Raw8<In> r;
            float v[8];
            load8(src + i, r);
            unpack8(r, v);
            *reinterpret_cast<float4*>(h + i) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(h + i + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
    } else {
        const In* src = table + (size_t)tok * hidden;
        for (int i = threadIdx.x; i < hidden; i += blockDim.x) h[i] = to_f32(src[i]);
    }
    if (threadIdx.x == 0) {
        const int pos = state[kPos];
        state[kStartPos] = pos;
        state[kIndptr0] = 0;
        state[kIndptr1] = pos / 16 + 1;
        state[kLastLen] = pos % 16 + 1;
    }
}

// Greedy next token (lowest index wins ties), appended to the history; advances the position.
// One cluster of kEndCtas CTAs per sequence (pos / step are that sequence's words), each with a share of the vocabulary; the shares'
// best meet in the first CTA's shared memory. One CTA alone read the row at the rate of one SM: 32768 fp32 logits 5.7 -> 2.8 us behind
// the output head. Where there are more sequences than the device holds clusters of eight at once, one larger CTA each: us by clusters / so,
// 32000 logits, 48 sequences 4.1 / 4.6, 64 4.3 / 4.6, 80 5.3 / 4.6, 256 10.9 / 6.0; 4096 logits, 48 3.7 / 3.8, 64 4.2 / 3.8. `parity`
// (optional) is flipped.
constexpr int end_ctas(int sequences, int vocab) { return sequences <= (vocab >= 16384 ? 64 : 48) ? 8 : 1; }
__host__ __device__ constexpr int end_threads(int ctas) { return ctas == 1 ? 1024 : 512; }

template <typename L, int kEndCtas>
__global__ void __cluster_dims__(kEndCtas, 1, 1) __launch_bounds__(end_threads(kEndCtas))
    decode_end_kernel(const L* logits, int vocab, long long* token, long long* history, int history_cap, int* pos, int* step_ptr,
                      int* parity) {
    constexpr int kEndThreads = end_threads(kEndCtas), kWarps = kEndThreads / 32;
    __shared__ float s_v[kWarps], s_best[kEndCtas];
    __shared__ int s_i[kWarps], s_at[kEndCtas];
    const int rank = blockIdx.x % kEndCtas, seq = blockIdx.x / kEndCtas;
    if constexpr (kEndCtas > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    pdl_begin();
    logits += (size_t)seq * vocab;
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    constexpr int kPer = 16 / (int)sizeof(L);
    const int nvec = vocab / kPer;   // 16-byte loads; indices ascend within a thread, so '>' keeps the lowest
    const int v0 = (int)((long long)nvec * rank / kEndCtas), v1 = (int)((long long)nvec * (rank + 1) / kEndCtas);
#pragma unroll 2
    for (int vi = v0 + threadIdx.x; vi < v1; vi += kEndThreads) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(logits) + vi);
        const L* hp = reinterpret_cast<const L*>(&a);
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const float v = to_f32(hp[q]);
            if (v > best) { best = v; best_i = vi * kPer + q; }
        }
    }
    if (rank == kEndCtas - 1)
        for (int i = nvec * kPer + threadIdx.x; i < vocab; i += kEndThreads) {
            const float v = to_f32(logits[i]);
            if (v > best || (v == best && i < best_i)) { best = v; best_i = i; }
        }
    const auto better = [](float v, int i, float w, int j) { return v > w || (v == w && i < j); };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (better(ov, oi, best, best_i)) { best = ov; best_i = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { s_v[warp] = best; s_i[warp] = best_i; }
    __syncthreads();
    if constexpr (kEndCtas > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");        // every CTA of the cluster runs
    if (warp == 0) {
        best = s_v[lane % kWarps];
        best_i = s_i[lane % kWarps];
#pragma unroll
        for (int o = kWarps / 2; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
            if (better(ov, oi, best, best_i)) { best = ov; best_i = oi; }
        }
        if (lane == 0) {
            uint32_t v, i;
            asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(v) : "r"((uint32_t)__cvta_generic_to_shared(&s_best[rank])));
            asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(i) : "r"((uint32_t)__cvta_generic_to_shared(&s_at[rank])));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(v), "f"(best) : "memory");
            asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(i), "r"(best_i) : "memory");
        }
        __syncwarp();
    }
    if constexpr (kEndCtas > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (rank == 0 && threadIdx.x == 0) {
        best = s_best[0];
        best_i = s_at[0];
#pragma unroll
        for (int r = 1; r < kEndCtas; ++r)
            if (better(s_best[r], s_at[r], best, best_i)) { best = s_best[r]; best_i = s_at[r]; }
        if (best_i == 0x7fffffff) best_i = 0;   // all-NaN row
        token[seq] = best_i;
        const int step = step_ptr[seq];
        if (step < history_cap) history[(size_t)seq * history_cap + step] = best_i;
        step_ptr[seq] = step + 1;
        pos[seq] += 1;
        if (parity != nullptr) *parity ^= 1;
    }
}

}  // namespace leankv
