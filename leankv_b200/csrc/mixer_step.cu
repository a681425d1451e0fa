// One decode step of a layer's token mixers, in one launch. The first thread-block cluster runs the window +
// pooled-block attention (its CTAs split the visible keys and merge through distributed shared memory), every
// further CTA one head of the matrix-state time mixing: the two mixers read the same projections and are
// independent, so they run side by side.

#include <algorithm>

#include "decode_frame.cuh"
#include "window_pool.cuh"

namespace leankv {
namespace {

constexpr int kStepThreads = 512;
constexpr int kStepSmemFloats = 200 * 1024 / 4;

struct StepParams {
    leankv_window_pool_t left;
    leankv_time_mix_t right;
    leankv_mixer_step_t s;
    int has_left, has_right, n_max, cluster, norms_aligned;
    float inv_dim, inv_vdim;
};

constexpr int kRowVecs = 6;        // float4s of the projection row a thread keeps: rows up to 12288 columns

template <typename T>
__device__ void left_step(const StepParams& p, float* sm, float* s_tmp, int rank) {
    const leankv_window_pool_t& a = p.left;
    const AttendPlan pl(a, kStepThreads, (p.n_max + p.cluster - 1) / p.cluster, kStepSmemFloats);
    const int tid = threadIdx.x, i = p.s.state[kPos], G = a.kv_heads;
    const int nq = a.heads * a.dim, nk = G * a.dim, nv = G * a.vdim;
    const float* y = p.s.y + p.s.qkv_off;       // biases are already in
    T* k_ring = static_cast<T*>(a.k_ring);
    T* v_ring = static_cast<T*>(a.v_ring);

    // before the projections are there: the mix, and this CTA's key / value rows on their way into L2
    put_talk(a, pl, sm);
    {
        const VisibleKeys vis(i, a.size, a.pool);
        const int j0 = (int)((long long)vis.n * rank / p.cluster), j1 = (int)((long long)vis.n * (rank + 1) / p.cluster);
        const int kb = G * a.dim_pad * (int)sizeof(T), per = (kb + 127) / 128;
        const int vb = G * a.vdim_pad * (int)sizeof(T), perv = (vb + 127) / 128;
        for (int e = tid; e < (j1 - j0) * (per + perv); e += kStepThreads) {
            const int jl = e / (per + perv), c = e - jl * (per + perv), j = j0 + jl;
            const int row = j < vis.n_blk ? j : (vis.w0 + j - vis.n_blk) % a.ring;
            const char* base = c < per ? static_cast<const char*>(j < vis.n_blk ? a.k_pool : a.k_ring) + (size_t)row * kb + c * 128
                                       : static_cast<const char*>(j < vis.n_blk ? a.v_pool : a.v_ring) + (size_t)row * vb + (c - per) * 128;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(base));
        }
    }
    pdl_begin();

    const int slot = i % a.ring;
    T* k_new = reinterpret_cast<T*>(sm + pl.knew);
    T* v_new = reinterpret_cast<T*>(sm + pl.vnew);
    auto put_k = [&](int g, int d, float v) {
        const T r = from_f32<T>(v);
        k_new[g * a.dim_pad + d] = r;
        if (rank == 0) k_ring[((size_t)slot * G + g) * a.dim_pad + d] = r;
    };
    auto put_v = [&](int g, int d, float v) {
        const T r = from_f32<T>(v);
        v_new[g * a.vdim_pad + d] = r;
        if (rank == 0) v_ring[((size_t)slot * G + g) * a.vdim_pad + d] = r;
    };
    if (a.dim % 4 == 0 && a.vdim % 4 == 0 && p.s.qkv_off % 4 == 0 && p.norms_aligned && nq + nk + nv <= kStepThreads * 4 * kRowVecs) {
        float4 x[kRowVecs];        // the row, read once
        float sq = 0.f, sk = 0.f;
#pragma unroll
        for (int n = 0; n < kRowVecs; ++n) {
            const int e = (tid + n * kStepThreads) * 4;
            x[n] = e < nq + nk + nv ? ld_cg_f32x4(y + e) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int n = 0; n < kRowVecs; ++n) {
            const int e = (tid + n * kStepThreads) * 4;
            const float ss = x[n].x * x[n].x + x[n].y * x[n].y + x[n].z * x[n].z + x[n].w * x[n].w;
            if (e < nq) sq += ss;
            else if (e < nq + nk) sk += ss;
        }
        const RowFactors f = norm_factors(sq, sk, nq, nk, a.q_norm != nullptr, a.k_norm != nullptr, a.eps, s_tmp);
#pragma unroll
        for (int n = 0; n < kRowVecs; ++n) {
            const int e = (tid + n * kStepThreads) * 4;
            if (e >= nq + nk + nv) continue;
            const bool is_q = e < nq, is_k = !is_q && e < nq + nk;
            const int at = is_q ? e : is_k ? e - nq : e - nq - nk, width = is_q || is_k ? a.dim : a.vdim;
            const int h = at / width, d = at - h * width;
            const float* w = is_q ? a.q_norm : is_k ? a.k_norm : nullptr;
            const float fac = is_q ? f.q * a.scale : is_k ? f.k : 1.f;
            float4 v = make_float4(x[n].x * fac, x[n].y * fac, x[n].z * fac, x[n].w * fac);
            if (w != nullptr) {
                const float4 g = *reinterpret_cast<const float4*>(w + at);
                v.x *= g.x; v.y *= g.y; v.z *= g.z; v.w *= g.w;
            }
            if (is_q) {
                put_query4<T>(pl, sm, a.heads, h, d, v);
            } else {
                const int to = h * (is_k ? a.dim_pad : a.vdim_pad) + d;
                store4((is_k ? k_new : v_new) + to, v);
                if (rank == 0)
                    store4((is_k ? k_ring : v_ring) + (size_t)slot * G * (is_k ? a.dim_pad : a.vdim_pad) + to, v);
            }
        }
    } else {
        const RowFactors f = row_factors(y, nullptr, nq, nk, a.q_norm != nullptr, a.k_norm != nullptr, a.eps, s_tmp);
        for (int e = tid; e < nq + nk + nv; e += kStepThreads) {
            if (e < nq) put_query<T>(pl, sm, a.heads, e / a.dim, e % a.dim, y[e] * f.q * (a.q_norm ? __ldg(a.q_norm + e) : 1.f) * a.scale);
            else if (e < nq + nk) put_k((e - nq) / a.dim, (e - nq) % a.dim, y[e] * f.k * (a.k_norm ? __ldg(a.k_norm + e - nq) : 1.f));
            else put_v((e - nq - nk) / a.vdim, (e - nq - nk) % a.vdim, y[e]);
        }
    }
    const int pd = a.dim_pad - a.dim, pv = a.vdim_pad - a.vdim;       // padding columns are zero
    for (int e = tid; e < a.heads * pd; e += kStepThreads) put_query<T>(pl, sm, a.heads, e / pd, a.dim + e % pd, 0.f);
    for (int e = tid; e < G * pd; e += kStepThreads) put_k(e / pd, a.dim + e % pd, 0.f);
    for (int e = tid; e < G * pv; e += kStepThreads) put_v(e / pv, a.vdim + e % pv, 0.f);
    __syncthreads();
    float* p_gmem = static_cast<float*>(p.s.ws) + (size_t)rank * 2 * a.heads * pl.ldp;
    attend_query<T, float>(a, pl, sm, p_gmem, i, true, rank, p.cluster, p.s.out, p.s.left_scale);

    // the block this token completes (not visible to it: it ends at i > i - size)
    if ((i + 1) % a.pool == 0 && (i + 1) / a.pool <= a.max_blocks) {
        const int b = i / a.pool, p0 = b * a.pool;
        auto mean = [&](const T* ring, const T* fresh, T* dst, int n) {
            for (int e = rank * kStepThreads + tid; e < n; e += p.cluster * kStepThreads) {
                float t = 0.f;
                for (int x = 0; x < a.pool - 1; ++x) t += to_f32(ring[(size_t)((p0 + x) % a.ring) * n + e]);
                dst[(size_t)b * n + e] = from_f32<T>((t + to_f32(fresh[e])) / (float)a.pool);
            }
        };
        mean(k_ring, k_new, static_cast<T*>(a.k_pool), G * a.dim_pad);
        mean(v_ring, v_new, static_cast<T*>(a.v_pool), G * a.vdim_pad);
    }
}

// ---- the attention step on tensor cores: bf16, up to 16 heads ----
//
// What bounds the step is its chain of short phases, each run once by a cold instruction cache, and the barriers between
// them. So: keys and values of the CTA's share come by cp.async, all at once; both products are a few MMA loops; and the mix across
// heads, being linear, follows the values instead of preceding them: every CTA multiplies its exponentials (against its own
// maximum) with the values of every kv head, pushes its sums and its statistics to the CTAs that own the columns, and one cluster
// barrier later these scale, add, mix and write. That is one exchange where mixing the weights first takes two.
// Exact where the FMA form is: queries are two bf16 numbers, exponentials three (24 bits), sums fp32. A step of six layers of
// width 1024 (1044 keys) took 247.6 us with the general kernel below and takes 197.4; four of width 2048 278 and 245. Behind the
// projections a layer's attention is 14 000 cycles: state and address arithmetic 1000, asking for the rows 3500 (the cp.async rate of
// one SM), norms and queries 2000, scores 1500, exponentials 1500, values 1700 (4400 at width 2048), the exchange 1500, the merge 3000.
constexpr int kTileHeads = 16;

struct TilePlan {
    int talk, q, s, p, stat, fac, recv, t, k, v, total;     // bytes
    int ldq, ldk, ldv, lds, ldp, hp, own;               // row lengths (elements); heads padded; value columns a CTA owns
    int rows, rows16;                                   // of a kv head's keys / values
    __host__ __device__ TilePlan(const leankv_window_pool_t& a, int cluster, int n_max) {
        const int n = (n_max + cluster - 1) / cluster, n16 = (n + 15) / 16 * 16;
        int o = 0;
        const auto take = [&](int bytes) { const int at = o; o += (bytes + 15) / 16 * 16; return at; };
        hp = a.heads > 8 ? 16 : 8;
        own = a.vdim / cluster;
        ldq = ldk = a.dim + 8;                          // 16 bytes past a multiple of 32: eight rows in different banks
        ldv = a.vdim + 8;
        lds = n16 + 4;
        ldp = n16 + 8;
        talk = take(a.heads * a.heads * 4);
        q = take(2 * a.heads * ldq * 2);
        s = take(a.heads * lds * 4);
        p = take(3 * hp * ldp * 2);
        stat = take(cluster * a.heads * 8);
        fac = take(cluster * hp * 4);
        recv = take(cluster * a.kv_heads * own * hp * 4);
        t = take(a.kv_heads * own * hp * 4);
        rows = n;
        rows16 = n16;
        k = take(n * a.kv_heads * ldk * 2);             // a last tile's rows beyond n are read and not used
        v = take(n16 * a.kv_heads * ldv * 2);
        const int read = k + (n * (a.kv_heads - 1) + n16) * ldk * 2;
        total = o > read ? o : read;
    }
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes, or zeros
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix2(uint32_t (&r)[2], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// 1 / sqrt(x): the approximation and a Newton step, without the subroutines of the exact division and root. Of a sum that is no longer
// finite it is 0, as those have it.
__device__ __forceinline__ float inv_sqrt(float x) {
    const float r = rsqrtf(x);
    return r > 0.f ? r * fmaf(-0.5f * x * r, r, 1.5f) : r;
}

// NT: blocks of eight heads. kTileVecs: float4s of the projection row a thread keeps. kSplit: half of the warps waits for the
// projections and makes queries of them while the other half, which need not wait, asks for the keys and values (the projections'
// launch holds the device's registers until it drains, so this one starts only shortly before it ends); with more than eight heads
// there is so much to ask for that all warps do that first (step of four layers 244 us, split 249; of six narrower ones 200, 197).
template <int NT, int kTileVecs, bool kSplit>
__device__ void left_tile(const StepParams& p, unsigned char* sm, float* s_tmp, int rank) {
    const leankv_window_pool_t& a = p.left;
    const int C = p.cluster;
    const TilePlan pl(a, C, p.n_max);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int H = a.heads, G = a.kv_heads, rep = H / G, dim = a.dim, vdim = a.vdim;
    float* s_talk = reinterpret_cast<float*>(sm + pl.talk);
    bf16* s_q = reinterpret_cast<bf16*>(sm + pl.q);
    float* s_s = reinterpret_cast<float*>(sm + pl.s);
    bf16* s_p = reinterpret_cast<bf16*>(sm + pl.p);
    float2* s_stat = reinterpret_cast<float2*>(sm + pl.stat);
    float* s_recv = reinterpret_cast<float*>(sm + pl.recv);
    float* s_t = reinterpret_cast<float*>(sm + pl.t);
    float* s_fac = reinterpret_cast<float*>(sm + pl.fac);
    bf16* s_k = reinterpret_cast<bf16*>(sm + pl.k);
    bf16* s_v = reinterpret_cast<bf16*>(sm + pl.v);

    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    if (!p.s.early_state) pdl_begin();
    const int i = p.s.state[kPos];
    constexpr int kFrontWarps = kStepThreads / 32 / (kSplit ? 2 : 1), kFront = kFrontWarps * 32;
    constexpr int kBack = kStepThreads / (kSplit ? 2 : 1);
    if (!kSplit || tid >= kFront) {
        // ---- keys and values of this CTA's share, the mix ----
        const VisibleKeys vis(i, a.size, a.pool);
        const int j0 = vis.n * rank / C, n = vis.n * (rank + 1) / C - j0, n16 = (n + 15) / 16 * 16;
        const int t = kSplit ? tid - kFront : tid, c = t & 15;
        int w0 = i % a.ring - (i - vis.w0);                 // ring slot of the window's first token
        if (w0 < 0) w0 += a.ring;
#pragma unroll 1
        for (int key = t >> 4; key < n16; key += kBack / 16) {
            const int j = j0 + key;
            const bool on = key < n, pooled = on && j < vis.n_blk;
            int row = pooled ? j : w0 + j - vis.n_blk;
            if (!pooled && row >= a.ring) row -= a.ring;
            if (!on) row = 0;
            const bf16* ks = static_cast<const bf16*>(pooled ? a.k_pool : a.k_ring) + (size_t)row * G * dim + c * 8;
            const bf16* vs = static_cast<const bf16*>(pooled ? a.v_pool : a.v_ring) + (size_t)row * G * vdim + c * 8;
            if (on && j == vis.n - 1) continue;             // this token's own row comes from its projections
#pragma unroll 1
            for (int g = 0; g < G; ++g) {
                if (on && c * 8 < dim) copy16(smem_addr(s_k + (g * pl.rows + key) * pl.ldk + c * 8), ks + g * dim, true);
                if (c * 8 < vdim) copy16(smem_addr(s_v + (g * pl.rows16 + key) * pl.ldv + c * 8), vs + g * vdim, on);
            }
        }
        if (a.talk != nullptr)
#pragma unroll 1
            for (int e = t; e < H * H; e += kBack) s_talk[e] = __ldg(a.talk + e);
        if (kSplit && p.s.early_state) pdl_begin();
    }
    if (!kSplit || tid < kFront) {
        // ---- this token's projections, norms, queries, the new row ----
        const int nq = H * dim, nk = G * dim, nv = G * vdim;
        const int mine = rank == C - 1 ? nq + nk + nv : nq;        // the last CTA also takes the token's own key and value
        const float* y = p.s.y + p.s.qkv_off;               // biases are already in
        float4 x[kTileVecs], gain[kTileVecs];
        int head[kTileVecs], col[kTileVecs];
#pragma unroll
        for (int u = 0; u < kTileVecs; ++u) {
            const int e = (tid + u * kFront) * 4, at = e < nq ? e : e < nq + nk ? e - nq : e - nq - nk;
            const int width = e < nq + nk ? dim : vdim;
            const float* w = e < nq ? a.q_norm : e < nq + nk ? a.k_norm : nullptr;
            gain[u] = w != nullptr && e < mine ? __ldg(reinterpret_cast<const float4*>(w + at)) : make_float4(1.f, 1.f, 1.f, 1.f);
            head[u] = (int)(((float)at + 0.5f) * (e < nq + nk ? p.inv_dim : p.inv_vdim));      // at < 2^13: exact
            col[u] = at - head[u] * width;
        }
        if (p.s.early_state) pdl_begin();
        float sq = 0.f, sk = 0.f;
#pragma unroll
        for (int u = 0; u < kTileVecs; ++u) {
            const int e = (tid + u * kFront) * 4;
            x[u] = e < mine ? ld_cg_f32x4(y + e) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kTileVecs; ++u) {
            const int e = (tid + u * kFront) * 4;
            const float ss = x[u].x * x[u].x + x[u].y * x[u].y + x[u].z * x[u].z + x[u].w * x[u].w;
            if (e < nq) sq += ss;
            else if (e < nq + nk) sk += ss;
        }
        sq = warp_sum(sq);
        sk = warp_sum(sk);
        if (lane == 0) { s_tmp[warp] = sq; s_tmp[kFrontWarps + warp] = sk; }
        if (kSplit) asm volatile("bar.sync 1, %0;" ::"n"(kFront) : "memory");
        else __syncthreads();
        sq = s_tmp[lane % kFrontWarps];
        sk = s_tmp[kFrontWarps + lane % kFrontWarps];
#pragma unroll
        for (int o = kFrontWarps / 2; o > 0; o >>= 1) {
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
            sk += __shfl_xor_sync(0xffffffffu, sk, o);
        }
        const float fq = (a.q_norm != nullptr ? inv_sqrt(sq / (float)nq + a.eps) : 1.f) * a.scale;
        const float fk = a.k_norm != nullptr ? inv_sqrt(sk / (float)nk + a.eps) : 1.f;
#pragma unroll
        for (int u = 0; u < kTileVecs; ++u) {
            const int e = (tid + u * kFront) * 4;
            if (e >= mine) break;
            const bool is_q = e < nq, is_k = !is_q && e < nq + nk;
            const int h = head[u], d = col[u];
            const float fac = is_q ? fq : is_k ? fk : 1.f;
            const float4 v = make_float4(x[u].x * fac * gain[u].x, x[u].y * fac * gain[u].y, x[u].z * fac * gain[u].z,
                                         x[u].w * fac * gain[u].w);
            if (is_q) {
                uint2 hi, lo;
                split_bf16(v.x, v.y, hi.x, lo.x);
                split_bf16(v.z, v.w, hi.y, lo.y);
                *reinterpret_cast<uint2*>(s_q + h * pl.ldq + d) = hi;
                *reinterpret_cast<uint2*>(s_q + (H + h) * pl.ldq + d) = lo;
            } else {
                const VisibleKeys vis(i, a.size, a.pool);
                const int last = vis.n - vis.n * rank / C - 1, slot = i % a.ring;
                store4(is_k ? s_k + (h * pl.rows + last) * pl.ldk + d : s_v + (h * pl.rows16 + last) * pl.ldv + d, v);
                store4((is_k ? static_cast<bf16*>(a.k_ring) : static_cast<bf16*>(a.v_ring)) +
                       ((size_t)slot * G + h) * (is_k ? dim : vdim) + d, v);
            }
        }
    }
    const VisibleKeys vis(i, a.size, a.pool);
    const int j0 = vis.n * rank / C, n = vis.n * (rank + 1) / C - j0, tiles = (n + 15) / 16;      // at most 2^27 keys fit any memory
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // ---- scores: a warp per (16 keys, kv head), keys as rows, the head's queries as columns ----
#pragma unroll 1
    for (int e = warp; e < tiles * G; e += kStepThreads / 32) {
        const int tile = e / G, g = e - tile * G;
        float hi[2][4] = {}, lo[2][4] = {};
        const uint32_t ka = smem_addr(s_k + (g * pl.rows + tile * 16 + (lane & 15)) * pl.ldk + (lane >> 4) * 8);
        const uint32_t qa = smem_addr(s_q + ((lane >> 4) * H + min(g * rep + (lane & 7), H - 1)) * pl.ldq + (lane >> 3 & 1) * 8);
#pragma unroll
        for (int d = 0; d < 128; d += 16) {
            if (d >= dim) break;
            uint32_t x[4], y[4];
            ldmatrix4(x, ka + d * 2);
            ldmatrix4(y, qa + d * 2);
            mma_bf16(hi[d / 16 % 2], x[0], x[1], x[2], x[3], y[0], y[1]);
            mma_bf16(lo[d / 16 % 2], x[0], x[1], x[2], x[3], y[2], y[3]);
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int h = 2 * (lane & 3) + (x & 1), key = tile * 16 + (lane >> 2) + (x < 2 ? 0 : 8);
            if (h < rep && key < n) s_s[(g * rep + h) * pl.lds + key] = (hi[0][x] + hi[1][x]) + (lo[0][x] + lo[1][x]);
        }
    }
    __syncthreads();

    // ---- exponentials against this CTA's maximum, as three bf16 numbers ----
#pragma unroll 1
    for (int h = warp; h < H; h += kStepThreads / 32) {
        float m = -INFINITY, l = 0.f;
#pragma unroll 1
        for (int j = lane; j < n; j += 32) m = fmaxf(m, s_s[h * pl.lds + j]);
        m = warp_max(m);
#pragma unroll 1
        for (int j = lane; j < tiles * 16; j += 32) {
            const float e = j < n ? expf(s_s[h * pl.lds + j] - m) : 0.f;
            l += e;
            const bf16 b0 = from_f32<bf16>(e);
            const float r0 = e - to_f32(b0);
            const bf16 b1 = from_f32<bf16>(r0);
            bf16* dst = s_p + h * pl.ldp + j;
            dst[0] = b0;
            dst[pl.hp * pl.ldp] = b1;
            dst[2 * pl.hp * pl.ldp] = from_f32<bf16>(r0 - to_f32(b1));
        }
        l = warp_sum(l);
        if (lane == 0) s_stat[rank * H + h] = make_float2(m, l);
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");        // every CTA of the cluster runs
#pragma unroll 1
    for (int e = tid; e < C * H; e += kStepThreads) {
        const int to = e / H, h = e - to * H;
        const float2 v = s_stat[rank * H + h];
        if (to != rank)
            asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};"
                         ::"r"(in_cta(smem_addr(s_stat + rank * H + h), to)), "f"(v.x), "f"(v.y) : "memory");
    }

    __syncwarp();

    // ---- values: a warp per 16 value columns of a kv head, columns as rows, all heads as columns ----
    const int blocks = vdim / 16;
#pragma unroll 1
    for (int e = warp; e < G * blocks; e += kStepThreads / 32) {
        const int g = e / blocks, d0 = (e - g * blocks) * 16;
        float acc[NT][4] = {}, mid[NT][4] = {}, low[NT][4] = {};
        const uint32_t va = smem_addr(s_v + (g * pl.rows16 + (lane & 7) + (lane >> 4) * 8) * pl.ldv + d0 + (lane >> 3 & 1) * 8);
        const uint32_t pa = smem_addr(s_p + ((lane >> 4) * pl.hp + (lane & 7)) * pl.ldp + (lane >> 3 & 1) * 8);
        const uint32_t pb = smem_addr(s_p + (2 * pl.hp + (lane & 7)) * pl.ldp + (lane >> 3 & 1) * 8);
#pragma unroll 1
        for (int t = 0; t < tiles; ++t) {
            uint32_t x[4];
            ldmatrix4_t(x, va + t * 16 * pl.ldv * 2);
#pragma unroll
            for (int b = 0; b < NT; ++b) {
                uint32_t w[4], r[2];
                ldmatrix4(w, pa + (b * 8 * pl.ldp + t * 16) * 2);
                ldmatrix2(r, pb + (b * 8 * pl.ldp + t * 16) * 2);
                mma_bf16(acc[b], x[0], x[1], x[2], x[3], w[0], w[1]);
                mma_bf16(mid[b], x[0], x[1], x[2], x[3], w[2], w[3]);
                mma_bf16(low[b], x[0], x[1], x[2], x[3], r[0], r[1]);
            }
        }
#pragma unroll
        for (int b = 0; b < NT; ++b)
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[b][u] += mid[b][u] + low[b][u];
#pragma unroll
        for (int u = 0; u < 2; ++u) {                       // to the CTA that owns the column
            const int d = d0 + (lane >> 2) + u * 8, to = d / pl.own;
            const uint32_t at = in_cta(smem_addr(s_recv + ((rank * G + g) * pl.own + d - to * pl.own) * pl.hp + 2 * (lane & 3)), to);
#pragma unroll
            for (int b = 0; b < NT; ++b)
                asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};"
                             ::"r"(at + b * 32), "f"(acc[b][2 * u]), "f"(acc[b][2 * u + 1]) : "memory");
        }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

    // ---- the owner: all shares on one scale, added in rank order, mixed across heads ----
#pragma unroll 1
    for (int e = tid; e < (H * C + 31) / 32 * 32; e += kStepThreads) {      // C lanes a head
        const int h = e / C, r = e - h * C;
        const float2 st = h < H ? s_stat[r * H + h] : make_float2(-INFINITY, 0.f);
        float m = st.x;
#pragma unroll 1
        for (int o = C / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const float w = st.y > 0.f ? expf(st.x - m) : 0.f;
        float l = st.y * w;
#pragma unroll 1
        for (int o = C / 2; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (h < H) s_fac[r * pl.hp + h] = w / l;
    }
    __syncthreads();
#pragma unroll 1
    for (int e = tid; e < G * pl.own * pl.hp; e += kStepThreads) {
        const int h = e & (pl.hp - 1), step = G * pl.own * pl.hp;
        float o = 0.f;
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r)
            if (r < C) o = fmaf(s_recv[r * step + e], s_fac[r * pl.hp + h], o);
        s_t[e] = o;
    }
    __syncthreads();
#pragma unroll 1
    for (int e = tid; e < H * pl.own; e += kStepThreads) {
        const int h = e / pl.own, d = e - h * pl.own;
        const float* t = s_t + ((h / rep) * pl.own + d) * pl.hp;
        float o = 0.f;
        if (a.talk != nullptr) {
#pragma unroll 4
            for (int x = 0; x < H; ++x) o = fmaf(s_talk[h * H + x], t[x], o);
        } else {
            o = t[h];
        }
        p.s.out[h * vdim + rank * pl.own + d] = o * p.s.left_scale;
    }

    // the block this token completes (not visible to it: it ends at i > i - size); the last CTA has its newest row
    if (rank == C - 1 && (i + 1) % a.pool == 0 && (i + 1) / a.pool <= a.max_blocks) {
        const int b = i / a.pool, p0 = b * a.pool;
        auto mean = [&](const bf16* ring, const bf16* fresh, bf16* dst, int width, int ld) {
#pragma unroll 1
            for (int e = tid; e < G * width; e += kStepThreads) {
                float t = 0.f;
                for (int x = 0; x < a.pool - 1; ++x) t += to_f32(ring[(size_t)((p0 + x) % a.ring) * G * width + e]);
                dst[(size_t)b * G * width + e] = from_f32<bf16>((t + to_f32(fresh[e / width * ld + e % width])) / (float)a.pool);
            }
        };
        mean(static_cast<const bf16*>(a.k_ring), s_k + (n - 1) * pl.ldk, static_cast<bf16*>(a.k_pool), dim, pl.rows * pl.ldk);
        mean(static_cast<const bf16*>(a.v_ring), s_v + (n - 1) * pl.ldv, static_cast<bf16*>(a.v_pool), vdim, pl.rows16 * pl.ldv);
    }
}

// One head of the recurrence. With early_state its state, decay matrix and constants are in registers by the time the projections
// are there (heads up to 64 x 64, decay inputs up to 64 numbers): what is left behind them is the chain of tanh, decay, update, norm.
constexpr int kKeptRows = 8;       // state rows a thread keeps
constexpr int kKeptDecays = 4;     // decay rows a warp keeps

template <typename T>
__device__ void right_step(const StepParams& p, float* sm, float* s_tmp, int head) {
    const leankv_time_mix_t& a = p.right;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d = a.dim, N = a.heads * d, c0 = head * d;
    float* s_r = sm;
    float* s_k = s_r + d;
    float* s_w = s_k + d;
    float* s_v = s_w + d;
    float* s_o = s_v + d;                      // [slices][d]
    if (!p.s.early_state) pdl_begin();
    const T* w2 = static_cast<const T*>(p.s.w2);
    const int slices = max(1, kStepThreads / d), sl = tid / d, col = tid - sl * d;
    const int k0 = d * min(sl, slices) / slices, k1 = d * min(sl + 1, slices) / slices;
    const bool kept = (d + slices - 1) / slices <= kKeptRows && d <= kKeptDecays * (kStepThreads / 32) && p.s.rank <= 64;
    float* S = a.S + (size_t)head * d * d;
    float S_old[kKeptRows], dec[kKeptDecays][2], w0[kKeptDecays];
    const float u = tid < d ? __ldg(a.u + c0 + tid) : 0.f, gain = tid < d ? __ldg(a.norm + c0 + tid) : 0.f;
    if (kept) {
#pragma unroll
        for (int x = 0; x < kKeptRows; ++x) S_old[x] = k0 + x < k1 ? S[(size_t)(k0 + x) * d + col] : 0.f;
#pragma unroll
        for (int x = 0; x < kKeptDecays; ++x) {
            const int c = warp + x * (kStepThreads / 32);
            const T* row = w2 + (size_t)(c0 + c) * p.s.rank;
            dec[x][0] = c < d && lane < p.s.rank ? to_f32(row[lane]) : 0.f;
            dec[x][1] = c < d && lane + 32 < p.s.rank ? to_f32(row[lane + 32]) : 0.f;
            w0[x] = c < d ? __ldg(a.w0 + c0 + c) : 0.f;
        }
    }
    if (p.s.early_state) pdl_begin();
    const float* y = p.s.y + p.s.rkvg_off + c0;
    const float* y1 = p.s.y + p.s.w1_off;
    float bonus = 0.f;
    const float gate = tid < d ? y[3 * N + tid] : 0.f;
    if (tid < d) {
        const float r = y[tid], k = y[N + tid];
        s_r[tid] = r;
        s_k[tid] = k;
        s_v[tid] = y[2 * N + tid];
        bonus = r * u * k;
    }
    if (kept) {
        const float t0 = lane < p.s.rank ? tanhf(y1[lane]) : 0.f, t1 = lane + 32 < p.s.rank ? tanhf(y1[lane + 32]) : 0.f;
#pragma unroll
        for (int x = 0; x < kKeptDecays; ++x) {
            const int c = warp + x * (kStepThreads / 32);
            const float z = warp_sum(fmaf(dec[x][1], t1, dec[x][0] * t0));
            if (lane == 0 && c < d) s_w[c] = expf(-expf(z + w0[x]));
        }
    } else {
        for (int c = warp; c < d; c += kStepThreads / 32) {
            float z = 0.f;
            for (int x = lane; x < p.s.rank; x += 32) z = fmaf(to_f32(w2[(size_t)(c0 + c) * p.s.rank + x]), tanhf(y1[x]), z);
            z = warp_sum(z);
            if (lane == 0) s_w[c] = expf(-expf(z + __ldg(a.w0 + c0 + c)));
        }
    }
    bonus = cta_sum(bonus, s_tmp);             // synchronises
    if (sl < slices) {
        const float v = s_v[col];
        float o = 0.f;
        if (kept) {
#pragma unroll
            for (int x = 0; x < kKeptRows; ++x) {
                const int k = k0 + x;
                if (k < k1) {
                    o = fmaf(s_r[k], S_old[x], o);
                    S[(size_t)k * d + col] = fmaf(s_w[k], S_old[x], s_k[k] * v);
                }
            }
        } else {
#pragma unroll 4
            for (int k = k0; k < k1; ++k) {
                const float s = S[(size_t)k * d + col];
                o = fmaf(s_r[k], s, o);
                S[(size_t)k * d + col] = fmaf(s_w[k], s, s_k[k] * v);
            }
        }
        s_o[sl * d + col] = o;
    }
    __syncthreads();
    float o = 0.f;
    if (tid < d) {
        for (int x = 0; x < slices; ++x) o += s_o[x * d + tid];
        o = fmaf(bonus, s_v[tid], o);
    }
    const float f = p.s.right_scale / sqrtf(cta_sum(o * o, s_tmp) / (float)d + a.eps);
    if (tid < d) p.s.out[p.s.right_off + c0 + tid] = o * f * gain * gate * sigmoid_f32(gate);
}

template <typename T>
__global__ void __launch_bounds__(kStepThreads) mixer_step_kernel(const __grid_constant__ StepParams p) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float s_tmp[32];
    const int first = p.has_left ? p.cluster : 0;
    if ((int)blockIdx.x < first) left_step<T>(p, sm, s_tmp, blockIdx.x);
    else if ((int)blockIdx.x - first < p.right.heads) right_step<T>(p, sm, s_tmp, blockIdx.x - first);
}

template <int NT, int kTileVecs, bool kSplit>
__global__ void __launch_bounds__(kStepThreads) mixer_step_tile_kernel(const __grid_constant__ StepParams p) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float s_tmp[32];
    if ((int)blockIdx.x < p.cluster) left_tile<NT, kTileVecs, kSplit>(p, reinterpret_cast<unsigned char*>(sm), s_tmp, blockIdx.x);
    else if ((int)blockIdx.x - p.cluster < p.right.heads) right_step<bf16>(p, sm, s_tmp, blockIdx.x - p.cluster);
}

int keys_bound(const leankv_window_pool_t& a, int max_pos) {
    return VisibleKeys(std::max(max_pos - 1, 0), a.size, a.pool).n;
}

// One cluster of 16 CTAs, or of 8 where the device does not place 16, and the heads of the recurrence behind it.
template <typename Kernel, typename Smem>
int launch_clusters(StepParams& p, Kernel kernel, Smem smem_of, cudaStream_t st) {
    LEANKV_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    for (p.cluster = kMaxCluster;; p.cluster = 8) {
        const size_t smem = smem_of();
        if (smem > 226 * 1024) return LEANKV_ELIMIT;
        LEANKV_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        const int heads = p.has_right ? p.right.heads : 0;
        const int grid = (p.has_left ? p.cluster : 0) + (heads + p.cluster - 1) / p.cluster * p.cluster;
        if (p.cluster > 8) {      // does a cluster of this size fit this device?
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(grid);
            cfg.blockDim = dim3(kStepThreads);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = p.cluster;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int fits = 0;
            if (cudaOccupancyMaxActiveClusters(&fits, kernel, &cfg) != cudaSuccess || fits < 1) {
                (void)cudaGetLastError();
                continue;
            }
        }
        LEANKV_CUDA_TRY(launch_cluster_kernel_ex(true, dim3(p.cluster), kernel, dim3(grid), dim3(kStepThreads), smem, st, p));
        return LEANKV_OK;
    }
}

template <typename T>
int launch_step(StepParams& p, cudaStream_t st) {
    const leankv_window_pool_t& a = p.left;
    const size_t right = p.has_right ? (size_t)(4 * p.right.dim + kStepThreads + p.right.dim) * 4 : 0;
    // The tensor-core kernel where the sums of all heads with every kv head fit: up to sixteen heads, whole 16-column pieces, and a
    // share of the keys that fits into shared memory (width 1024: 2800 visible keys, width 2048: 1200); else the general one.
    if (sizeof(T) == 2 && p.has_left && a.heads <= kTileHeads && a.heads / a.kv_heads <= 8 && a.dim == a.dim_pad && a.vdim == a.vdim_pad &&
        a.dim <= 128 && a.vdim <= 128 && p.s.qkv_off % 4 == 0 && p.norms_aligned && aligned16(a.k_ring) && aligned16(a.v_ring) &&
        aligned16(a.k_pool) && aligned16(a.v_pool)) {
        const auto smem_of = [&] { return std::max((size_t)TilePlan(a, p.cluster, p.n_max).total, right); };
        const int row = a.heads * a.dim + a.kv_heads * (a.dim + a.vdim);
        const int rc = a.heads > 8 ? launch_clusters(p, mixer_step_tile_kernel<2, 3, false>, smem_of, st)
                       : row > 2048 ? launch_clusters(p, mixer_step_tile_kernel<1, 3, false>, smem_of, st)
                                    : launch_clusters(p, mixer_step_tile_kernel<1, 2, true>, smem_of, st);
        if (rc != LEANKV_ELIMIT) return rc;
    }
    return launch_clusters(p, mixer_step_kernel<T>, [&] {
        const size_t left = p.has_left
            ? 4 * (size_t)AttendPlan(a, kStepThreads, (p.n_max + p.cluster - 1) / p.cluster, kStepSmemFloats).total : 0;
        return std::max(left, right);
    }, st);
}

}  // namespace
}  // namespace leankv

using namespace leankv;

extern "C" size_t leankv_mixer_step_workspace_bytes(const leankv_window_pool_t* left, int max_pos) {
    if (!left || max_pos <= 0) return 0;
    const int n = keys_bound(*left, max_pos);
    size_t need = 0;
    for (int c = 8; c <= kMaxCluster; c *= 2) {
        const AttendPlan pl(*left, kStepThreads, (n + c - 1) / c, kStepSmemFloats);
        if (!pl.p_in_smem) need = std::max(need, (size_t)c * 2 * left->heads * pl.ldp * 4);
    }
    return need;
}

extern "C" int leankv_mixer_step(const leankv_window_pool_t* left, const leankv_time_mix_t* right,
                                 const leankv_mixer_step_t* s, void* stream) {
    if (!s || (!left && !right) || !s->y || !s->out || !s->state || s->max_pos <= 0) return LEANKV_EINVAL;
    StepParams p{};
    p.s = *s;
    int dtype = 0;
    if (left) {
        if (left->heads <= 0 || left->kv_heads <= 0 || left->heads % left->kv_heads || left->dim <= 0 ||
            left->vdim <= 0 || left->size <= 0 || left->pool <= 0 || !left->k_ring || !left->v_ring)
            return LEANKV_EINVAL;
        if (left->ring < std::max(left->size, left->pool) ||
            VisibleKeys(s->max_pos - 1, left->size, left->pool).n_blk > left->max_blocks)
            return LEANKV_ELIMIT;
        if (left->dim_pad % 16 || left->vdim_pad % 16 || left->dim_pad < left->dim || left->vdim_pad < left->vdim)
            return LEANKV_EALIGN;
        if (leankv_mixer_step_workspace_bytes(left, s->max_pos) > (s->ws ? s->ws_bytes : 0)) return LEANKV_EWORKSPACE;
        p.left = *left;
        p.has_left = 1;
        p.norms_aligned = aligned16(left->q_norm) && aligned16(left->k_norm) && aligned16(s->y);
        p.n_max = keys_bound(*left, s->max_pos);
        p.inv_dim = 1.f / (float)left->dim;
        p.inv_vdim = 1.f / (float)left->vdim;
        dtype = left->dtype;
    }
    if (right) {
        if (right->heads <= 0 || right->dim <= 0 || right->dim > kStepThreads || !right->S || !right->u || !right->w0 ||
            !right->norm || !s->w2 || s->rank <= 0 || (left && left->dtype != right->dtype))
            return LEANKV_EINVAL;
        p.right = *right;
        p.has_right = 1;
        dtype = right->dtype;
    }
    if (dtype != LEANKV_DT_BF16 && dtype != LEANKV_DT_F32) return LEANKV_EUNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return dtype == LEANKV_DT_BF16 ? launch_step<bf16>(p, st) : launch_step<float>(p, st);
}
