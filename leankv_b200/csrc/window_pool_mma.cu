// Window + pooled-block attention of a prompt portion on the fifth-generation tensor cores (bf16 operands, fp32 scores, weights,
// outputs and mix). The mix of the softmax weights across heads is linear, so it follows the values instead of preceding them:
//
//   out[h'] = sum over h of talk[h'][h] * (weights of h times the values of h's kv head)
//
// A CTA holds 128 rows, (token, query head) pairs of one kv head g, and multiplies their weights with the values of one kv head gv,
// tile after tile as the causal kernel does. At the end it mixes its own heads into the query heads of gv; the CTAs of all g are one
// cluster and add their shares, in order of g, through distributed shared memory. Every head meets the values of every kv
// head that way: kv_heads times the products of plain attention, on units that do sixteen times what mma.sync does, and the
// weights of all heads never have to be in one place.
//
// What bounds it is the tensor pipe and the exponentials beside it (scores and weights are computed once per gv): 805 TFLOP/s with 16
// heads of 4 kv heads. 2048 tokens, window 1024, pool 16, with the mma.sync kernel (window_pool_tile.cu) / here: 16 heads, 4 kv heads
// 194 / 108 us; 8 heads, 2 kv heads 127 / 39; 48 tokens of the first 18.7 / 12.7. Error against 64 bits 2.3e-3 / 1.6e-3 (there a mixed
// weight is rounded to bf16). With 8 kv heads the products are too many: 32 heads 396 / 424, 8 heads of 64 numbers 43.4 / 44.4.
//
// Key tiles are 64 pooled blocks, or 64 tokens of the window; where the ring wraps a tile ends at its end. Rows of a tile that no
// query of the portion may see are zeros (beyond what the sequence has written) or finite.

#include <algorithm>

#include "tile_softmax.cuh"
#include "tma.cuh"
#include "window_pool.cuh"

namespace leankv {
namespace {

constexpr int kThreads = 192;
constexpr int kMaxRep = 8;                       // query heads per kv head
constexpr int kMaxKvHeads = 4;                   // CTAs of a cluster

struct MixArgs {
    CUtensorMap q, k, k_pool, v, v_pool;
    const float* talk;
    bf16* out;
    int* status;
    int out_ld, rows, start, size, pool, ring;
    int heads, kv_heads, rep, tq;                // tq: tokens of a CTA
    int dim_pad, vdim, vdim_pad, nb, nbv, vec;   // nb, nbv: 64-column blocks
    uint32_t q_box;
    float c, out_scale;                          // c: scale * log2(e)
};

// The key tiles that the tokens of a CTA see: pooled blocks, then the window up to the ring's end, then from its start.
struct KeyTiles {
    int n_pool, n_a, n, tok0, len_a, slot0;
    __device__ KeyTiles(const VisibleKeys& first, const VisibleKeys& last, int i_last, int ring) {
        n_pool = (last.n_blk + kKeys - 1) / kKeys;
        tok0 = first.w0;
        slot0 = tok0 % ring;
        const int n_tok = i_last - tok0 + 1;
        len_a = min(n_tok, ring - slot0);
        n_a = (len_a + kKeys - 1) / kKeys;
        n = n_pool + n_a + (n_tok - len_a + kKeys - 1) / kKeys;
    }
    struct Tile { bool pooled; int at, slot, count; };       // first key's number or position, its row, rows that count
    __device__ Tile operator()(int j) const {
        if (j < n_pool) return {true, j * kKeys, j * kKeys, kKeys};
        j -= n_pool;
        if (j < n_a) return {false, tok0 + j * kKeys, slot0 + j * kKeys, min(kKeys, len_a - j * kKeys)};
        j -= n_a;
        return {false, tok0 + len_a + j * kKeys, j * kKeys, kKeys};
    }
};

enum { kQ, kO, kKFull, kKFree = kKFull + 2, kVFull = kKFree + 2, kS = kVFull + 2, kP = kS + 2, kPV = kP + 2, kBars = kPV + 2 };

__global__ void __launch_bounds__(kThreads, 2) window_pool_mma_kernel(const __grid_constant__ MixArgs p) {
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ __align__(8) uint64_t s_bar[kBars];
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    __shared__ float s_talk[kMaxRep][kMaxRep];           // [head of gv][head of g]
    pdl_begin();
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t base = (umma::smem_addr(raw) + 1023u) & ~1023u;
    const uint32_t k_bytes = p.nb * kKeyBlock, v_bytes = p.nbv * kKeyBlock;      // of a buffer
    const uint32_t sq = base, sk = sq + p.nb * kBlock, sv = sk + 2 * k_bytes;
    // barrier pairs: tile j uses b + (j & 1), in its phase j / 2
    auto bar = [&](int b) { return umma::smem_addr(&s_bar[b]); };
    auto wait = [&](int b, int j) { return umma::bar_wait(bar(b + (j & 1)), (j >> 1) & 1); };
    const int g = blockIdx.y, gv = blockIdx.z;
    if (tid == 0) {
        for (int b = 0; b < kBars; ++b) umma::bar_init_n(bar(b), b == kP || b == kP + 1 ? kTile : 1);
        s_fail = 0;
    }
    if (tid < p.rep * p.rep)
        s_talk[tid / p.rep][tid % p.rep] = __ldg(p.talk + (size_t)(gv * p.rep + tid / p.rep) * p.heads + g * p.rep + tid % p.rep);
    if (warp == 4) umma::tmem_alloc_n(umma::smem_addr(&s_tmem), 256);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0), tm_s = tmem, tm_o = tmem + kTile;

    const int q0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * p.tq;        // the longest rows first
    const int nt = min(p.tq, p.rows - q0), used = p.rep * nt, i_last = p.start + q0 + nt - 1;
    const KeyTiles tiles(VisibleKeys(p.start + q0, p.size, p.pool), VisibleKeys(i_last, p.size, p.pool), i_last, p.ring);
    const int n_tiles = tiles.n, ld = (p.vdim_pad + 31) / 32 * 32 + 4;
    float* rows = reinterpret_cast<float*>(raw + (base - umma::smem_addr(raw)));
    bool ok = true;

    if (tid == 128) {                                    // ---- copies ----
        tma::expect(bar(kQ), p.nb * p.q_box);
        for (int b = 0; b < p.nb; ++b) tma::load3(sq + b * kBlock, &p.q, b * 64, g * p.rep, q0, bar(kQ));
        int nk = 0, nv = 0;
        for (int j = 0; j < n_tiles; ++j) {
            const KeyTiles::Tile t = tiles(j);
            const int odd = j & 1;
            if (j > 1) ok = wait(kKFree, j - 2);
            if (!ok) break;
            tma::expect(bar(kKFull + odd), k_bytes);
            for (int b = 0; b < p.nb; ++b)
                tma::load3(sk + odd * k_bytes + b * kKeyBlock, t.pooled ? &p.k_pool : &p.k, b * 64, g, t.slot, bar(kKFull + odd));
            ++nk;
            if (j > 1) ok = wait(kPV, j - 2);
            if (!ok) break;
            tma::expect(bar(kVFull + odd), v_bytes);
            for (int b = 0; b < p.nbv; ++b)
                tma::load3(sv + odd * v_bytes + b * kKeyBlock, t.pooled ? &p.v_pool : &p.v, b * 64, gv, t.slot, bar(kVFull + odd));
            ++nv;
        }
        if (!ok) {                                       // give up only once the copies in flight have landed
            umma::bar_wait(bar(kQ), 0);
            for (int j = max(nk - 2, 0); j < nk; ++j) wait(kKFull, j);
            for (int j = max(nv - 2, 0); j < nv; ++j) wait(kVFull, j);
        }
    } else if (warp == 5) {                              // ---- products: the whole warp waits, one lane issues ----
        constexpr uint32_t idesc_s = tma::idesc_bf16(kKeys, false);
        const uint32_t idesc_o = tma::idesc_bf16(p.vdim_pad, true);
        const uint64_t desc_q = tma::swizzled(sq, 16), desc_k = tma::swizzled(sk, 16), desc_v = tma::swizzled(sv, kKeyBlock);
        auto all = [&](bool done) { return __all_sync(0xffffffffu, done) != 0; };
        auto scores = [&](int j) {
            ok = all(wait(kKFull, j));
            if (!ok) return;
            umma::fence_after_sync();
            const uint32_t to = tm_s + (j & 1) * kKeys;
            uint64_t dq = desc_q, dk = desc_k + (j & 1) * (k_bytes >> 4);
            if (umma::elect()) {
                for (int b = 0; b < p.nb; ++b, dq += kBlock >> 4, dk += kKeyBlock >> 4) {
                    const int steps = p.dim_pad / 16 - b * 4;
                    umma::mma_f16_n(to, dq, dk, idesc_s, b > 0);
#pragma unroll
                    for (int s = 1; s < 4; ++s)
                        if (s < steps) umma::mma_f16_n(to, dq + 2 * s, dk + 2 * s, idesc_s, 1);
                }
                umma::commit(bar(kS + (j & 1)));
                umma::commit(bar(kKFree + (j & 1)));
            }
            __syncwarp();
        };
        ok = all(umma::bar_wait(bar(kQ), 0));
        for (int j = 0; j < min(2, n_tiles) && ok; ++j) scores(j);
        for (int j = 0; j < n_tiles && ok; ++j) {
            ok = all(wait(kVFull, j));
            ok = ok && all(wait(kP, j));
            if (!ok) break;
            umma::fence_after_sync();
            const uint64_t dv = desc_v + (j & 1) * (v_bytes >> 4);
            const uint32_t pa = tm_s + (j & 1) * kKeys;
            if (umma::elect()) {
#pragma unroll
                for (int s = 0; s < kKeys / 16; ++s) {   // 16 keys: high parts, then low parts
                    umma::mma_f16_ts(tm_o, pa + (s >> 1) * 32 + (s & 1) * 8, dv + s * (2048 >> 4), idesc_o, j > 0 || s > 0);
                    umma::mma_f16_ts(tm_o, pa + (s >> 1) * 32 + (s & 1) * 8 + 16, dv + s * (2048 >> 4), idesc_o, 1);
                }
                umma::commit(bar(kPV + (j & 1)));
            }
            __syncwarp();
            if (j + 2 < n_tiles) {                       // its scores go over these weights
                ok = all(wait(kPV, j));
                if (ok) scores(j + 2);
            }
        }
        if (umma::elect()) umma::commit(bar(kO));
        __syncwarp();
        if (!ok) umma::bar_wait(bar(kO), 0);
    } else if (tid < kTile) {                            // ---- rows ----
        const int row0 = warp * 32, i = p.start + q0 + min(tid, used - 1) / p.rep;
        const VisibleKeys vis(i, p.size, p.pool);
        float m = -1e30f, l = 0.f;
        for (int j = 0; j < n_tiles; ++j) {
            ok = __all_sync(0xffffffffu, wait(kS, j));      // the warp stays together
            if (!ok) break;
            umma::fence_after_sync();
            const KeyTiles::Tile t = tiles(j);
            const uint32_t tm = tm_s + (j & 1) * kKeys;
            // this row's keys of the tile: from k0 to k1
            const int k0 = t.pooled ? 0 : vis.w0 - t.at, k1 = t.pooled ? vis.n_blk - 1 - t.at : min(i - t.at, t.count - 1);
            uint32_t s[2][32];
            umma::ld32_async(s[0], tm, row0, 0);
            umma::ld32_async(s[1], tm, row0, 32);
            umma::settle(s[0]);
            umma::settled(s[1]);
            if (__any_sync(0xffffffffu, k0 > 0 || k1 < kKeys - 1)) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int x = 0; x < 32; ++x)
                        if (c * 32 + x < k0 || c * 32 + x > k1) s[c][x] = 0xff800000u;      // -inf
            }
            const float best = largest(s);
            const bool raise = best * p.c > m + kSlack;
            if (__any_sync(0xffffffffu, raise)) {
                const float mn = raise ? best * p.c : m, f = ex2(m - mn);
                m = mn;
                l *= f;
                if (j > 0) {
                    ok = __all_sync(0xffffffffu, wait(kPV, j - 1));      // nothing is being added to the outputs
                    if (!ok) break;
                    umma::fence_after_sync();
                    scale_outputs(tm_o, row0, p.vdim_pad, f);
                }
            }
            l += put_weights(s, p.c, m, tm, row0);
            umma::stored();
            umma::fence_before_sync();
            umma::bar_arrive(bar(kP + (j & 1)));
        }
        if (ok) ok = __all_sync(0xffffffffu, umma::bar_wait(bar(kO), 0));
        umma::fence_after_sync();
        // normalised rows to shared memory (all copies and products are done); 16 bytes past a multiple of 128 apart
        const float inv = 1.f / l;
#pragma unroll 1
        for (int c = 0; c < p.vdim_pad; c += 32) {
            uint32_t o[32];
            umma::ld32(o, tm_o, row0, c);
#pragma unroll
            for (int x = 0; x < 32; x += 4)
                *reinterpret_cast<float4*>(rows + tid * ld + c + x) =
                    make_float4(__uint_as_float(o[x]) * inv, __uint_as_float(o[x + 1]) * inv, __uint_as_float(o[x + 2]) * inv,
                                __uint_as_float(o[x + 3]) * inv);
        }
    }
    if (!ok) s_fail = 1;
    __syncwarp();
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 4) {
        umma::fence_after_sync();
        umma::tmem_free_n(tmem, 256);
    }

    // ---- this CTA's heads mixed into the heads of gv, in place: a thread owns four columns of a token's heads ----
    const int quads = p.vdim_pad / 4;
    for (int e = tid; e < nt * quads; e += kThreads) {
        const int t = e / quads, d = (e - t * quads) * 4;
        float4 u[kMaxRep];
#pragma unroll
        for (int r = 0; r < kMaxRep; ++r)
            u[r] = r < p.rep ? *reinterpret_cast<const float4*>(rows + (t * p.rep + r) * ld + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int x = 0; x < p.rep; ++x) {
            float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int r = 0; r < kMaxRep; ++r)
                if (r < p.rep) {
                    const float w = s_talk[x][r];
                    y.x = fmaf(w, u[r].x, y.x); y.y = fmaf(w, u[r].y, y.y); y.z = fmaf(w, u[r].z, y.z); y.w = fmaf(w, u[r].w, y.w);
                }
            *reinterpret_cast<float4*>(rows + (t * p.rep + x) * ld + d) = y;
        }
    }
    if (s_fail) {                                        // a wait ran out: the portion's rows are not numbers
        if (tid == 0 && p.status != nullptr) atomicExch(p.status, 1);
        __syncthreads();
        for (int e = tid; e < used * ld; e += kThreads) rows[e] = __int_as_float(0x7fc00000);
    }
    // ---- the shares of all kv heads g: each CTA adds and writes its part of the rows ----
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    const int G = p.kv_heads, r0 = used * g / G, r1 = used * (g + 1) / G;
    for (int e = tid; e < (r1 - r0) * quads; e += kThreads) {
        const int r = r0 + e / quads, d = (e % quads) * 4;
        const uint32_t at = umma::smem_addr(rows + r * ld + d);
        float4 part[kMaxKvHeads];
#pragma unroll
        for (int c = 0; c < kMaxKvHeads; ++c) {
            uint32_t from;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from) : "r"(at), "r"(c < G ? c : g));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(part[c].x), "=f"(part[c].y), "=f"(part[c].z), "=f"(part[c].w) : "r"(from) : "memory");
        }
        float4 y = part[0];
#pragma unroll
        for (int c = 1; c < kMaxKvHeads; ++c)
            if (c < G) { y.x += part[c].x; y.y += part[c].y; y.z += part[c].z; y.w += part[c].w; }
        bf16* to = p.out + (size_t)(q0 + r / p.rep) * p.out_ld + (size_t)(gv * p.rep + r % p.rep) * p.vdim + d;
        y.x *= p.out_scale; y.y *= p.out_scale; y.z *= p.out_scale; y.w *= p.out_scale;
        if (p.vec) {
            if (d < p.vdim) store4(to, y);
        } else {
            const float v[4] = {y.x, y.y, y.z, y.w};
            for (int x = 0; x < 4; ++x)
                if (d + x < p.vdim) to[x] = from_f32<bf16>(v[x]);
        }
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");        // the others still read this CTA's rows
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

}  // namespace

int window_pool_mma_attend(const leankv_window_pool_t& a, const void* q, void* out, int out_ld, float out_scale, int rows, int start,
                           int* status, cudaStream_t st) {
    const int rep = a.heads / a.kv_heads;
    if (a.dtype != LEANKV_DT_BF16 || a.talk == nullptr || a.k_pool == nullptr || a.v_pool == nullptr || !(a.scale > 0.f) || a.dim_pad > 128 || a.vdim_pad > 128 || rep > kMaxRep ||
        a.kv_heads > kMaxKvHeads || !aligned16(q) || !aligned16(a.k_ring) || !aligned16(a.v_ring) || !aligned16(a.k_pool) ||
        !aligned16(a.v_pool))
        return LEANKV_EUNSUPPORTED;
    MixArgs p{};
    p.talk = a.talk;
    p.out = static_cast<bf16*>(out);
    p.status = status;
    p.out_ld = out_ld;
    p.rows = rows;
    p.start = start;
    p.size = a.size;
    p.pool = a.pool;
    p.ring = a.ring;
    p.heads = a.heads;
    p.kv_heads = a.kv_heads;
    p.rep = rep;
    p.tq = kTile / rep;
    p.dim_pad = a.dim_pad;
    p.vdim = a.vdim;
    p.vdim_pad = a.vdim_pad;
    p.nb = (a.dim_pad + 63) / 64;
    p.nbv = (a.vdim_pad + 63) / 64;
    p.vec = a.vdim % 4 == 0 && out_ld % 4 == 0 && aligned16(out);
    p.q_box = 128u * rep * p.tq;
    p.c = a.scale * 1.4426950408889634f;
    p.out_scale = out_scale;
    // operands, then the rows; more than a third of an SM's shared memory, so that no third CTA waits for tensor memory while
    // its cluster's others hold theirs
    size_t smem = std::max((size_t)(2 * p.nb + p.nbv) * kBlock, (size_t)kTile * ((a.vdim_pad + 31) / 32 * 32 + 4) * 4) + 1024;
    smem = std::max(smem, (size_t)80 * 1024);
    const cuuint64_t G = a.kv_heads, H = a.heads;
    const auto map = [](CUtensorMap* m, const void* base, cuuint64_t d, cuuint64_t h, cuuint64_t n, cuuint32_t bh, cuuint32_t bn) {
        const cuuint64_t dims[3] = {d, h, n}, strides[2] = {d, d * h};
        const cuuint32_t box[3] = {(cuuint32_t)tma::kBoxCols, bh, bn};
        return tma::make_map(m, base, 3, dims, strides, box);
    };
    // what the sequence has written so far; beyond it a copy reads zeros
    const cuuint64_t written = std::min(a.ring, start + rows), blocks = std::max(1, std::min(a.max_blocks, (start + rows) / a.pool));
    int rc = map(&p.q, q, a.dim_pad, H, rows, rep, p.tq);
    if (!rc) rc = map(&p.k, a.k_ring, a.dim_pad, G, written, 1, kKeys);
    if (!rc) rc = map(&p.v, a.v_ring, a.vdim_pad, G, written, 1, kKeys);
    if (!rc) rc = map(&p.k_pool, a.k_pool, a.dim_pad, G, blocks, 1, kKeys);
    if (!rc) rc = map(&p.v_pool, a.v_pool, a.vdim_pad, G, blocks, 1, kKeys);
    if (rc) return LEANKV_EUNSUPPORTED;                  // sizes that a tensor map does not describe
    LEANKV_CUDA_TRY(cudaFuncSetAttribute(window_pool_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    LEANKV_CUDA_TRY(launch_cluster_kernel_ex(false, dim3(1, a.kv_heads, 1), window_pool_mma_kernel,
                                             dim3((rows + p.tq - 1) / p.tq, a.kv_heads, a.kv_heads), dim3(kThreads), smem, st, p));
    return LEANKV_OK;
}

}  // namespace leankv
