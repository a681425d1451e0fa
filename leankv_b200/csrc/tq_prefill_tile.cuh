// Causal attention of a chunk of prompt tokens over the packed pages, in two kernels (included by tq_attn.cu, inside
// namespace leankv::{anonymous}).
//
// The page-walking kernel (tq_prefill_t5_kernel) de-quantizes every page once per query tile, 32 keys at a time, which is
// what its 184 us for 512 tokens after 3584 went into (the two products need 25 us). Here the pages are
// looked up once: tq_expand_kernel writes the centroids of 128 tokens at a time (fp16, as they are: norms stay
// apart) in the very layout the tensor cores read, keys [token][coordinate] and values [coordinate][token], so that
// the attention kernel fetches a tile with one bulk copy. The expansion is scratch of one layer's call, 520 bytes a token
// and kv head; it is written and read through L2 (4096 tokens, 8 heads: 17 MB, 8 us with cold caches).
//
// tq_prefill_tile_kernel: a CTA takes 32 query tokens of one kv head = 128 rows (token, GQA head) and a range of
// 128-key tiles. Both rotations are part of it:
//   before   Q' = q Pi_K^T on the tensor cores (q is exact in fp16, Pi_K in two fp16 parts), scaled, split into high and low
//            fp16 parts, which are the A operand of the scores
//   loop     S = Q'_h K^T + Q'_l K^T; a thread a row: key norm, mask, maximum, exponential, value norm; O += P V with P in
//            tensor memory over its own scores
//   after    (where the CTA saw all keys) O / l in two fp16 parts times Pi_V, fp16 out; else the partial result, which
//            tq_rot_rows_kernel<false> merges
// Even and odd tiles are two streams with a score buffer, a running maximum and an accumulator of their own (4 x 128
// columns: all of tensor memory), so that the products of one run under the exponentials of the other; the streams
// are added up at the end. A tile is 1536 tensor cycles (scores count twice), 1024 of ex2 and about 700 issue slots.
// 512 tokens (8 kv heads) at position 0 / after 3584: 47.8 / 176.1 us with the page-walking kernel and its two rotation
// launches, 20.2 / 62.9 here; 4096 tokens at 0: 1057 -> 241; 16 after 8000: 82.7 -> 46.4; 200 after 100: 44.3 -> 18.9.
// 128 keys, because at N = 64 the A operand's reads alone would exceed what shared memory delivers.

constexpr int kPtKeys = 128;                                // keys of a tile
constexpr int kPtTokens = 32;                               // query tokens of a CTA
constexpr int kPtThreads = 320;                             // two streams of 128 row threads, issuing warp, copying warp
constexpr uint32_t kPtK = umma::kTileBytes;                 // record of a key tile
constexpr uint32_t kPtV = umma::kTileBytes + 2 * kPtKeys * 4;       // of a value tile, with the key and value norms of its tokens
constexpr size_t kPtSmemBytes = 2 * (size_t)umma::kTileBytes + 2 * (size_t)kPtK + 2 * (size_t)kPtV + 1024;
constexpr float kPtSlack = 8.0f;

struct ExpandParams {
    const uint8_t* pool;
    int n_pages, H;
    const int32_t* seq_pages;
    int n_tokens, n_tiles;
    uint32_t tl0, tl1, th0, th1;
    float inv_alpha;
    const float* Pi_k;
    const float* Pi_v;
    uint8_t* records;          // [kv head][tile][K | V]
    uint8_t* images;           // B operands of the rotations: Pi_K high, low, Pi_V high, low
    int* status;
};

// One CTA = the eight pages of a tile of one kv head, a warp a page; the last row of the grid writes the rotations.
__global__ void __launch_bounds__(256) tq_expand_kernel(const ExpandParams p) {
    pdl_begin();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.y == (unsigned)p.H) {
        // rows 16 x + 2 warp .. of both images: lane = (row, 8 k)
        if (blockIdx.x >= 8) return;
        const int n = 16 * blockIdx.x + 2 * warp + (lane & 1), k8 = lane >> 1;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            uint32_t h[4], l[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float x[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int k = 8 * k8 + 2 * e + i;
                    x[i] = which == 0 ? __ldg(p.Pi_k + n * kDim + k) : __ldg(p.Pi_v + k * kDim + n);
                }
                const __half2 hh = __floats2half2_rn(x[0], x[1]);
                const float2 hf = __half22float2(hh);
                const __half2 ll = __floats2half2_rn(x[0] - hf.x, x[1] - hf.y);
                h[e] = *reinterpret_cast<const uint32_t*>(&hh);
                l[e] = *reinterpret_cast<const uint32_t*>(&ll);
            }
            uint8_t* to = p.images + (size_t)which * 2 * umma::kTileBytes + umma::offset(n, k8);
            *reinterpret_cast<uint4*>(to) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4*>(to + umma::kTileBytes) = make_uint4(l[0], l[1], l[2], l[3]);
        }
        return;
    }
    const int tile = blockIdx.x, h = blockIdx.y;
    if (tile >= p.n_tiles) return;
    uint8_t* rec_k = p.records + ((size_t)h * p.n_tiles + tile) * (kPtK + kPtV);
    uint8_t* rec_v = rec_k + kPtK;
    const int page_ord = tile * (kPtKeys / kPage) + warp, valid = p.n_tokens - page_ord * kPage;
    int id = -1;
    if (valid > 0) {
        id = p.seq_pages[page_ord];
        if (id < 0 || id >= p.n_pages) {
            if (lane == 0) atomicOr(p.status, kStatusBadPage);
            id = -1;
        }
    }
    const size_t kv_stride = (size_t)p.H * kChunkBytes;
    const uint8_t* chunk = p.pool + ((size_t)(id < 0 ? 0 : id) * 2 * p.H + h) * kChunkBytes;
    auto values = [&](const uint8_t* c, int ui, uint32_t (&h2)[16]) {
        uint32_t w[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) w[i] = id < 0 ? 0u : __ldg(reinterpret_cast<const uint32_t*>(c) + 64 * i + ui);
        const uint32_t sel[4] = {w[0] & 0x77777777u, w[1] & 0x77777777u, w[2] & 0x77777777u,
                                 ((w[0] >> 3) & 0x11111111u) | ((w[1] >> 2) & 0x22222222u) | ((w[2] >> 1) & 0x44444444u)};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t sa = sel[q], sb = sa >> 16;
            const uint32_t la = __byte_perm(p.tl0, p.tl1, sa), ha = __byte_perm(p.th0, p.th1, sa);
            const uint32_t lb = __byte_perm(p.tl0, p.tl1, sb), hb = __byte_perm(p.th0, p.th1, sb);
            h2[4 * q + 0] = __byte_perm(la, ha, 0x5140);
            h2[4 * q + 1] = __byte_perm(la, ha, 0x7362);
            h2[4 * q + 2] = __byte_perm(lb, hb, 0x5140);
            h2[4 * q + 3] = __byte_perm(lb, hb, 0x7362);
        }
    };
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        // keys: quarter kq of token lane & 15; eight lanes fill a core matrix
        uint32_t h2[16];
        const int ktok = lane & 15, kq = (lane >> 4) + 2 * i;
        values(chunk, 4 * ktok + kq, h2);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            *reinterpret_cast<uint4*>(rec_k + umma::offset(16 * warp + ktok, 4 * kq + q)) =
                make_uint4(h2[4 * q], h2[4 * q + 1], h2[4 * q + 2], h2[4 * q + 3]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        // values: register c of unit (group, pair) holds coordinate 16 group + c of two tokens; a 4 x 4 transpose between the
        // four lanes of a group leaves each with eight tokens of a coordinate
        uint32_t h2[16];
        values(chunk + kv_stride, lane + 32 * i, h2);
        const int grp = lane >> 2, pl = lane & 3;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t* a = h2 + 4 * j;
#pragma unroll
            for (int c = 0; c < 4; c += 2) {
                const uint32_t send = (pl & 1) ? a[c] : a[c + 1];
                const uint32_t got = __shfl_xor_sync(0xffffffffu, send, 1);
                if (pl & 1) a[c] = got; else a[c + 1] = got;
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint32_t send = (pl & 2) ? a[c] : a[c + 2];
                const uint32_t got = __shfl_xor_sync(0xffffffffu, send, 2);
                if (pl & 2) a[c] = got; else a[c + 2] = got;
            }
            *reinterpret_cast<uint4*>(rec_v + umma::offset(16 * grp + 4 * j + pl, 2 * warp + i)) = make_uint4(a[0], a[1], a[2], a[3]);
        }
    }
    // norms (times 1 / alpha) of this page's tokens; 0 for a token that is not there
    const int tok = lane & 15;
    const uint8_t* src = chunk + (lane < 16 ? 0 : kv_stride) + kNormOffsetBytes;
    const float n = id >= 0 && tok < valid ? __half2float(reinterpret_cast<const __half*>(src)[tok]) * p.inv_alpha : 0.f;
    reinterpret_cast<float*>(rec_v + umma::kTileBytes)[(lane < 16 ? 0 : kPtKeys) + 16 * warp + tok] = n;
}

struct TileAttnParams {
    const __half* q;
    long long q_token, q_head; // elements from a token / a head of q to the next
    float qscale;              // softmax scale * log2(e)
    const uint8_t* records;
    const uint8_t* images;
    __half* out;               // [T][Hq][128], or
    float* o_part;             // [n_splits][T][Hq][128] and
    float* ml_part;            // [n_splits][T][Hq][2]
    int n_splits, H, T, start_pos, n_tiles;
    int* status;
};

struct PtTwo { float x, y; };
__device__ __forceinline__ PtTwo pt_mul2(PtTwo a, PtTwo b) {
    PtTwo d;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ PtTwo pt_add2(PtTwo a, PtTwo b) {
    PtTwo d;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
// eight numbers as fp16 high and low parts
__device__ __forceinline__ void pt_split8(const float (&x)[8], uint8_t* hi, uint8_t* lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const __half2 hh = __floats2half2_rn(x[2 * e], x[2 * e + 1]);
        const float2 hf = __half22float2(hh);
        const __half2 ll = __floats2half2_rn(x[2 * e] - hf.x, x[2 * e + 1] - hf.y);
        h[e] = *reinterpret_cast<const uint32_t*>(&hh);
        l[e] = *reinterpret_cast<const uint32_t*>(&ll);
    }
    *reinterpret_cast<uint4*>(hi) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(lo) = make_uint4(l[0], l[1], l[2], l[3]);
}

enum { kPtPiBar, kPtRotBar, kPtKFull, kPtVFull = kPtKFull + 2, kPtS = kPtVFull + 2, kPtP = kPtS + 2, kPtPV = kPtP + 2, kPtBars = kPtPV + 2 };

__global__ void __launch_bounds__(kPtThreads, 1) tq_prefill_tile_kernel(const TileAttnParams p) {
    extern __shared__ __align__(16) uint8_t pt_raw[];
    __shared__ __align__(8) uint64_t s_bar[kPtBars];
    __shared__ uint32_t s_tmem;
    __shared__ float2 s_ml[2][umma::kRows];
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    uint8_t* base = pt_raw + ((1024u - (smem_u32(pt_raw) & 1023u)) & 1023u);
    uint8_t* s_qh = base;                                   // the rows' A operand: q, then Q' high, then O high
    uint8_t* s_ql = s_qh + umma::kTileBytes;                // Pi_K high, then Q' low, then O low
    uint8_t* s_k = s_ql + umma::kTileBytes;                 // two key tiles (Pi_K low in the second, at first); at the end Pi_V
    uint8_t* s_v = s_k + 2 * kPtK;                          // two value tiles with norms
    auto bar = [&](int b) { return smem_u32(&s_bar[b]); };
    // barrier pairs: tile j uses b + (j & 1), in its phase j / 2
    auto wait = [&](int b, int j) { return umma::bar_wait(bar(b + (j & 1)), (uint32_t)((j >> 1) & 1)); };

    if (warp == 8) umma::tmem_alloc_n(smem_u32(&s_tmem), 512);
    if (tid == 0) {
        for (int b = 0; b < kPtBars; ++b) umma::bar_init_n(bar(b), b == kPtP || b == kPtP + 1 ? umma::kRows : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_begin();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    const uint32_t tm_o = tmem, tm_s = tmem + 2 * kDim;     // O of the streams, scores of the streams

    const int Hq = p.H * kGroup, kvh = blockIdx.y;
    const int tile = (int)gridDim.x - 1 - (int)blockIdx.x;                  // the longest first
    const int tok0 = tile * kPtTokens, last_tok = min(tok0 + kPtTokens, p.T) - 1;
    const int n_all = (p.start_pos + last_tok) / kPtKeys + 1;
    const int t0 = (int)((long long)n_all * blockIdx.z / p.n_splits);
    const int n = (int)((long long)n_all * (blockIdx.z + 1) / p.n_splits) - t0;      // tiles of this CTA; may be 0
    const uint8_t* rec = p.records + ((size_t)kvh * p.n_tiles + t0) * (kPtK + kPtV);
    bool ok = true;
    int nk = 0, nv = 0;                                     // tiles that the copying thread has asked for
    auto copy_k = [&](int j) {
        mbar_expect_tx(bar(kPtKFull + (j & 1)), kPtK);
        bulk_g2s(smem_u32(s_k + (j & 1) * kPtK), rec + (size_t)j * (kPtK + kPtV), kPtK, bar(kPtKFull + (j & 1)));
        nk = j + 1;
    };
    auto copy_v = [&](int j) {
        mbar_expect_tx(bar(kPtVFull + (j & 1)), kPtV);
        bulk_g2s(smem_u32(s_v + (j & 1) * kPtV), rec + (size_t)j * (kPtK + kPtV) + kPtK, kPtV, bar(kPtVFull + (j & 1)));
        nv = j + 1;
    };

    // ---- queries: rows (token, head) as they are; then rotated, scaled and split ----
    const int stream = warp >> 2, lane0 = 32 * (warp & 3), row = lane0 + lane;       // of the row threads
    if (warp == 9 && lane == 0) {
        mbar_expect_tx(bar(kPtPiBar), 2 * umma::kTileBytes);
        bulk_g2s(smem_u32(s_ql), p.images, umma::kTileBytes, bar(kPtPiBar));
        bulk_g2s(smem_u32(s_k + kPtK), p.images + umma::kTileBytes, umma::kTileBytes, bar(kPtPiBar));
        if (n > 0) {
            copy_k(0);
            copy_v(0);
        }
        if (n > 1) copy_v(1);
    } else if (warp < 8) {
        // lanes: eight rows of one piece fill a core matrix, four pieces = 64 bytes of a row
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = 8 * (2 * warp + (i & 1)) + (lane & 7), k8 = 4 * (i >> 1) + (lane >> 3);
            const int tok = tok0 + (r >> 2);
            uint4 v = make_uint4(0, 0, 0, 0);
            if (tok < p.T) v = __ldg(reinterpret_cast<const uint4*>(p.q + tok * p.q_token + (kvh * kGroup + (r & 3)) * p.q_head) + k8);
            *reinterpret_cast<uint4*>(s_qh + umma::offset(r, k8)) = v;
        }
    }
    __syncwarp();
    umma::fence_operands();
    __syncthreads();
    // a product over K = 128: D (+)= A . B, all operands blocked K-major
    auto product = [&](uint32_t d, const uint8_t* a, const uint8_t* b, bool first) {
        const uint64_t da = umma::desc(smem_u32(a)), db = umma::desc(smem_u32(b));
#pragma unroll
        for (int ks = 0; ks < kDim / 16; ++ks) {
            const uint64_t off = (uint64_t)ks * (2 * umma::kLbo >> 4);
            umma::mma_f16(d, da + off, db + off, !(first && ks == 0));
        }
    };
    auto all = [&](bool done) { return __all_sync(0xffffffffu, done) != 0; };
    if (warp == 8) {
        ok = all(umma::bar_wait(bar(kPtPiBar), 0));
        if (ok && umma::elect()) {
            product(tm_o, s_qh, s_ql, true);
            product(tm_o, s_qh, s_k + kPtK, false);
            umma::commit(bar(kPtRotBar));
        }
        __syncwarp();
    } else if (warp < 8) {
        ok = all(umma::bar_wait(bar(kPtRotBar), 0));
        if (ok) {
            umma::fence_after_sync();
#pragma unroll
            for (int c0 = 0; c0 < 64; c0 += 32) {
                uint32_t r[32];
                umma::ld32(r, tm_o, lane0, 64 * stream + c0);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float x[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(r[8 * c + e]) * p.qscale;
                    const uint32_t at = umma::offset(row, 8 * stream + c0 / 8 + c);
                    pt_split8(x, s_qh + at, s_ql + at);
                }
            }
        }
    }
    umma::fence_operands();
    umma::fence_before_sync();
    ok = !__syncthreads_or(!ok);
    umma::fence_after_sync();

    const bool whole = p.n_splits == 1;
    // the copies in flight at the end of the copying thread's work land before the block can leave
    auto landed = [&] {
        for (int j = max(nk - 2, 0); j < nk; ++j) wait(kPtKFull, j);
        for (int j = max(nv - 2, 0); j < nv; ++j) wait(kPtVFull, j);
    };
    if (!ok) {
        if (warp == 9 && lane == 0) {
            umma::bar_wait(bar(kPtPiBar), 0);
            landed();
        }
    } else if (warp == 9) {
        // ---- copies ----
        if (lane == 0) {
            if (n > 1) copy_k(1);
            for (int j = 2; j < n && ok; ++j) {
                ok = wait(kPtS, j - 2);
                if (!ok) break;
                copy_k(j);
                ok = wait(kPtPV, j - 2);
                if (!ok) break;
                copy_v(j);
            }
            // Pi_V over the key tiles, once the last scores are done
            if (ok && whole) {
                if (n > 1) ok = wait(kPtS, n - 2);
                ok = ok && wait(kPtS, n - 1);
                if (ok) {
                    mbar_expect_tx(bar(kPtPiBar), 2 * umma::kTileBytes);
                    bulk_g2s(smem_u32(s_k), p.images + 2 * umma::kTileBytes, 2 * umma::kTileBytes, bar(kPtPiBar));
                    ok = umma::bar_wait(bar(kPtPiBar), 1);
                }
            }
            landed();
        }
    } else if (warp == 8) {
        // ---- products ----
        auto scores = [&](int j) {
            ok = all(wait(kPtKFull, j));
            if (!ok) return;
            umma::fence_after_sync();
            if (umma::elect()) {
                const uint8_t* k = s_k + (j & 1) * kPtK;
                product(tm_s + (j & 1) * kPtKeys, s_ql, k, true);
                product(tm_s + (j & 1) * kPtKeys, s_qh, k, false);
                umma::commit(bar(kPtS + (j & 1)));
            }
            __syncwarp();
        };
        for (int j = 0; j < min(2, n) && ok; ++j) scores(j);
        for (int j = 0; j < n && ok; ++j) {
            ok = all(wait(kPtVFull, j)) && all(wait(kPtP, j));
            if (!ok) break;
            umma::fence_after_sync();
            if (umma::elect()) {
                const uint64_t dv = umma::desc(smem_u32(s_v + (j & 1) * kPtV));
#pragma unroll
                for (int ks = 0; ks < kPtKeys / 16; ++ks)
                    umma::mma_f16_ts(tm_o + (j & 1) * kDim, tm_s + (j & 1) * kPtKeys + 8 * ks,
                                     dv + (uint64_t)ks * (2 * umma::kLbo >> 4), umma::kIdesc, j > 1 || ks > 0);
                umma::commit(bar(kPtPV + (j & 1)));
            }
            __syncwarp();
            if (j + 2 < n) {                                 // its scores go over these weights
                ok = all(wait(kPtPV, j));
                if (ok) scores(j + 2);
            }
        }
    } else {
        // ---- rows ----
        const int qpos = p.start_pos + tok0 + (row >> 2);
        float m = kNoRef, l = 0.f;
        for (int j = stream; j < n; j += 2) {
            ok = all(wait(kPtVFull, j) && wait(kPtS, j));
            if (!ok) break;
            umma::fence_after_sync();
            const uint32_t tm = tm_s + stream * kPtKeys;
            uint32_t s[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) umma::ld32_async(s[c], tm, lane0, 32 * c);
            const float4* kn = reinterpret_cast<const float4*>(s_v + stream * kPtV + umma::kTileBytes);
            const float4* vn = kn + kPtKeys / 4;
            umma::settle(s[0]);
            umma::settled(s[1]);
            umma::settled(s[2]);
            umma::settled(s[3]);
            float top[4] = {kNoRef, kNoRef, kNoRef, kNoRef};
            const int k1 = qpos - (t0 + j) * kPtKeys;        // the row's last key of the tile
            const bool cut = __any_sync(0xffffffffu, k1 < kPtKeys - 1);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
#pragma unroll
                for (int x = 0; x < 32; x += 4) {
                    const float4 w = kn[8 * c + x / 4];
                    const PtTwo a = pt_mul2({__uint_as_float(s[c][x]), __uint_as_float(s[c][x + 1])}, {w.x, w.y});
                    const PtTwo b = pt_mul2({__uint_as_float(s[c][x + 2]), __uint_as_float(s[c][x + 3])}, {w.z, w.w});
                    float v[4] = {a.x, a.y, b.x, b.y};
                    if (cut) {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (32 * c + x + e > k1) v[e] = -INFINITY;
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        s[c][x + e] = __float_as_uint(v[e]);
                        top[e] = fmaxf(top[e], v[e]);
                    }
                }
            }
            const float best = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
            const bool raise = best > m + kPtSlack;
            if (__any_sync(0xffffffffu, raise)) {
                // nothing is being added to this stream's outputs: these scores were asked for after the last value product
                const float mn = raise ? best : m, f = ex2_approx(m - mn);
                m = mn;
                l *= f;
                if (j > 1) {
#pragma unroll 1
                    for (int c = 0; c < kDim; c += 32) {
                        uint32_t o[32];
                        umma::ld32(o, tm_o + stream * kDim, lane0, c);
#pragma unroll
                        for (int x = 0; x < 32; ++x) o[x] = __float_as_uint(__uint_as_float(o[x]) * f);
                        umma::st32(o, tm_o + stream * kDim, lane0, c);
                    }
                }
            }
            PtTwo sum[2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t w16[16];
#pragma unroll
                for (int x = 0; x < 32; x += 4) {
                    const float4 w = vn[8 * c + x / 4];
                    PtTwo a = pt_add2({__uint_as_float(s[c][x]), __uint_as_float(s[c][x + 1])}, {-m, -m});
                    PtTwo b = pt_add2({__uint_as_float(s[c][x + 2]), __uint_as_float(s[c][x + 3])}, {-m, -m});
                    a = {ex2_approx(a.x), ex2_approx(a.y)};
                    b = {ex2_approx(b.x), ex2_approx(b.y)};
                    sum[0] = pt_add2(sum[0], a);
                    sum[1] = pt_add2(sum[1], b);
                    a = pt_mul2(a, {w.x, w.y});
                    b = pt_mul2(b, {w.z, w.w});
                    w16[x / 2] = pack_h2(a.x, a.y);
                    w16[x / 2 + 1] = pack_h2(b.x, b.y);
                }
                umma::st16_async(w16, tm, lane0, 16 * c);
            }
            l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
            umma::stored();
            umma::fence_before_sync();
            umma::bar_arrive(bar(kPtP + stream));
        }
        // this stream's last value products (a barrier of the other stream may be a phase behind)
        const int last = n - 1 - ((n - 1 - stream) & 1);
        if (ok && last >= stream) ok = all(wait(kPtPV, last));
        umma::fence_after_sync();
        s_ml[stream][row] = make_float2(m, l);
    }
    __syncwarp();
    umma::fence_before_sync();
    ok = !__syncthreads_or(!ok);
    umma::fence_after_sync();

    if (ok && warp < 8) {
        // ---- the streams added up; a thread has a row and half its coordinates ----
        const float2 a = s_ml[0][row], b = s_ml[1][row];
        const float m = fmaxf(a.x, b.x);
        const float fa = ex2_approx(a.x - m), fb = ex2_approx(b.x - m), l = a.y * fa + b.y * fb;
        const int tok = tok0 + (row >> 2);
        const size_t v = (size_t)tok * Hq + kvh * kGroup + (row & 3), n_vec = (size_t)p.T * Hq;
        const float inv = whole ? (l > 0.f ? 1.f / l : 0.f) : 1.f;
#pragma unroll
        for (int c0 = 0; c0 < 64; c0 += 32) {
            uint32_t x[32], y[32];
            if (n > 0) umma::ld32(x, tm_o, lane0, 64 * stream + c0);
            if (n > 1) umma::ld32(y, tm_o + kDim, lane0, 64 * stream + c0);
            float o[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                o[i] = n > 0 ? __uint_as_float(x[i]) * fa : 0.f;
                if (n > 1) o[i] = fmaf(__uint_as_float(y[i]), fb, o[i]);
                o[i] *= inv;
            }
            if (whole) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float w[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) w[e] = o[8 * c + e];
                    const uint32_t at = umma::offset(row, 8 * stream + c0 / 8 + c);
                    pt_split8(w, s_qh + at, s_ql + at);
                }
            } else if (tok < p.T) {
                float4* dst = reinterpret_cast<float4*>(p.o_part + ((size_t)blockIdx.z * n_vec + v) * kDim + 64 * stream + c0);
#pragma unroll
                for (int q = 0; q < 8; ++q) dst[q] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
            }
        }
        if (!whole && stream == 0 && tok < p.T)
            *reinterpret_cast<float2*>(p.ml_part + ((size_t)blockIdx.z * n_vec + v) * 2) = make_float2(m, l);
    }
    if (whole) {
        umma::fence_operands();
        umma::fence_before_sync();
        __syncthreads();
        umma::fence_after_sync();
        if (ok && warp == 8) {
            ok = all(umma::bar_wait(bar(kPtPiBar), 1));
            if (ok && umma::elect()) {
                product(tm_s, s_ql, s_k, true);
                product(tm_s, s_qh, s_k + umma::kTileBytes, false);
                product(tm_s, s_qh, s_k, false);
                umma::commit(bar(kPtRotBar));
            }
            __syncwarp();
        } else if (ok && warp < 8) {
            ok = all(umma::bar_wait(bar(kPtRotBar), 1));
            if (ok) {
                umma::fence_after_sync();
                const int tok = tok0 + (row >> 2);
                __half* dst = p.out + ((size_t)min(tok, p.T - 1) * Hq + kvh * kGroup + (row & 3)) * kDim + 64 * stream;
#pragma unroll
                for (int c0 = 0; c0 < 64; c0 += 32) {
                    uint32_t r[32];
                    umma::ld32(r, tm_s, lane0, 64 * stream + c0);
                    if (tok < p.T) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t w[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) w[e] = pack_h2(__uint_as_float(r[8 * q + 2 * e]), __uint_as_float(r[8 * q + 2 * e + 1]));
                            *reinterpret_cast<uint4*>(dst + c0 + 8 * q) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
            }
        }
    }
    if (!ok && lane == 0) atomicOr(p.status, kStatusWaitTimeout);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 8) {
        umma::fence_after_sync();
        umma::tmem_free_n(tmem, 512);
    }
}
