// Multi-token pool append with the rotation on tensor cores (included by tq_quantize.cu inside
// namespace leankv::{anonymous}).
//
// The arithmetic contract of this file's header still holds bit for bit: a code is defined by the
// sequential fp32 fma chain y_j = fma(Pi[j][k], u[k], y_j), k ascending. Tensor cores cannot run
// that chain, so the rotation is done twice over:
//   1. fast: u and Pi are split into fp16 high and low parts (x = hi + lo, |lo| <= 2^-11 |hi|) and
//      y ~ Pi_hi u_hi + Pi_hi u_lo + Pi_lo u_hi on m16n8k16 MMAs with fp32 accumulation. The result
//      differs from the chain's value by less than the band: kBand, widened where rows of Pi are longer than 1;
//   2. exact: a coordinate whose fast value lies within the band around a decision boundary (one per
//      thousand) is recomputed with the sequential chain from the fp32 unit vector kept in shared
//      memory, and that value decides the code.
// Every other coordinate is farther from all boundaries than the fast path's error, so its code is
// the chain's code. The fp32 kernels above remain the definition; tests compare whole pools.
//
// A CTA of 8 warps quantizes tiles of 64 tokens (4 pages, two warps each: half the coordinates a warp) of one
// (sequence, head, K|V); CTAs are persistent over a contiguous range of tiles and keep the fp16 copies of Pi in
// shared memory, reloading them only when their range crosses from K to V.
//
// A prompt chunk is one tile a CTA, so its time is the chain of a tile's phases, none of which fills the issue slots. 512 tokens of 8
// heads, cycles: indexes and positions 2000, staging Pi 2000 (3600 from HBM), norms 850, division 2100, band 650, products 3700 (the rate of
// mma.sync), codes 2000, exact chains 2500, packing 1450: 11.0 us (13.1 with a rotation that is not in L2). With one warp a page
// they took 24, with Pi staged by 8-byte loads, four in flight, 12.4 (16.4); 16 sequences of 2048 tokens 329, now 301 (tiles without a
// token are left out, rows without one not divided).

constexpr int kTcThreads = 256;
constexpr int kTcTokens = 64;
constexpr int kPiStride = 136;            // halves per row (272 bytes): conflict-free 8 x 16-byte ldmatrix rows
constexpr int kUStride = 136;             // floats per row of the unit-vector tile
// Where rows of Pi and unit vectors have norm 1, sums over k of |Pi u| are at most 1: the chain's own rounding is at most
// 128 x 2^-24 = 7.6e-6, the fast value's (splits and fp16's subnormals 1.2e-6, the dropped lo x lo 2.4e-7, 24 accumulations
// of two units in the last place each 5.7e-6) 7.2e-6. All of these grow with the norm of a row of Pi, so the band does too:
// band_for takes the squared norm of half a row's high parts from each thread (two neighbours share a row) and
// returns kBand times the longest row's norm, at least kBand; infinite, and so every coordinate exact, where a sum of squares
// is beyond fp16 (norms above 256 to 724, by how even the row is) or no number. s_top: a number a warp. It runs whenever Pi is staged: 12.1 -> 12.45 us for
// 512 tokens of 8 heads, nothing where a CTA has several tiles (16 sequences of 2048 tokens: 329 -> 326).
constexpr float kBand = 2.5e-5f;
struct HalfRow {
    __half2 sum[2] = {__floats2half2_rn(0.f, 0.f), __floats2half2_rn(0.f, 0.f)};
    __device__ __forceinline__ void add(const uint4& w) {       // each sum is rounded sixteen times: 1 % at most
        const __half2* h = reinterpret_cast<const __half2*>(&w);
        sum[0] = __hfma2(h[0], h[0], sum[0]);
        sum[1] = __hfma2(h[1], h[1], sum[1]);
        sum[0] = __hfma2(h[2], h[2], sum[0]);
        sum[1] = __hfma2(h[3], h[3], sum[1]);
    }
    __device__ __forceinline__ float total() const {
        const float2 a = __half22float2(sum[0]), b = __half22float2(sum[1]);
        return (a.x + a.y) + (b.x + b.y);
    }
};
template <int kWarps>
__device__ __forceinline__ float band_for(float half_row, float* s_top) {
    const float row = half_row + __shfl_xor_sync(0xffffffffu, half_row, 1);
    // bits of numbers that are not negative order as the numbers do, and a NaN above all of them
    const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(row) & 0x7fffffffu);
    if ((threadIdx.x & 31) == 0) s_top[threadIdx.x >> 5] = __uint_as_float(top);
    __syncthreads();
    unsigned all = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) all = max(all, __float_as_uint(s_top[w]));
    const float norm = 1.01f * sqrtf(__uint_as_float(all));           // half of that 1 %, and the low parts' 2^-11
    return norm < 1e30f ? kBand * fmaxf(norm, 1.f) : __int_as_float(0x7f800000);
}
constexpr int kCodeStride = 132;          // bytes per token row of the code tile: 4-byte reads of 8 tokens x 4 quarters hit 32 banks
constexpr int kListCap = 64;              // queue of boundary-band coordinates: flushed whenever it holds a full warp's worth
constexpr size_t kTcSmemBytes = 2 * (size_t)kDim * kPiStride * sizeof(__half) +
                                (size_t)kTcTokens * kUStride * sizeof(float) + (size_t)kTcTokens * kCodeStride;

struct AppendTcParams {
    AppendParams a;
    int groups;                       // 4-page groups per (sequence, head, K|V)
    long long n_tiles;
    unsigned long long* stats;        // [0] += coordinates recomputed exactly, [1] += coordinates quantized (may be null)
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void mma_f16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// hi = fp16(x) for both elements, lo = fp16(x - hi)
__device__ __forceinline__ void split_h2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x0, x1);
    const float2 hf = __half22float2(h);
    const __half2 l = __floats2half2_rn(x0 - hf.x, x1 - hf.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

__global__ void __launch_bounds__(kTcThreads, 2) tq_pool_append_tc_kernel(const AppendTcParams tp) {
    extern __shared__ __align__(16) unsigned char tc_smem[];
    __half* s_pih = reinterpret_cast<__half*>(tc_smem);
    __half* s_pil = s_pih + kDim * kPiStride;
    float* s_u = reinterpret_cast<float*>(s_pil + kDim * kPiStride);                 // [64][kUStride]
    uint8_t* s_code = reinterpret_cast<uint8_t*>(s_u + kTcTokens * kUStride);        // [64][kCodeStride]
    __shared__ float s_norm[kTcTokens];
    __shared__ uint16_t s_list[kTcThreads / 32][kListCap];      // per warp: (slot << 7 | coordinate) awaiting the exact chain
    __shared__ float s_bounds[8];
    __shared__ float s_top[kTcThreads / 32];

    const AppendParams& p = tp.a;
    pdl_begin();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int pgw = warp >> 1, side = warp & 1;           // page of the tile, half of the coordinates
    if (tid < 8) s_bounds[tid] = tid < 7 ? p.bounds[tid] : __int_as_float(0x7f800000);

    const long long tile_lo = (long long)blockIdx.x * tp.n_tiles / gridDim.x;
    const long long tile_hi = ((long long)blockIdx.x + 1) * tp.n_tiles / gridDim.x;
    const long long per_which = (long long)p.B * p.H * tp.groups;
    int loaded_which = -1;
    float band = 0.f;
    unsigned long long n_exact = 0, n_coords = 0;

    for (long long tile = tile_lo; tile < tile_hi; ++tile) {
        const int which = tile < per_which ? 0 : 1;
        const unsigned r = (unsigned)(tile - (which ? per_which : 0));       // the grid's tiles of a side fit 32 bits
        const unsigned r2 = r / (unsigned)tp.groups, grp = r - r2 * (unsigned)tp.groups;
        const int b = (int)(r2 / (unsigned)p.H), h = (int)(r2 - (unsigned)b * (unsigned)p.H);
        const float* Pi = which == 0 ? p.Pi_k : p.Pi_v;

        const int pos0 = p.start_pos[b];
        const int ord0 = pos0 / 16 + 4 * (int)grp;            // first page ordinal of this tile
        const int pos_end = pos0 + p.T_new;
        if (ord0 * 16 >= pos_end) continue;                   // one group more than needed where the start is a page's
        const __half* src = append_source(p, which, b, h);

        __syncthreads();                 // the previous tile's readers of s_u / s_pi* are done
        // the tile's vectors are asked for ahead of Pi, and Pi in two trips of eight 16-byte loads a thread
        const int row = tid >> 2, qr = tid & 3;               // four threads per token, 32 coordinates each
        const int pos = ord0 * 16 + row;
        uint4 raw[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            raw[i] = pos >= pos0 && pos < pos_end
                         ? __ldg(reinterpret_cast<const uint4*>(src + (size_t)(pos - pos0) * kDim + qr * 32) + i)
                         : make_uint4(0, 0, 0, 0);
        const bool staged = which != loaded_which;
        if (staged) {
            constexpr int kTrip = 8;
            static_assert(kDim * kDim / 4 == 2 * kTrip * kTcThreads, "two trips");
#pragma unroll 1
            for (int i0 = tid; i0 < kDim * kDim / 4; i0 += kTrip * kTcThreads) {
                float4 v[kTrip];
#pragma unroll
                for (int x = 0; x < kTrip; ++x) v[x] = __ldg(reinterpret_cast<const float4*>(Pi) + i0 + x * kTcThreads);
#pragma unroll
                for (int x = 0; x < kTrip; ++x) {
                    const int i = i0 + x * kTcThreads, at = (i >> 5) * kPiStride + (i & 31) * 4;
                    uint2 hi, lo;
                    split_h2(v[x].x, v[x].y, hi.x, lo.x);
                    split_h2(v[x].z, v[x].w, hi.y, lo.y);
                    *reinterpret_cast<uint2*>(&s_pih[at]) = hi;
                    *reinterpret_cast<uint2*>(&s_pil[at]) = lo;
                }
            }
            loaded_which = which;
        }

        // ---- norms and unit vectors. The norm is the contract's: the squares of
        // each half one after another, so the second thread of a half goes on from the first one's sum ----
        {
            float xr[32];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 a = h2_to_f2(raw[i].x), bb = h2_to_f2(raw[i].y), c = h2_to_f2(raw[i].z), d = h2_to_f2(raw[i].w);
                xr[8 * i + 0] = a.x; xr[8 * i + 1] = a.y; xr[8 * i + 2] = bb.x; xr[8 * i + 3] = bb.y;
                xr[8 * i + 4] = c.x; xr[8 * i + 5] = c.y; xr[8 * i + 6] = d.x; xr[8 * i + 7] = d.y;
            }
            double sum = 0.0;
#pragma unroll
            for (int i = 0; i < 32; ++i) sum = fma((double)xr[i], (double)xr[i], sum);
            const double before = __shfl_up_sync(0xffffffffu, sum, 1);
            if (qr & 1) {
                sum = before;
#pragma unroll
                for (int i = 0; i < 32; ++i) sum = fma((double)xr[i], (double)xr[i], sum);
            }
            const int l0 = lane & ~3;
            const double tot = __shfl_sync(0xffffffffu, sum, l0 + 1) + __shfl_sync(0xffffffffu, sum, l0 + 3);
            const float norm = (float)sqrt(tot);
            const float denom = norm + 1e-10f;
            if (qr == 0) s_norm[row] = norm;
            float4* dst = reinterpret_cast<float4*>(&s_u[row * kUStride + qr * 32]);
            if (norm > 0.f) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    dst[i] = make_float4(xr[4 * i] / denom, xr[4 * i + 1] / denom, xr[4 * i + 2] / denom, xr[4 * i + 3] / denom);
            } else {      // no token or a zero vector (whose division by 1e-10 takes 9400 cycles a tile), or no numbers
#pragma unroll
                for (int i = 0; i < 8; ++i) dst[i] = norm == 0.f ? make_float4(xr[4 * i], xr[4 * i + 1], xr[4 * i + 2], xr[4 * i + 3])
                                                                 : make_float4(norm, norm, norm, norm);
            }
        }
        __syncthreads();
        if (staged) {
            const uint4* half = reinterpret_cast<const uint4*>(s_pih + (tid >> 1) * kPiStride + 64 * (tid & 1));
            HalfRow row;
#pragma unroll
            for (int i = 0; i < 8; ++i) row.add(half[i ^ (4 * (tid & 1))]);       // eight threads' reads in 32 banks
            band = band_for<kTcThreads / 32>(row.total(), s_top);
        }

        // ---- this warp's page ----
        const int page_ord = ord0 + pgw;
        const int first = max(pos0, page_ord * 16), last = min(pos_end, page_ord * 16 + 16);
        const int nt_valid = last - first;                    // tokens of this launch in the page
        if (nt_valid <= 0) continue;                          // the same in both warps of the page; CTA-wide syncs are above
        const int slot0 = first - page_ord * 16;
        const int page = p.kv_page_indices[p.kv_indptr[b] + page_ord];
        const bool page_ok = page >= 0 && page < p.n_pages;

        // ---- fast rotation on tensor cores: rows = the page's 16 token slots, columns = coordinates ----
        float acc[8][4];                                      // columns 64 side + 8 n ..
#pragma unroll
        for (int n = 0; n < 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
        const float* u_lo_row = &s_u[(16 * pgw + g) * kUStride];
        const float* u_hi_row = u_lo_row + 8 * kUStride;
        const uint32_t pi_addr = (uint32_t)__cvta_generic_to_shared((lane < 16 ? s_pih : s_pil)) +
                                 (uint32_t)(((64 * side + (lane & 7)) * kPiStride + ((lane >> 3) & 1) * 8) * sizeof(__half));
#pragma unroll 1
        for (int ks = 0; ks < 8; ++ks) {
            uint32_t ah[4], al[4];
            {
                const float2 v0 = *reinterpret_cast<const float2*>(u_lo_row + ks * 16 + 2 * t);
                const float2 v1 = *reinterpret_cast<const float2*>(u_hi_row + ks * 16 + 2 * t);
                const float2 v2 = *reinterpret_cast<const float2*>(u_lo_row + ks * 16 + 8 + 2 * t);
                const float2 v3 = *reinterpret_cast<const float2*>(u_hi_row + ks * 16 + 8 + 2 * t);
                split_h2(v0.x, v0.y, ah[0], al[0]);
                split_h2(v1.x, v1.y, ah[1], al[1]);
                split_h2(v2.x, v2.y, ah[2], al[2]);
                split_h2(v3.x, v3.y, ah[3], al[3]);
            }
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                uint32_t bh0, bh1, bl0, bl1;
                ldmatrix_x4(bh0, bh1, bl0, bl1, pi_addr + (uint32_t)((n * 8 * kPiStride + ks * 16) * sizeof(__half)));
                mma_f16_16816(acc[n], al, bh0, bh1);
                mma_f16_16816(acc[n], ah, bl0, bl1);
                mma_f16_16816(acc[n], ah, bh0, bh1);
            }
        }

        // ---- codes; coordinates close to a boundary are queued for the sequential fp32 chain ----
        const float b1 = s_bounds[4], b2 = s_bounds[5], b3 = s_bounds[6];       // 0 < b1 < b2 < b3 (s_bounds[3] = 0)
        uint8_t* code_rows = s_code + (size_t)(16 * pgw) * kCodeStride;
        // exact value of one coordinate: y = fma chain over k ascending, from the fp32 unit vector
        auto exact_code = [&](int slot, int coord) -> int {
            const float4* pr = reinterpret_cast<const float4*>(Pi + (size_t)coord * kDim);
            const float4* ur = reinterpret_cast<const float4*>(&s_u[(16 * pgw + slot) * kUStride]);
            float ye = 0.f;
#pragma unroll
            for (int part = 0; part < 2; ++part) {                               // two round trips for the row
                float4 pv[kDim / 8];
#pragma unroll
                for (int k4 = 0; k4 < kDim / 8; ++k4) pv[k4] = __ldg(pr + part * (kDim / 8) + k4);
#pragma unroll
                for (int k4 = 0; k4 < kDim / 8; ++k4) {
                    const float4 uv = ur[part * (kDim / 8) + k4];
                    ye = fmaf(pv[k4].x, uv.x, ye);
                    ye = fmaf(pv[k4].y, uv.y, ye);
                    ye = fmaf(pv[k4].z, uv.z, ye);
                    ye = fmaf(pv[k4].w, uv.w, ye);
                }
            }
            int code = 0;
#pragma unroll
            for (int q = 0; q < 7; ++q) code += (ye > s_bounds[q]) ? 1 : 0;
            return code;
        };
        uint32_t near = 0;                                     // bit 4n + i: value (n, i) of this lane is in the band
#pragma unroll
        for (int n = 0; n < 8; ++n) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int slot = g + 8 * r;
                const bool mine = slot >= slot0 && slot < slot0 + nt_valid;
                int code[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float y = acc[n][2 * r + c];
                    const float ay = fabsf(y);
                    const int mag = (ay > b1 ? 1 : 0) + (ay > b2 ? 1 : 0) + (ay > b3 ? 1 : 0);
                    code[c] = y > 0.f ? 4 + mag : 3 - mag;
                    const float gap = fminf(fminf(ay, fabsf(ay - b1)), fminf(fabsf(ay - b2), fabsf(ay - b3)));
                    if (!(gap > band) && mine) near |= 1u << (4 * n + 2 * r + c);
                }
                *reinterpret_cast<uint16_t*>(&code_rows[slot * kCodeStride + 64 * side + n * 8 + 2 * t]) =
                    (uint16_t)(code[0] | (code[1] << 8));
            }
        }
        n_coords += (unsigned long long)nt_valid * 2;          // per lane: 64 coordinates / 32 lanes
        n_exact += __popc(near);
        // The band coordinates of all lanes are compacted into a queue; whenever it holds 32 of them every
        // lane runs one exact chain. (A page of all-zero vectors puts all 2048 coordinates in the band.)
        if (const unsigned any = __reduce_or_sync(0xffffffffu, near)) {
            int cnt = 0;                                       // warp-uniform
            auto flush = [&](int n_take) {
                __syncwarp();
                if (lane < n_take) {
                    const int ent = s_list[warp][lane];
                    code_rows[(ent >> 7) * kCodeStride + (ent & 127)] = (uint8_t)exact_code(ent >> 7, ent & 127);
                }
                const int rest = cnt - n_take;                 // < 32
                const uint16_t moved = lane < rest ? s_list[warp][n_take + lane] : (uint16_t)0;
                __syncwarp();
                if (lane < rest) s_list[warp][lane] = moved;
                cnt = rest;
            };
#pragma unroll 1
            for (unsigned left = any; left != 0u; left &= left - 1u) {
                const int idx = __ffs(left) - 1;
                const bool flag = ((near >> idx) & 1u) != 0u;
                const unsigned m = __ballot_sync(0xffffffffu, flag);
                if (flag) {
                    const int n = idx >> 2, i = idx & 3;
                    const int slot = g + (i >> 1) * 8, coord = 64 * side + n * 8 + 2 * t + (i & 1);
                    s_list[warp][cnt + __popc(m & ((1u << lane) - 1u))] = (uint16_t)((slot << 7) | coord);
                }
                cnt += __popc(m);
                if (cnt >= 32) flush(32);
            }
            if (cnt > 0) flush(cnt);
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + pgw) : "memory");       // both halves' codes are there
        if (!page_ok) continue;                                // invalid table entry: write nothing

        // ---- pack this page's chunk (same words as tq_pool_append_kernel), four codes per shared-memory read ----
        uint8_t* chunk = p.pool + (((size_t)page * 2 + which) * p.H + h) * kChunkBytes;
        uint32_t* words = reinterpret_cast<uint32_t*>(chunk);
        __half* norms = reinterpret_cast<__half*>(chunk + kNormOffsetBytes);
        if (side == 0 && lane >= slot0 && lane < slot0 + nt_valid) norms[lane] = __float2half_rn(s_norm[16 * pgw + lane]);
        // squeezes the low nibbles of 4 bytes into 16 bits
        auto pack4 = [](uint32_t v) -> uint32_t {
            const uint32_t t2 = (v | (v >> 4)) & 0x00FF00FFu;
            return (t2 | (t2 >> 8)) & 0xFFFFu;
        };
        for (int w = lane + 32 * side; w < kChunkWords; w += 64) {
            const int kk = w >> 6, ui = w & 63;
            if (which == 0) {
                // unit (slot, quarter t4): codes e = coordinates 32 t4 + e; word kk holds codes 8kk..8kk+7 as
                // nibbles and bit kk of codes 24..31 in the nibbles' spare bits
                const int slot = ui >> 2, t4 = ui & 3;
                if (slot < slot0 || slot >= slot0 + nt_valid) continue;
                const uint32_t* c4 = reinterpret_cast<const uint32_t*>(&code_rows[slot * kCodeStride + 32 * t4]);
                const uint32_t lo = c4[2 * kk] & 0x07070707u, hi = c4[2 * kk + 1] & 0x07070707u;
                const uint32_t s_lo = ((c4[6] >> kk) & 0x01010101u) << 3, s_hi = ((c4[7] >> kk) & 0x01010101u) << 3;
                words[w] = pack4(lo) | (pack4(hi) << 16) | pack4(s_lo) | (pack4(s_hi) << 16);
            } else {
                // unit (pair pr, group gg): coordinates 16 gg .. +15 of slots 2 pr (low nibbles) and 2 pr + 1
                const int pr = ui < 32 ? (ui & 3) : 4 + (ui & 3);
                const int gg = (ui & 31) >> 2;
                const int sa = 2 * pr, sb = sa + 1;
                const bool has_a = sa >= slot0 && sa < slot0 + nt_valid, has_b = sb >= slot0 && sb < slot0 + nt_valid;
                if (!has_a && !has_b) continue;
                const uint32_t* ca = reinterpret_cast<const uint32_t*>(&code_rows[sa * kCodeStride + 16 * gg]);
                const uint32_t* cb = reinterpret_cast<const uint32_t*>(&code_rows[sb * kCodeStride + 16 * gg]);
                uint32_t bits = 0;
                if (has_a) bits |= (ca[kk] & 0x07070707u) | (((ca[3] >> kk) & 0x01010101u) << 3);
                if (has_b) bits |= ((cb[kk] & 0x07070707u) << 4) | (((cb[3] >> kk) & 0x01010101u) << 7);
                if (!(has_a && has_b)) {
                    // the other token of the pair was (or will be) written by another launch
                    const uint32_t keep = has_a ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
                    bits |= words[w] & keep;
                }
                words[w] = bits;
            }
        }
    }
    if (tp.stats != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            n_exact += __shfl_xor_sync(0xffffffffu, n_exact, o);
            n_coords += __shfl_xor_sync(0xffffffffu, n_coords, o);
        }
        if (lane == 0 && n_coords != 0) {
            atomicAdd(tp.stats, n_exact);
            atomicAdd(tp.stats + 1, n_coords);
        }
    }
}
