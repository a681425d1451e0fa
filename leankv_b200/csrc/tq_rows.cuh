// Quantize and de-quantize of many vectors (included by tq_quantize.cu inside namespace leankv::{anonymous}).
//
// Quantize: the rotation is 32 kflop a vector. On the fp32 units (an 8 x 8 register tile, with the norm, the codes and
// the packing of a tile one after another) 65 544 vectors took 159 us where HBM needs 4. Here the products are on the
// tensor cores and the conversions around them are the work. The kernel is persistent, one CTA per SM with three
// roles that meet at mbarriers, so that three consecutive tiles of 128 vectors overlap:
//
//   256 input threads   half a vector each: norm, fp16 high and low parts into the A operand (two buffers)
//   256 result threads  a vector and half its coordinates: accumulator lanes back, codes, packing
//   1 issuing warp      tcgen05.mma, M = N = 128, accumulators in tensor memory (two buffers)
//   3 exact warps       the coordinates that the fast product cannot decide: a tile a warp in turn, a coordinate a lane
//
// The contract of tq_quantize.cu is kept bit for bit as tq_append_tc.cuh does: with x = hi + lo, both fp16, the product
// y ~ P_hi u_hi + P_hi u_lo + P_lo u_hi decides a code unless it lies within kRowsBand of a decision boundary (0.1 % of the
// coordinates), and the sequential fp32 chain decides the rest. A chain is 128 dependent steps, so it runs beside the next
// tiles' work and corrects the stored word (with the chains inside the result warps the kernel took 57.6 us). The norm
// is the contract's fp64 sum; the fast product may take u = x * (1 / denom).
//
// kRowsBand: with rows of Pi and vectors of norm 1, sums over k of |P u| are at most 1. The chain's own rounding is at most
// 128 x 2^-24 = 7.6e-6; the product's: u 2e-7, the splits and fp16's subnormals 1.2e-6, the dropped lo x lo 2.4e-7,
// 24 accumulations of two units in the last place each 5.7e-6. Together 1.5e-5.
//
// De-quantize has no such second look: its result is the fp32 chain, k ascending, so 2^14 multiply-adds a vector on the
// FMA units are its floor (28.8 us for 65 544 vectors at 128 a clock and SM). What it lost was the time between tiles;
// here four warps unpack the next tile while eight run the chains, two vectors an instruction (fma.rn.f32x2 rounds
// each half like fmaf). CTAs take equal ranges of vectors in units of sixteen, so that the last tile of each is short.
//
// 65 544 vectors, fp16 in, fp32 out: quantize 155.5 -> 28.9 us (4.7 us for every 148 tiles, 10 us before the first result:
// staging and the first vectors' norms), de-quantize 77.4 -> 44.8 us (0.73 of the multiply-add rate). 16 vectors: 50.2 ->
// 13.0 and 22.0 -> 10.1 us. fp32 in, 65 544: 159.4 -> 40.9 us.

constexpr int kRowsTile = umma::kRows;                       // vectors of a tile
constexpr int kRowsIn = 256, kRowsOut = 256;                 // threads of the two roles; then the issuing warp
constexpr float kRowsBand = 2.5e-5f;
constexpr int kRowsExact = 96;
constexpr int kRowsThreads = kRowsIn + kRowsOut + 32 + kRowsExact;
constexpr int kRowsStagers = kRowsThreads - kRowsIn;         // the others stage the rotation while the first input is on its way
constexpr uint32_t kRowsTmemCols = 256;
constexpr int kRowsQueue = 512;                              // coordinates of a tile that may be listed for the exact chain
// Norms are kept for 16 tiles. Input writes those of tile j once the products of j - 2 are complete, and these were issued
// once every result thread had read the accumulators of j - 4; it does that before it waits for the list of j - 8 to be
// cleared. So an exact warp may still read norms of tile j - 8 (not of j - 9, whose list the results of j - 5 waited for).
constexpr int kRowsNorms = 16;
constexpr int kRowsStageWords = 9;                           // words of a result row in shared memory (8 and one of padding)
constexpr size_t kRowsSmemBytes = 6 * (size_t)umma::kTileBytes + (size_t)(kRowsOut / 32) * 32 * kRowsStageWords * 4 +
                                  4 * (size_t)kRowsQueue * sizeof(uint16_t);

struct RowsParams {
    const void* x;            // quantize: vectors
    long long n_vec;
    const float* Pi;
    const float* table;       // decision boundaries, or centroids
    uint8_t* indices;
    float* norms;
    void* out;                // de-quantize: vectors
    int out_dtype;
    int wide;                 // indices are 16-byte aligned
    int* status;
};

// The barriers of the two buffers, and the bounded waits on them.
struct RowsBars {
    uint32_t full, done, taken;          // A written; products complete; accumulators read: + 8 for buffer 1
    uint32_t listed, cleared;            // four lists: a tile's words and undecided coordinates written; worked off
    __device__ __forceinline__ bool wait(uint32_t bar, int use) const {      // use-th completion of a buffer's barrier
        return umma::bar_wait(bar, (uint32_t)(use & 1));
    }
};

// two fused multiply-adds, each rounded like fmaf
__device__ __forceinline__ float2 fma_two(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, c, d;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

__device__ __forceinline__ void rows_stagers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kRowsStagers) : "memory"); }

// Stages the rotation as the B operand, high and low parts, scaled by a power of two so that its largest row norm lies
// in [1, 2). Returns that norm; *scale is what it was multiplied by. All stagers call it. `part`: 8 x 128 floats.
// A warp takes 8 rows x 16 columns at a time: whole sectors from memory, half core matrices into shared memory.
__device__ __forceinline__ float stage_rotation(const float* Pi, uint8_t* s_bh, uint8_t* s_bl, float* part, float* s_top,
                                                float* scale) {
    constexpr int kWarps = kRowsStagers / 32, kMine = (128 + kWarps - 1) / kWarps;
    const int t = threadIdx.x - kRowsIn, w = t >> 5, lane = t & 31;
    float4 v[kMine];
#pragma unroll
    for (int m = 0; m < kMine; ++m) {
        const int i = w + m * kWarps, n = 8 * (i >> 3) + (lane & 7), k = 16 * (i & 7) + 4 * (lane >> 3);
        if (i < 128) v[m] = __ldg(reinterpret_cast<const float4*>(Pi + n * kDim + k));
    }
#pragma unroll
    for (int m = 0; m < kMine; ++m) {
        const int i = w + m * kWarps;
        if (i < 128) {
            float ss = fmaf(v[m].x, v[m].x, fmaf(v[m].y, v[m].y, fmaf(v[m].z, v[m].z, v[m].w * v[m].w)));
            ss += __shfl_xor_sync(0xffffffffu, ss, 8);
            ss += __shfl_xor_sync(0xffffffffu, ss, 16);
            if (lane < 8) part[(i & 7) * kDim + 8 * (i >> 3) + lane] = ss;
        }
    }
    rows_stagers_sync();
    if (t < kDim) {
        float ss = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) ss += part[c * kDim + t];
        // a NaN orders above every number here, so that it reaches the result
        const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(ss) & 0x7fffffffu);
        if (lane == 0) s_top[w] = __uint_as_float(top);
    }
    rows_stagers_sync();
    unsigned top = 0;
#pragma unroll
    for (int i = 0; i < kDim / 32; ++i) top = max(top, __float_as_uint(s_top[i]));
    const float norm = sqrtf(__uint_as_float(top));
    const int e = (int)((__float_as_uint(norm) >> 23) & 255u) - 127;
    const float s = __uint_as_float((unsigned)(127 - min(max(e, -50), 50)) << 23);
#pragma unroll
    for (int m = 0; m < kMine; ++m) {
        const int i = w + m * kWarps, n = 8 * (i >> 3) + (lane & 7), k4 = 4 * (i & 7) + (lane >> 3);
        if (i < 128) {
            uint32_t h[2], l[2];
            split_h2(v[m].x * s, v[m].y * s, h[0], l[0]);
            split_h2(v[m].z * s, v[m].w * s, h[1], l[1]);
            const uint32_t at = umma::offset(n, k4 >> 1) + 8u * (k4 & 1);
            *reinterpret_cast<uint2*>(s_bh + at) = make_uint2(h[0], h[1]);
            *reinterpret_cast<uint2*>(s_bl + at) = make_uint2(l[0], l[1]);
        }
    }
    *scale = s;
    return norm;
}

// Barriers, tensor memory, and the end that both kernels share.
struct RowsFrame {
    RowsBars bars;
    uint32_t tmem;
};
__device__ __forceinline__ RowsFrame rows_begin(uint64_t* s_bar, uint32_t* s_tmem) {
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t b0 = umma::smem_addr(s_bar);
    RowsFrame f;
    f.bars.full = b0;
    f.bars.done = b0 + 16;
    f.bars.taken = b0 + 32;
    f.bars.listed = b0 + 48;
    f.bars.cleared = b0 + 80;
    if (warp == kRowsIn / 32) umma::tmem_alloc_n(umma::smem_addr(s_tmem), kRowsTmemCols);
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            umma::bar_init_n(f.bars.full + 8 * i, kRowsIn);
            umma::bar_init_n(f.bars.done + 8 * i, 1);
            umma::bar_init_n(f.bars.taken + 8 * i, kRowsOut);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            umma::bar_init_n(f.bars.listed + 8 * i, kRowsOut);
            umma::bar_init_n(f.bars.cleared + 8 * i, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    return f;
}
// The end, which every thread reaches: whether a wait of this CTA ran out.
__device__ __forceinline__ bool rows_end(const RowsFrame& f, bool ok, int* status) {
    if (!ok) atomicOr(status, 1);
    umma::fence_before_sync();
    const bool failed = __syncthreads_or(!ok) != 0;
    if ((threadIdx.x >> 5) == kRowsIn / 32) {
        umma::fence_after_sync();
        umma::tmem_free_n(f.tmem, kRowsTmemCols);
    }
    return failed;
}
// The issuing warp: `products(buffer)` issues a tile's MMAs from one elected lane.
template <typename Products>
__device__ __forceinline__ bool rows_issue(const RowsFrame& f, int n_mine, Products products) {
    for (int j = 0; j < n_mine; ++j) {
        const int buf = j & 1, use = j >> 1;
        bool ok = f.bars.wait(f.bars.full + 8 * buf, use);
        if (use > 0) ok = ok && f.bars.wait(f.bars.taken + 8 * buf, use - 1);
        if (!__all_sync(0xffffffffu, ok)) return false;
        umma::fence_after_sync();
        if (umma::elect()) {
            products(buf);
            umma::commit(f.bars.done + 8 * buf);
        }
        __syncwarp();
    }
    return true;
}

// a / b, correctly rounded, from inv = 1 / b rounded to nearest: two Newton corrections of the quotient, each with its
// exact remainder (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990: the
// first makes the quotient faithful, the second rounds it correctly). No remainder may underflow: here a is an fp16
// number and b at least its magnitude.
__device__ __forceinline__ float divided(float a, float b, float inv) {
    float q = a * inv;
    q = fmaf(fmaf(-q, b, a), inv, q);
    return fmaf(fmaf(-q, b, a), inv, q);
}

// Code of y by binary search in sorted boundaries; *gap: distance to the nearest one (the boundaries on both sides of
// y are among those it is compared with). kLevel: the bit decided next, of value 1 << kLevel; `at`: boundaries of the
// 1 << (kBits - 1 - kLevel) ranges that are left, one of which is picked by the bits decided so far.
template <int kBits>
__device__ __forceinline__ uint32_t search(float y, const float (&b)[(1 << kBits) - 1], float* gap) {
    bool p[kBits];
    float near = 0.f;
    uint32_t code = 0;
#pragma unroll
    for (int level = 0; level < kBits; ++level) {
        const int span = 1 << (kBits - level);                           // codes of a range at this level
        float pick[1 << (kBits - 1)];
#pragma unroll
        for (int r = 0; r < (1 << level); ++r) pick[r] = b[r * span + span / 2 - 1];
#pragma unroll
        for (int q = 0; q < level; ++q)                                  // halve the choice, first decided bit last
#pragma unroll
            for (int r = 0; r < (1 << (level - 1 - q)); ++r) pick[r] = p[level - 1 - q] ? pick[2 * r + 1] : pick[2 * r];
        const float t = y - pick[0];
        near = level == 0 ? fabsf(t) : fminf(near, fabsf(t));
        p[level] = y > pick[0];
        code |= p[level] ? 1u << (kBits - 1 - level) : 0u;
    }
    *gap = near;
    return code;
}

template <int kBits, typename Raw>
__global__ void __launch_bounds__(kRowsThreads, 1) tq_quantize_rows_kernel(const RowsParams p) {
    constexpr bool kHalf = sizeof(Raw) == 2;
    constexpr int kBounds = (1 << kBits) - 1;
    constexpr int kField = kBits == 1 ? 1 : kBits == 2 ? 2 : 4;          // bits of a packed code
    constexpr int kPerWord = 32 / kField, kWords = 64 / kPerWord;        // words of half a vector
    constexpr int kLen = kDim * kField / 8;                              // bytes of a packed vector
    extern __shared__ __align__(1024) uint8_t rows_smem[];
    uint8_t* s_bh = rows_smem;
    uint8_t* s_bl = s_bh + umma::kTileBytes;
    uint8_t* s_a = s_bl + umma::kTileBytes;                              // [buffer][high | low]
    uint32_t* s_stage = reinterpret_cast<uint32_t*>(s_a + 4 * (size_t)umma::kTileBytes);
    uint16_t* s_queue = reinterpret_cast<uint16_t*>(s_stage + (kRowsOut / 32) * 32 * kRowsStageWords);      // [buffer][..]
    __shared__ __align__(8) uint64_t s_bar[14];
    __shared__ uint32_t s_tmem;
    __shared__ int s_listed[4];
    __shared__ float s_top[4];
    __shared__ float s_bounds[16];
    __shared__ float s_norm[kRowsNorms][kRowsTile];
    auto norms = [&](int j) { return s_norm[j & (kRowsNorms - 1)]; };

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    RowsFrame f = rows_begin(s_bar, &s_tmem);
    if (tid < kBounds) s_bounds[tid] = p.table[tid];
    if (tid < 4) s_listed[tid] = 0;
    __syncthreads();
    float scale = 1.f, row_norm = 1.f;
    if (warp >= kRowsIn / 32) {
        row_norm = stage_rotation(p.Pi, s_bh, s_bl, reinterpret_cast<float*>(s_stage), s_top, &scale);
        umma::fence_operands();
        umma::fence_before_sync();
        rows_stagers_sync();
        umma::fence_after_sync();
        f.tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    }

    const long long n_tiles = (p.n_vec + kRowsTile - 1) / kRowsTile;
    const int n_mine = (int)((n_tiles - 1 - blockIdx.x) / gridDim.x) + 1;            // grid <= n_tiles
    auto first_vec = [&](int j) { return ((long long)blockIdx.x + (long long)j * gridDim.x) * kRowsTile; };
    bool ok = true;

    // The contract's chain for coordinate `coord` of vector first_vec(j) + r, and what it changes in a word that holds
    // its fast code: a correction to be added by exclusive or.
    float b[kBounds];
#pragma unroll
    for (int q = 0; q < kBounds; ++q) b[q] = s_bounds[q];
    auto correction = [&](int j, int r, int coord, uint32_t word) -> uint32_t {
        const float denom = norms(j)[r] + 1e-10f, inv = 1.0f / denom;
        auto over = [&](float x) { return kHalf ? divided(x, denom, inv) : x / denom; };
        const float4* pr = reinterpret_cast<const float4*>(p.Pi + (size_t)coord * kDim);
        const long long at = (first_vec(j) + r) * kDim;
        float y = 0.f;
#pragma unroll 4
        for (int c = 0; c < kDim / 8; ++c) {
            float v[8];
            if (kHalf) {
                const uint4 w = __ldg(reinterpret_cast<const uint4*>(static_cast<const __half*>(p.x) + at) + c);
                const float2 a = h2_to_f2(w.x), d = h2_to_f2(w.y), e = h2_to_f2(w.z), g = h2_to_f2(w.w);
                v[0] = a.x; v[1] = a.y; v[2] = d.x; v[3] = d.y; v[4] = e.x; v[5] = e.y; v[6] = g.x; v[7] = g.y;
            } else {
                const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(p.x) + at) + 2 * c;
                const float4 a = __ldg(src), d = __ldg(src + 1);
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = d.x; v[5] = d.y; v[6] = d.z; v[7] = d.w;
            }
            const float4 p0 = __ldg(pr + 2 * c), p1 = __ldg(pr + 2 * c + 1);
            y = fmaf(p0.x, over(v[0]), y); y = fmaf(p0.y, over(v[1]), y);
            y = fmaf(p0.z, over(v[2]), y); y = fmaf(p0.w, over(v[3]), y);
            y = fmaf(p1.x, over(v[4]), y); y = fmaf(p1.y, over(v[5]), y);
            y = fmaf(p1.z, over(v[6]), y); y = fmaf(p1.w, over(v[7]), y);
        }
        uint32_t code = 0;
#pragma unroll
        for (int q = 0; q < kBounds; ++q) code += y > b[q] ? 1 : 0;
        const int sh = kField * (coord % kPerWord);
        return ((code << sh) ^ word) & (((1u << kField) - 1u) << sh);
    };

    if (warp < kRowsIn / 32) {
        // ---- input: lane 16 h + r holds half h of vector 16 * warp + r, so that eight lanes fill a core matrix. An fp16
        // half stays in registers, loaded a tile ahead; an fp32 one is read twice, 32 numbers at a time ----
        const int row = 16 * warp + (lane & 15), hf = lane >> 4;
        constexpr int kParts = kHalf ? 1 : 2, kPieces = 8 / kParts;      // pieces of 8 coordinates in registers at once
        uint4 raw[8];
        auto fetch = [&](int j, int part) {
            const long long gv = first_vec(j) + row;
            const uint4* src = reinterpret_cast<const uint4*>(static_cast<const Raw*>(p.x) + gv * kDim + hf * 64) + 8 * part;
#pragma unroll
            for (int i = 0; i < 8; ++i) raw[i] = gv < p.n_vec ? __ldg(src + i) : make_uint4(0, 0, 0, 0);
        };
        auto value = [&](int c, float (&v)[8]) {
            if (kHalf) {
                const uint4 w = raw[c];
                const float2 a = h2_to_f2(w.x), b = h2_to_f2(w.y), d = h2_to_f2(w.z), e = h2_to_f2(w.w);
                v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = d.x; v[5] = d.y; v[6] = e.x; v[7] = e.y;
            } else {
                const uint4 w = raw[(2 * c) & 7], z = raw[(2 * c + 1) & 7];
                v[0] = __uint_as_float(w.x); v[1] = __uint_as_float(w.y); v[2] = __uint_as_float(w.z);
                v[3] = __uint_as_float(w.w); v[4] = __uint_as_float(z.x); v[5] = __uint_as_float(z.y);
                v[6] = __uint_as_float(z.z); v[7] = __uint_as_float(z.w);
            }
        };
        if (kHalf) fetch(0, 0);
        for (int j = 0; j < n_mine; ++j) {
            const int buf = j & 1, use = j >> 1;
            double mine = 0.0;                                           // ascending, as the contract has it
#pragma unroll
            for (int part = 0; part < kParts; ++part) {
                if (!kHalf) fetch(j, part);
#pragma unroll
                for (int c = 0; c < kPieces; ++c) {
                    float v[8];
                    value(c, v);
#pragma unroll
                    for (int e = 0; e < 8; ++e) mine = fma((double)v[e], (double)v[e], mine);
                }
            }
            const double other = __shfl_xor_sync(0xffffffffu, mine, 16);
            const float norm = (float)sqrt(hf == 0 ? mine + other : other + mine);
            const float inv = 1.0f / (norm + 1e-10f);
            if (use > 0) ok = __all_sync(0xffffffffu, f.bars.wait(f.bars.done + 8 * buf, use - 1));
            if (!ok) break;
            uint8_t* ah = s_a + (size_t)buf * 2 * umma::kTileBytes;
#pragma unroll
            for (int part = 0; part < kParts; ++part) {
                if (!kHalf) fetch(j, part);
#pragma unroll
                for (int c = 0; c < kPieces; ++c) {
                    float v[8];
                    value(c, v);
                    uint32_t h[4], l[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) split_h2(v[2 * e] * inv, v[2 * e + 1] * inv, h[e], l[e]);
                    const uint32_t off = umma::offset(row, 8 * hf + part * kPieces + c);
                    *reinterpret_cast<uint4*>(ah + off) = make_uint4(h[0], h[1], h[2], h[3]);
                    *reinterpret_cast<uint4*>(ah + umma::kTileBytes + off) = make_uint4(l[0], l[1], l[2], l[3]);
                }
            }
            if (hf == 0) {
                norms(j)[row] = norm;
                const long long gv = first_vec(j) + row;
                if (gv < p.n_vec) p.norms[gv] = norm;
            }
            umma::fence_operands();
            umma::bar_arrive(f.bars.full + 8 * buf);
            if (kHalf && j + 1 < n_mine) fetch(j + 1, 0);
        }
    } else if (warp > (kRowsIn + kRowsOut) / 32) {
        // ---- exact chains: a tile a warp in turn, a coordinate a lane; two coordinates of one word meet in an atomic ----
        for (int j = warp - (kRowsIn + kRowsOut) / 32 - 1; j < n_mine; j += kRowsExact / 32) {
            const int slot = j & 3;
            ok = __all_sync(0xffffffffu, f.bars.wait(f.bars.listed + 8 * slot, j >> 2));
            if (!ok) break;
            const int n = min(*reinterpret_cast<volatile int*>(&s_listed[slot]), kRowsQueue);
            for (int i = lane; i < n; i += 32) {
                const int e = s_queue[slot * kRowsQueue + i], r = e >> 7, coord = e & 127;
                if (e == 0xffff) continue;
                uint32_t* word = reinterpret_cast<uint32_t*>(p.indices + (first_vec(j) + r) * kLen) + coord / kPerWord;
                const uint32_t fix = correction(j, r, coord, __ldcg(word));
                if (fix != 0) atomicXor(word, fix);
            }
            __syncwarp();
            if (lane == 0) {
                s_listed[slot] = 0;
                umma::bar_arrive(f.bars.cleared + 8 * slot);
            }
        }
    } else if (warp == (kRowsIn + kRowsOut) / 32) {
        const uint64_t bh = umma::desc(umma::smem_addr(s_bh)), bl = umma::desc(umma::smem_addr(s_bl));
        const uint64_t a0 = umma::desc(umma::smem_addr(s_a));
        ok = rows_issue(f, n_mine, [&](int buf) {
            const uint64_t ah = a0 + (uint64_t)buf * (2 * umma::kTileBytes >> 4), al = ah + (umma::kTileBytes >> 4);
            const uint32_t d = f.tmem + (uint32_t)buf * kDim;
#pragma unroll
            for (int ks = 0; ks < kDim / 16; ++ks) {
                const uint64_t off = (uint64_t)ks * (2 * umma::kLbo >> 4);
                umma::mma_f16(d, al + off, bh + off, ks > 0);
                umma::mma_f16(d, ah + off, bl + off, 1);
                umma::mma_f16(d, ah + off, bh + off, 1);
            }
        });
    } else {
        // ---- results: accumulator lanes 32 * (warp % 4) .., columns 64 * half .. ----
        const int w8 = warp - kRowsIn / 32, lane0 = 32 * (warp & 3), half = w8 >> 2, row = lane0 + lane;      // kRowsIn / 32 % 4 == 0
        uint32_t* stage = s_stage + w8 * 32 * kRowsStageWords;
        uint32_t* mine = stage + lane * kRowsStageWords;
        bool sorted = row_norm < 1e18f;                                  // also false for a NaN
        float bs[kBounds];                                               // in the units of the accumulators
#pragma unroll
        for (int q = 0; q < kBounds; ++q) {
            if (q > 0) sorted = sorted && b[q - 1] <= b[q];
            bs[q] = b[q] * scale;
        }
        // where the fast value may be off by more than the band (no such table or matrix is made here): all exact
        const float band = sorted ? kRowsBand * fmaxf(row_norm, 1.0f) * scale : __int_as_float(0x7f800000);
        for (int j = 0; j < n_mine; ++j) {
            const int buf = j & 1, use = j >> 1;
            ok = __all_sync(0xffffffffu, f.bars.wait(f.bars.done + 8 * buf, use));
            if (!ok) break;
            umma::fence_after_sync();
            const long long v0 = first_vec(j);
            uint32_t near[2] = {0, 0};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t acc[32];
                umma::ld32(acc, f.tmem + (uint32_t)buf * kDim, lane0, 64 * half + 32 * c);
                if (c == 1) {
                    umma::fence_before_sync();
                    umma::bar_arrive(f.bars.taken + 8 * buf);
                }
#pragma unroll
                for (int w = 0; w < 32 / kPerWord; ++w) {
                    uint32_t word = 0;
#pragma unroll
                    for (int i = 0; i < kPerWord; ++i) {
                        float gap;
                        word |= search<kBits>(__uint_as_float(acc[w * kPerWord + i]), bs, &gap) << (kField * i);
                        if (!(gap > band)) near[c] |= 1u << (w * kPerWord + i);      // a NaN too
                    }
                    mine[c * (kWords / 2) + w] = word;
                }
            }
            // a zero vector's fast values are exact
            if (v0 + row >= p.n_vec || norms(j)[row] == 0.f) near[0] = near[1] = 0;
            // ---- what lies near a boundary goes to the exact warps, or, where the list or the indices' alignment does
            // not allow it, is done here ----
            const int slot = j & 3;
            if (j > 3) ok = __all_sync(0xffffffffu, f.bars.wait(f.bars.cleared + 8 * slot, (j >> 2) - 1));
            if (!ok) break;
            const int count = __popc(near[0]) + __popc(near[1]);
            int before = count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += t;
            }
            const int total = __shfl_sync(0xffffffffu, before, 31);
            int at = 0;
            if (lane == 0 && total > 0 && p.wide) at = atomicAdd(&s_listed[slot], total);
            at = __shfl_sync(0xffffffffu, at, 0);
            if (p.wide && at + total <= kRowsQueue) {
                at += before - count;
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    for (uint32_t m = near[c]; m != 0; m &= m - 1)
                        s_queue[slot * kRowsQueue + at++] = (uint16_t)((row << 7) | (64 * half + 32 * c + __ffs(m) - 1));
            } else {
                // entries of this list that are not filled in: an exact warp passes them over
                if (p.wide)
                    for (int i = at + lane; i < min(at + total, kRowsQueue); i += 32) s_queue[slot * kRowsQueue + i] = 0xffffu;
#pragma unroll 1
                for (int c = 0; c < 2; ++c)
#pragma unroll 1
                    for (uint32_t m = near[c]; m != 0; m &= m - 1) {
                        const int x = 32 * c + __ffs(m) - 1;
                        mine[x / kPerWord] ^= correction(j, row, 64 * half + x, mine[x / kPerWord]);
                    }
            }
            __syncwarp();
            // ---- whole words out, rows one after another ----
            uint8_t* dst = p.indices + (v0 + lane0) * kLen + half * (kLen / 2);
            const int n_rows = (int)min((long long)32, p.n_vec - (v0 + lane0));
            for (int i = lane; i < n_rows * kWords; i += 32) {
                const int r = i / kWords, w = i % kWords;
                const uint32_t word = stage[r * kRowsStageWords + w];
                uint8_t* to = dst + r * kLen + 4 * w;
                if (p.wide) {
                    *reinterpret_cast<uint32_t*>(to) = word;
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) to[e] = (uint8_t)(word >> (8 * e));
                }
            }
            __syncwarp();
            umma::bar_arrive(f.bars.listed + 8 * slot);
        }
    }
    if (rows_end(f, ok, p.status)) {
        // codes are missing: no vector of this CTA may pass for one that was quantized
        for (int j = 0; j < n_mine; ++j)
            if (tid < kRowsTile && first_vec(j) + tid < p.n_vec) p.norms[first_vec(j) + tid] = __int_as_float(0x7fffffff);
    }
}

constexpr int kChainWarps = 8, kUnpackThreads = 128;
constexpr int kDequantThreads = kChainWarps * 32 + kUnpackThreads;
constexpr size_t kDequantSmemBytes = 3 * (size_t)kDim * kRowsTile * sizeof(float) + 256 * sizeof(float2);

__global__ void __launch_bounds__(kDequantThreads, 1) tq_dequantize_rows_kernel(const RowsParams p, int bits) {
    extern __shared__ __align__(1024) uint8_t rows_smem[];
    float* s_b = reinterpret_cast<float*>(rows_smem);                    // [k][coordinate]
    float* s_a = s_b + kDim * kDim;                                      // [buffer][k][vector]
    float2* s_pair = reinterpret_cast<float2*>(s_a + 2 * kDim * kRowsTile);      // two codes of four bits -> centroids
    __shared__ float s_norm[2][kRowsTile];

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    // a lookup's place: the low code's bank bits mixed with the high code's, so that lanes spread over the banks
    auto place = [](uint32_t pair) { return pair ^ ((pair >> 3) & 14u); };
    if (tid < 256) {
        auto centroid = [&](int code) { return code < (1 << bits) ? p.table[code] : __int_as_float(0x7f800000); };
        s_pair[place((uint32_t)tid)] = make_float2(centroid(tid & 15), centroid(tid >> 4));
    }
    __syncthreads();
    if (warp < kChainWarps) {                                            // beside the unpacking of the first tile
        for (int i = tid; i < kDim * kDim / 4; i += kChainWarps * 32)
            reinterpret_cast<float4*>(s_b)[i] = __ldg(reinterpret_cast<const float4*>(p.Pi) + i);
        asm volatile("bar.sync 5, %0;" ::"n"(kChainWarps * 32) : "memory");
    }

    // this CTA's vectors, in units of sixteen
    const long long units = (p.n_vec + 15) / 16;
    const long long lo = units * blockIdx.x / gridDim.x * 16;
    const long long hi = min(p.n_vec, units * (blockIdx.x + 1) / gridDim.x * 16);
    const int n_mine = (int)((hi - lo + kRowsTile - 1) / kRowsTile);
    // named barriers 1, 2: buffer filled; 3, 4: buffer read. The side that goes on arrives, the side that waits syncs.
    auto sync = [](int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kDequantThreads) : "memory"); };
    auto arrive = [](int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kDequantThreads) : "memory"); };

    if (warp >= kChainWarps) {
        // ---- unpacking: a vector a thread, lanes on neighbouring vectors of a row of the panel ----
        const int v = tid - kChainWarps * 32;
        auto work = [&](auto width) {
            constexpr int kField = decltype(width)::value, kBytes = 16 * kField;      // of a vector
            for (int j = 0; j < n_mine; ++j) {
                const long long gv = lo + (long long)j * kRowsTile + v;
                const bool live = gv < hi;
                const uint8_t* src = p.indices + gv * kBytes;
                uint4 raw[kField];
#pragma unroll
                for (int i = 0; i < kField; ++i) {
                    raw[i] = make_uint4(0, 0, 0, 0);
                    if (live && p.wide) {
                        raw[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
                    } else if (live) {
                        uint32_t w[4] = {0, 0, 0, 0};
                        for (int e = 0; e < 16; ++e) w[e >> 2] |= (uint32_t)src[16 * i + e] << (8 * (e & 3));
                        raw[i] = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
                const float norm = live ? __ldg(p.norms + gv) : 0.f;
                if (j > 1) sync(3 + (j & 1));
                float* a = s_a + (j & 1) * kDim * kRowsTile + v;
#pragma unroll
                for (int i = 0; i < 4 * kField; ++i) {
                    const uint4& r = raw[i >> 2];
                    const uint32_t word = (i & 3) == 0 ? r.x : (i & 3) == 1 ? r.y : (i & 3) == 2 ? r.z : r.w;
#pragma unroll
                    for (int q = 0; q < 16 / kField; ++q) {               // two codes
                        const uint32_t two = word >> (2 * kField * q), mask = (1u << kField) - 1u;
                        const uint32_t pair = kField == 4 ? two & 255u : (two & mask) | (((two >> kField) & mask) << 4);
                        const float2 c = s_pair[place(pair)];
                        const int k = i * (32 / kField) + 2 * q;
                        a[k * kRowsTile] = c.x;
                        a[(k + 1) * kRowsTile] = c.y;
                    }
                }
                s_norm[j & 1][v] = norm;
                arrive(1 + (j & 1));
            }
        };
        if (bits == 1) work(std::integral_constant<int, 1>{});
        else if (bits == 2) work(std::integral_constant<int, 2>{});
        else work(std::integral_constant<int, 4>{});
    } else {
        // ---- chains: a warp has sixteen vectors and all coordinates, or in a tile of at most 64 vectors half of them (a
        // single warp on a scheduler would leave it half idle); a thread eight vectors and 8 or 4 coordinates ----
        const int tn = lane & 15;
        auto chains = [&](auto width, int j, int first, int col) {
            constexpr int kCols = decltype(width)::value;
            const long long v0 = lo + (long long)j * kRowsTile + first;
            const float* a = s_a + (j & 1) * kDim * kRowsTile + first;
            const float* b = s_b + col;
            float2 acc[4][kCols];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int c = 0; c < kCols; ++c) acc[i][c] = make_float2(0.f, 0.f);
#pragma unroll 4
            for (int k = 0; k < kDim; ++k) {
                const float4 a0 = *reinterpret_cast<const float4*>(a + k * kRowsTile);
                const float4 a1 = *reinterpret_cast<const float4*>(a + k * kRowsTile + 4);
                const float2 av[4] = {{a0.x, a0.y}, {a0.z, a0.w}, {a1.x, a1.y}, {a1.z, a1.w}};
#pragma unroll
                for (int q = 0; q < kCols / 4; ++q) {
                    const float4 w = *reinterpret_cast<const float4*>(b + k * kDim + 64 * q);
                    const float bv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            acc[i][4 * q + c] = fma_two(av[i], make_float2(bv[c], bv[c]), acc[i][4 * q + c]);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (v0 + i >= hi) continue;
                const float n = s_norm[j & 1][first + i];
#pragma unroll
                for (int q = 0; q < kCols / 4; ++q) {
                    float r[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) r[c] = ((i & 1) ? acc[i >> 1][4 * q + c].y : acc[i >> 1][4 * q + c].x) * n;
                    const long long at = (v0 + i) * kDim + col + 64 * q;
                    if (p.out_dtype == 1) {
                        *reinterpret_cast<float4*>(static_cast<float*>(p.out) + at) = make_float4(r[0], r[1], r[2], r[3]);
                    } else {
                        __half2 h[2] = {__floats2half2_rn(r[0], r[1]), __floats2half2_rn(r[2], r[3])};
                        *reinterpret_cast<uint2*>(static_cast<__half*>(p.out) + at) = *reinterpret_cast<uint2*>(h);
                    }
                }
            }
        };
        for (int j = 0; j < n_mine; ++j) {
            sync(1 + (j & 1));
            const int rows = (int)min((long long)kRowsTile, hi - lo - (long long)j * kRowsTile);
            if (rows > kRowsTile / 2) {
                if (16 * warp < rows) chains(std::integral_constant<int, 8>{}, j, 16 * warp + 8 * (lane >> 4), 4 * tn);
            } else if (16 * (warp & 3) < rows) {
                chains(std::integral_constant<int, 4>{}, j, 16 * (warp & 3) + 8 * (lane >> 4), 64 * (warp >> 2) + 4 * tn);
            }
            if (j + 2 < n_mine) arrive(3 + (j & 1));
        }
    }
}
