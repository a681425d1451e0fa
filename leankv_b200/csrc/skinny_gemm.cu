// y[rows][N] = x[rows][K] W[K][N] for few rows (fp16, fp32 sums): the projections of a batched decode step, whose time is that of
// streaming W once.
//
// W's columns are the 128 rows of a tcgen05 product and the batch its columns, so a tile of W goes from HBM by TMA into swizzled shared
// memory and from there to the tensor core as it lies (MN-major operand): no register touches it. A CTA takes 128 columns of W and
// a share of K; the shares of a column block are one cluster, whose CTAs add their sums through distributed shared memory, each a part
// of the rows, in rank order. Stages of 64 rows of W (16 KB) beside the batch's columns, as many as half an SM holds (six up to 16 rows, five up to 32,
// four up to 64, three at 128), and two CTAs an SM keep 96 to 192 KB of W an SM in flight.
//
//   warp 0   copies: W's tiles, ahead of the dependency wait where the caller says that the launch ahead does not write them,
//            and the batch's columns of the same K
//   warp 1   products, one elected lane
//   all      sums out of tensor memory, exchange, output

#include <algorithm>

#include "common.cuh"
#include "tma.cuh"

namespace leankv {
namespace {

constexpr int kThreads = 128;
constexpr int kCols = 128;                       // columns of W a CTA
constexpr int kKStep = 64;                       // rows of W a stage: one 128-byte swizzle atom of x
constexpr int kMaxStages = 6;
constexpr int kMaxRows = 128;
constexpr int kMaxSplit = 8;                     // CTAs of a cluster
constexpr uint32_t kWBytes = kKStep * kCols * 2; // two blocks of 64 columns

struct SkinnyArgs {
    CUtensorMap w, x;
    __half* y;
    int* status;
    int rows, rows_pad, N, steps, stages, early, tmem_first;     // steps: of K
    uint32_t tmem_cols;
};

__host__ __device__ constexpr uint32_t idesc_f16_at(int n) {      // D fp32, A and B fp16, A MN-major, M = 128
    return (1u << 4) | (1u << 15) | ((uint32_t)(n / 8) << 17) | (8u << 24);
}

__device__ __forceinline__ void load2(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

__global__ void __launch_bounds__(kThreads, 2) skinny_gemm_kernel(const __grid_constant__ SkinnyArgs p) {
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ __align__(8) uint64_t s_full[kMaxStages], s_free[kMaxStages], s_done;
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t base = (umma::smem_addr(raw) + 1023u) & ~1023u;
    const uint32_t x_bytes = (uint32_t)p.rows_pad * 128u, stage_bytes = kWBytes + (x_bytes + 1023u) / 1024u * 1024u;
    auto addr = [](const void* q) { return umma::smem_addr(q); };
    if (tid == 0) {
        for (int s = 0; s < p.stages; ++s) {
            umma::bar_init_n(addr(&s_full[s]), 1);
            umma::bar_init_n(addr(&s_free[s]), 1);
        }
        umma::bar_init_n(addr(&s_done), 1);
        s_fail = 0;
    }
    if (p.tmem_first && warp == 1) umma::tmem_alloc_n(addr(&s_tmem), p.tmem_cols);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();

    const int split = blockIdx.y, n_split = gridDim.y, n0 = blockIdx.x * kCols;
    const int s0 = p.steps * split / n_split, n_steps = p.steps * (split + 1) / n_split - s0;
    bool ok = true;
    if (tid == 0) {                                      // ---- copies ----
        auto load_w = [&](int j) {
            const int s = j % p.stages;
            tma::expect(addr(&s_full[s]), kWBytes + x_bytes);
            for (int b = 0; b < kCols / 64; ++b)
                load2(base + s * stage_bytes + b * (kWBytes / 2), &p.w, n0 + b * 64, (s0 + j) * kKStep, addr(&s_full[s]));
        };
        auto load_x = [&](int j) {
            const int s = j % p.stages;
            load2(base + s * stage_bytes + kWBytes, &p.x, (s0 + j) * kKStep, 0, addr(&s_full[s]));
        };
        const int first = min(p.stages, n_steps);
        if (!p.early) pdl_wait();
        for (int j = 0; j < first; ++j) load_w(j);
        if (p.early) pdl_wait();
        for (int j = 0; j < first; ++j) load_x(j);
        int j = first;
        for (; j < n_steps; ++j) {
            ok = umma::bar_wait(addr(&s_free[j % p.stages]), (j / p.stages - 1) & 1);
            if (!ok) break;
            load_w(j);
            load_x(j);
        }
        if (!ok)                                         // give up only once the copies in flight have landed
            for (int i = max(j - p.stages, 0); i < j; ++i) umma::bar_wait(addr(&s_full[i % p.stages]), (i / p.stages) & 1);
    } else if (warp == 1) {                              // ---- products ----
        // Tensor memory is taken before later launches are let in: one of them could hold it while it waits for this one. And it is taken
        // behind the wait, where no block of a launch ahead can still be asking for its own; only where the caller says that the
        // launch ahead takes none it is taken while that one drains (2048 x 2048, 16 rows, launches of this kernel one behind the other
        // 5.4 us so, 5.7 behind the wait; steps of two to four layers 1 to 5 us).
        pdl_wait();
        if (!p.tmem_first) umma::tmem_alloc_n(addr(&s_tmem), p.tmem_cols);
        pdl_launch();
        umma::fence_before_sync();
        __syncwarp();
        umma::fence_after_sync();
        const uint32_t tmem = __shfl_sync(0xffffffffu, *static_cast<volatile uint32_t*>(&s_tmem), 0);
        const uint32_t idesc = idesc_f16_at(p.rows_pad);
        auto all = [&](bool done) { return __all_sync(0xffffffffu, done) != 0; };
        for (int j = 0; j < n_steps; ++j) {
            const int s = j % p.stages;
            ok = all(umma::bar_wait(addr(&s_full[s]), (j / p.stages) & 1));
            if (!ok) break;
            umma::fence_after_sync();
            const uint64_t dw = tma::swizzled(base + s * stage_bytes, kWBytes / 2), dx = tma::swizzled(base + s * stage_bytes + kWBytes, 16);
            if (umma::elect()) {
#pragma unroll
                for (int k = 0; k < kKStep / 16; ++k)    // 16 rows of W are 2048 bytes further, 16 columns of x 32
                    umma::mma_f16_n(tmem, dw + k * (2048 >> 4), dx + k * 2, idesc, j > 0 || k > 0);
                umma::commit(addr(&s_free[s]));
            }
            __syncwarp();
        }
        if (umma::elect()) umma::commit(addr(&s_done));
        __syncwarp();
    } else {
        pdl_wait();
    }
    __syncwarp();                                        // no lane polls beside the copying one
    if (!umma::bar_wait(addr(&s_done), 0)) ok = false;
    if (!ok) s_fail = 1;
    umma::fence_before_sync();
    __syncthreads();                                     // the address of the tensor memory is there
    umma::fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    // ---- this CTA's sums to shared memory, [row][column of W]: the stages are free ----
    float* sums = reinterpret_cast<float*>(raw + (base - addr(raw)));
#pragma unroll 1
    for (int c = 0; c < p.rows_pad; c += 32) {
        uint32_t o[32];
        umma::ld32(o, tmem, warp * 32, c);
#pragma unroll
        for (int b = 0; b < 32; ++b)
            if (c + b < p.rows) sums[(c + b) * kCols + tid] = __uint_as_float(o[b]);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        umma::fence_after_sync();
        umma::tmem_free_n(tmem, p.tmem_cols);
    }
    if (s_fail) {                                        // a wait ran out: no numbers
        for (int e = tid; e < p.rows * kCols; e += kThreads) sums[e] = __int_as_float(0x7fc00000);
        if (tid == 0 && p.status != nullptr) atomicOr(p.status, LEANKV_SKINNY_GAVE_UP);
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    // ---- four columns a thread, this CTA's part of the rows ----
    const int r0 = p.rows * split / n_split, r1 = p.rows * (split + 1) / n_split, c4 = lane * 4;
    for (int r = r0 + warp; r < r1; r += kThreads / 32) {
        const uint32_t at = addr(sums + r * kCols + c4);
        float4 part[kMaxSplit];
#pragma unroll
        for (int c = 0; c < kMaxSplit; ++c)
            if (c < n_split) {
                uint32_t from;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from) : "r"(at), "r"(c));
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(part[c].x), "=f"(part[c].y), "=f"(part[c].z), "=f"(part[c].w) : "r"(from) : "memory");
            }
        float4 t = part[0];
#pragma unroll
        for (int c = 1; c < kMaxSplit; ++c)
            if (c < n_split) { t.x += part[c].x; t.y += part[c].y; t.z += part[c].z; t.w += part[c].w; }
        if (n0 + c4 < p.N) {                             // N % 8 == 0
            const __half2 a = __floats2half2_rn(t.x, t.y), b = __floats2half2_rn(t.z, t.w);
            *reinterpret_cast<uint2*>(p.y + (size_t)r * p.N + n0 + c4) =
                make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        }
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");        // the others still read this CTA's sums
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

}  // namespace
}  // namespace leankv

using namespace leankv;

extern "C" int leankv_skinny_gemm_f16_status(const void* x, const void* w, void* y, int rows, int K, int N, int flags, int32_t* status,
                                             void* stream) {
    if ((flags & ~(LEANKV_SKINNY_EARLY_WEIGHTS | LEANKV_SKINNY_EARLY_TMEM)) != 0) return LEANKV_EINVAL;
    if (!x || !w || !y || rows <= 0 || K <= 0 || N <= 0) return LEANKV_EINVAL;
    if (rows > kMaxRows) return LEANKV_ELIMIT;
    if (K % 8 || N % 8 || !aligned16(x) || !aligned16(w) || !aligned16(y)) return LEANKV_EALIGN;
    SkinnyArgs p{};
    p.y = static_cast<__half*>(y);
    p.status = status;
    p.rows = rows;
    p.rows_pad = (rows + 15) / 16 * 16;
    p.N = N;
    p.steps = (K + kKStep - 1) / kKStep;
    p.tmem_first = (flags & LEANKV_SKINNY_EARLY_TMEM) != 0;
    // Weights ahead of the wait pay only where the tensor memory is there, too: taken beside copies in flight it comes late (launches one behind the
    // other, 16 rows, us with both early / only the weights / neither: 4096 x 6144 11.0 / 11.9 / 10.9, 2048 x 2048 5.4 / 6.1 / 5.7, 14336 x 4096
    // 20.7 / 22.2 / 21.1; in steps of a batch both early is the best).
    p.early = p.tmem_first && (flags & LEANKV_SKINNY_EARLY_WEIGHTS) != 0;
    p.tmem_cols = p.rows_pad <= 32 ? 32 : p.rows_pad <= 64 ? 64 : 128;
    const size_t x_bytes = ((size_t)p.rows_pad * 128 + 1023) / 1024 * 1024;
    p.stages = (int)std::min<size_t>(kMaxStages, (110 * 1024 - 1024) / (kWBytes + x_bytes));
    const size_t smem = std::max(p.stages * (kWBytes + x_bytes), (size_t)rows * kCols * 4) + 1024;
    const int blocks = (N + kCols - 1) / kCols;
    // as many CTAs as clusters of up to eight find room for (6144 columns, us by CTAs: 144 13.4, 192 12.1, 240 11.7, 288 18.1)
    const int split = std::max(1, std::min(std::min(kMaxSplit, 256 / blocks), p.steps / 2));
    const auto map = [](CUtensorMap* m, const void* base, cuuint64_t inner, cuuint64_t outer, cuuint32_t box_rows) {
        const cuuint64_t dims[2] = {inner, outer}, strides[1] = {inner};
        const cuuint32_t box[2] = {(cuuint32_t)tma::kBoxCols, box_rows};
        return tma::make_map(m, base, 2, dims, strides, box, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    };
    int rc = map(&p.w, w, N, K, kKStep);
    if (!rc) rc = map(&p.x, x, K, rows, p.rows_pad);
    if (rc) return rc;
    LEANKV_CUDA_TRY(cudaFuncSetAttribute(skinny_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    LEANKV_CUDA_TRY(launch_cluster_kernel_ex(true, dim3(1, split, 1), skinny_gemm_kernel, dim3(blocks, split), dim3(kThreads), smem,
                                             static_cast<cudaStream_t>(stream), p));
    return LEANKV_OK;
}

extern "C" int leankv_skinny_gemm_f16(const void* x, const void* w, void* y, int rows, int K, int N, int flags, void* stream) {
    return leankv_skinny_gemm_f16_status(x, w, y, rows, K, N, flags, nullptr, stream);
}
