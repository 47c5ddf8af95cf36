// True 32-bit matrix product on the CUDA cores: C[M,N] = A[M,K] * B[N,K]^T, the
// y = x W^T of every projection (xiyiji/paged-llm llama.py:141-144, :166-168,
// :208).  No tensor cores and no reduced-precision mode.  The k axis is cut into
// parts whose length depends on K alone (part_length); within a part the even and
// the odd k are one chain of float32 fused multiply-adds each, in order, the two
// are added, and the parts are added in order.  So a row's result does not depend
// on which other rows are in the batch, on the tile shape, or on whether the
// parts ran in one block or in the blocks of a cluster.
//
// What bounds it: the FMA pipes from some 16 rows on, the read of B below.  So
//   - a thread's operands are 16 bytes along k of one row (both matrices are
//     contiguous along k: cp.async brings them into shared memory as they are, four
//     stages or more ahead, no transposition), and a packed fma.rn.f32x2 takes an even
//     and an odd k at once: half the issue slots, no packing moves;
//   - rows in shared memory are 4 words longer than a multiple of 8 words, so the eight
//     rows that a quarter of a warp reads 16 bytes of lie in different banks;
//   - few tiles: the parts run in the blocks of a cluster, which add them up through
//     distributed shared memory.
//
// Measured on a B200 (cold L2), us, against the 64 x 64 x 16 tile with scalar loads and no stages before:
//   1 x 32000 x 2048        70    (3.8 TB/s)
//   128 x 2048 x 2048       43    (650 on average over the products of a layer of 128 tokens before, 112 now)
//   128 x 11264 x 2048     181    (33 TFLOP/s)
//   2048 x 2560 x 2048     580    (37 TFLOP/s; 8 x 4 elements per thread and plain fmaf: 565 and 596)
// The relative error against 64 bits is 2.1e-7 at K = 2048 (one chain over all k: 8.1e-7).
#include <cooperative_groups.h>

#include "common.cuh"

namespace {

namespace cg = cooperative_groups;

struct SgemmParams {
    const float *A, *B;
    float* C;
    int M, N, K, lda, ldb, ldc;
    int part_len;            // k per part, a multiple of 32
};

constexpr int SG_MAX_PARTS = 8;

// k per part: about 256, at most SG_MAX_PARTS parts.
int part_length(int K) {
    int parts = (K + 255) / 256;
    parts = parts < 1 ? 1 : parts > SG_MAX_PARTS ? SG_MAX_PARTS : parts;
    const int len = (K + parts - 1) / parts;
    return (len + 31) / 32 * 32;
}

typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& acc, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum2(f32x2 v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }

template <int BYTES> __device__ __forceinline__ void sg_copy(void* dst, const void* src, int bytes) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(bytes));
}

// One stage's box of a matrix: ROWS rows from row0, BK k from k0; what lies outside [rows, K] becomes zero.
template <int ROWS, int BK, int THREADS, bool VEC>
__device__ __forceinline__ void sg_load(float* dst, const float* src, int ld, int row0, int rows, int k0, int K) {
    constexpr int W = VEC ? 4 : 1, PER_ROW = BK / W;
#pragma unroll
    for (int e0 = 0; e0 < ROWS * PER_ROW; e0 += THREADS) {
        const int e = e0 + (int)threadIdx.x;
        if (ROWS * PER_ROW % THREADS != 0 && e >= ROWS * PER_ROW) break;
        const int r = e / PER_ROW, k = k0 + (e % PER_ROW) * W;
        const bool in = row0 + r < rows && k < K;
        const int bytes = in ? min(W, K - k) * 4 : 0;
        sg_copy<W * 4>(dst + r * (BK + 4) + (e % PER_ROW) * W, in ? src + (size_t)(row0 + r) * ld + k : src, bytes);
    }
}

// Thread (tx, ty) of a block owns rows ty + i * (BM / TM) and columns tx + j * (BN / TN).  gridDim.z > 1: the blocks
// of a cluster take a part of k each; else a block takes all parts one after the other and keeps the sum of the
// finished ones in shared memory behind the stages (registers are full: 8 x 8 pairs).
template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) sgemm_nt_kernel(SgemmParams p) {
    constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY;
    constexpr int WX = TX < 8 || TY < 4 ? TX : 8;              // threads of a warp along n: 8 x 4 where both fit
    constexpr int ROW = BK + 4, A_FLOATS = BM * ROW, STAGE = (BM + BN) * ROW;
    static_assert(TY == 1 ? TX % 32 == 0 : (TX % 8 == 0 && TY % 4 == 0), "whole warps");
    extern __shared__ __align__(16) float sg_smem[];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = TY == 1 ? tid : (warp % (TX / 8)) * WX + lane % WX;
    const int ty = TY == 1 ? 0 : (warp / (TX / 8)) * 4 + lane / WX;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const bool split = gridDim.z > 1;
    const int steps_per_part = p.part_len / BK;
    const int all = (p.K + BK - 1) / BK;
    const int first = split ? min(all, (int)blockIdx.z * steps_per_part) : 0;
    const int steps = (split ? min(all, first + steps_per_part) : all) - first;

    pdl_launch_dependents();
    // the weights do not depend on the kernel in front: their first stages are asked for before the wait for it
    int loaded = 0;
    for (; loaded < STAGES - 1 && loaded < steps; ++loaded)
        sg_load<BN, BK, THREADS, VEC>(sg_smem + loaded * STAGE + A_FLOATS, p.B, p.ldb, n0, p.N, (first + loaded) * BK, p.K);
    pdl_wait();
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < loaded) sg_load<BM, BK, THREADS, VEC>(sg_smem + s * STAGE, p.A, p.lda, m0, p.M, (first + s) * BK, p.K);
        asm volatile("cp.async.commit_group;\n" ::);
    }

    f32x2 acc[TM][TN];
    float* total = sg_smem + STAGES * STAGE + tid;              // [TM * TN][THREADS] (one after the other only)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

    int left = steps_per_part;                                  // steps to the end of the current part
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
        __syncthreads();
        const int next = s + STAGES - 1;
        if (next < steps) {
            float* st = sg_smem + (next % STAGES) * STAGE;
            sg_load<BN, BK, THREADS, VEC>(st + A_FLOATS, p.B, p.ldb, n0, p.N, (first + next) * BK, p.K);
            sg_load<BM, BK, THREADS, VEC>(st, p.A, p.lda, m0, p.M, (first + next) * BK, p.K);
        }
        asm volatile("cp.async.commit_group;\n" ::);
        const float* as = sg_smem + (s % STAGES) * STAGE + ty * ROW;
        const float* bs = sg_smem + (s % STAGES) * STAGE + A_FLOATS + tx * ROW;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            ulonglong2 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(as + i * TY * ROW + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bs + j * TX * ROW + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
                for (int i = 0; i < TM; ++i) fma2(acc[i][j], a[i].y, b.y);
            }
        }
        if (!split && --left == 0 && s + 1 < steps) {
            left = steps_per_part;
            const bool start = s + 1 == steps_per_part;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    float* t = total + (i * TN + j) * THREADS;
                    *t = (start ? 0.f : *t) + sum2(acc[i][j]);
                    acc[i][j] = 0ull;
                }
        }
    }

    if (!split) {
        const bool one = steps <= steps_per_part;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int m = m0 + ty + i * TY;
            if (m >= p.M) continue;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int n = n0 + tx + j * TX;
                if (n < p.N) p.C[(size_t)m * p.ldc + n] = (one ? 0.f : total[(i * TN + j) * THREADS]) + sum2(acc[i][j]);
            }
        }
        return;
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();                                            // the stages are free: the part's sums take their place
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sg_smem[(ty + i * TY) * BN + tx + j * TX] = sum2(acc[i][j]);
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int parts = (int)gridDim.z;
    for (int e = (int)blockIdx.z * THREADS + tid; e < BM * BN; e += parts * THREADS) {
        const int m = m0 + e / BN, n = n0 + e % BN;
        if (m >= p.M || n >= p.N) continue;
        float v[SG_MAX_PARTS];
#pragma unroll
        for (int z = 0; z < SG_MAX_PARTS; ++z)
            v[z] = z < parts ? cluster.map_shared_rank(sg_smem, z)[e] : 0.f;
        float sum = 0.f;
#pragma unroll
        for (int z = 0; z < SG_MAX_PARTS; ++z)
            if (z < parts) sum += v[z];
        p.C[(size_t)m * p.ldc + n] = sum;
    }
    cluster.sync();                                             // nobody leaves while its sums are still read
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool VEC>
int launch_sgemm(const SgemmParams& p, int serial_from, cudaStream_t stream) {
    constexpr int stages = STAGES * (BM + BN) * (BK + 4) * 4, tile = BM * BN * 4;
    static_assert(stages >= tile, "a part's sums fit where the stages were");
    static PerDevice<char> ready;
    if (!ready.get("gemm_f32", [&](char&) {
            PL_CUDA(cudaFuncSetAttribute(sgemm_nt_kernel<BM, BN, TM, TN, BK, STAGES, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, stages + tile));
            return 0;
        }))
        return 1;
    const int parts = (p.K + p.part_len - 1) / p.part_len;
    const long long tiles = (long long)((p.N + BN - 1) / BN) * ((p.M + BM - 1) / BM);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, tiles < serial_from ? parts : 1);
    cfg.blockDim = dim3((BM / TM) * (BN / TN));
    cfg.dynamicSmemBytes = cfg.gridDim.z > 1 || parts == 1 ? stages : stages + tile;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = cfg.gridDim.z;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    static const bool no_pdl = getenv("PAGED_LLM_B200_NO_PDL") != nullptr;
    cfg.attrs = attr;
    cfg.numAttrs = no_pdl ? 1 : 2;
    PL_CUDA(cudaLaunchKernelEx(&cfg, sgemm_nt_kernel<BM, BN, TM, TN, BK, STAGES, VEC>, p));
    return 0;
}

template <bool VEC> int dispatch_sgemm(const SgemmParams& p, cudaStream_t stream) {
    constexpr int NEVER = 1 << 30;
    if (p.M <= 2) return launch_sgemm<2, 64, 2, 1, 32, 6, VEC>(p, NEVER, stream);
    if (p.M <= 4) return launch_sgemm<4, 64, 4, 1, 32, 6, VEC>(p, NEVER, stream);
    if (p.M <= 8) return launch_sgemm<8, 64, 8, 1, 32, 6, VEC>(p, NEVER, stream);
    if (p.M <= 32) return launch_sgemm<32, 64, 8, 4, 16, 4, VEC>(p, 1480, stream);
    return launch_sgemm<64, 64, 8, 8, 16, 4, VEC>(p, 1480, stream);
}

}  // namespace

PL_EXPORT int pl_gemm_f32(const float* A, const float* B, float* C, int M, int N, int K, int lda, int ldb, int ldc,
                          cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    PL_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    PL_REQUIRE(lda >= K && ldb >= K && ldc >= N, "gemm_f32: leading dimensions too small");
    SgemmParams p = {A, B, C, M, N, K, lda, ldb, ldc, part_length(K)};
    const bool vec = lda % 4 == 0 && ldb % 4 == 0 && (((uintptr_t)A | (uintptr_t)B) & 15) == 0;
    return vec ? dispatch_sgemm<true>(p, stream) : dispatch_sgemm<false>(p, stream);
}
