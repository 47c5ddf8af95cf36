// Matrix product for a middling number of tokens (decode steps of a busy server, short prompts: 17 to 64 rows of X) on
// the 5th-generation tensor cores: Y[M,N] = X[M,K] * W[N,K]^T, bfloat16 in, float32 accumulation in tensor memory.
//
// What bounds it is the read of W, so the machine is filled with readers of W: a block takes 128 rows of W (the 128 lanes
// of the accumulator; the tokens are its columns, so a tile is never wider than the step) and one part of k; the blocks of
// a cluster share the rows and add their parts up through distributed shared memory, each for its own tokens, in a fixed
// order.  The number of parts depends on the product (N, K, what follows it) and the GPU alone: a token's result does not
// depend on the batch.  Two blocks fit an
// SM, so the copies of one run on while the other drains, and since W does not depend on the kernel in front, a block
// fills its ring with W before it waits for that kernel and adds the X boxes afterwards.
//
// One kernel per projection: what follows the product is done where its sums come together, a warp per token:
//   plain   y = s acc (bfloat16 or float32)
//   SiLU    the 128 rows are 64 gate rows and the 64 matching up rows; y = act(s gate) * (s up)  (xiyiji/paged-llm llama.py:171)
//   add     x += bf16(acc) in float32 (llama.py:183-184), and for the norm that follows (llama.py:80-83):
//           h = bf16(x * w) and the sum of squares of the 128 new x
// where s is 1, or, for X = h of an "add" product, the token's 1 / rms(x) from those sums: RMSNorm(x) * w = s * h, and a
// factor per token can wait until after the product (h is rounded relative to its size either way).
//
// Every wait is bounded; a thread that gave up waits once more for the copies in flight and stops.
//
// Measured on a B200, us per product among others of its kind (graph of 16, cold weights), in brackets the library's
// product with the kernel that then adds and norms, or multiplies by the activation, and the read of W at 6.45 TB/s:
//                              24 tokens        64 tokens       128 tokens
//   2,560 x 2,048, plain      6.3 ( 6.0)       8.0 ( 6.0)      11.9 ( 6.3)     1.6
//   2,048 x 2,048, add        6.0 ( 8.8)       7.4 ( 9.0)      10.5 ( 9.2)     1.3
//   5,632 x 2,048, SiLU      11.3 (13.4)      12.9 (13.6)      15.2 (13.3)     7.2
//   2,048 x 5,632, add        8.9 (13.2)      10.3 (13.3)      14.2 (13.7)     3.6
//   2,048 x 8,192, add       10.8 (16.2)      12.4 (16.5)      16.6 (16.7)     5.2
//   4,096 x 14,336, add      25.9 (29.1)      27.9 (29.5)      33.9 (30.7)    18.2
// The sum over a layer meets the library's near 96 tokens, since every block reads all of X for its k: MID_MAX_COLS.
#include "tcgen05.cuh"
#include "tensor_map.cuh"

enum { MID_BF16 = 0, MID_F32 = 1, MID_SILU = 2, MID_ADD = 3 };

struct MidParams {
    void* Y;                     // [M, ldy] (plain, SiLU)
    float* resid;                // [M, N] (add)
    __nv_bfloat16* h;            // [M, N] (add)
    const void* norm_w;          // [N] (add)
    float* part_out;             // [N / 128][MID_PART] (add)
    const float* part_in;        // [K / 128][MID_PART] or null: s = 1
    float eps;
    int norm_w_bf16;
    int ldy, M, N, K, I, act;
    int cols;                    // tokens rounded up to 32: the accumulator's columns
    int stages;
};

namespace {

using namespace tc;

constexpr int MID_ROWS = 128, MID_BK = 64, MID_THREADS = 384, MID_MAX_STAGES = 5, MID_MAX_COLS = 64, MID_MAX_PARTS = 8;
constexpr int MID_PART = 256;                                    // tokens a row of the sums of squares has room for
constexpr int MID_W_BYTES = MID_ROWS * 128;
constexpr int MID_RING = 100 * 1024;                             // two blocks per SM
static_assert(MID_MAX_COLS * MID_ROWS * 4 <= MID_RING, "a block's sums take the place of its ring");

__device__ __forceinline__ void mid_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mid_tma(uint32_t dst, const CUtensorMap* map, int col, int row, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
        "l"(map), "r"(col), "r"(row), "r"(saddr(bar))
        : "memory");
}
__device__ __forceinline__ uint32_t mid_peer(uint32_t addr, int rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(addr), "r"(rank));
    return remote;
}
__device__ __forceinline__ float4 mid_read4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 mid_read2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t mid_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float mid_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// grid: (tiles of 128 rows of W) x (parts of k), the parts of a tile being a cluster.
template <int EPI>
__global__ void __launch_bounds__(MID_THREADS, 2) gemm_mid_kernel(MidParams p, const __grid_constant__ CUtensorMap x_map,
                                                                  const __grid_constant__ CUtensorMap w_map) {
    extern __shared__ unsigned char mid_smem[];
    __shared__ uint64_t full[MID_MAX_STAGES], empty[MID_MAX_STAGES], acc_full;
    __shared__ uint32_t tmem_slot;
    __shared__ float scale_of[MID_MAX_COLS];
    unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)mid_smem + 1023) & ~(uintptr_t)1023);
    float* partial = reinterpret_cast<float*>(ring);             // [cols][128], once the ring is used up
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t rank, parts;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(parts));
    const int tile = blockIdx.x / parts;
    const int all = p.K / MID_BK, k_lo = (int)(all * rank / parts), steps = (int)(all * (rank + 1) / parts) - k_lo;
    const uint32_t stage_bytes = MID_W_BYTES + p.cols * 128;
    const int tmem_cols = p.cols;                                // 32 or 64: a power of two

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(&tmem_slot)), "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (tid == 0) {
        for (int s = 0; s < MID_MAX_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&acc_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        fence_async_smem();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    pdl_launch_dependents();
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        // ---------------------------------------------------------------- copies
        if (lane == 0) {
            auto ask_w = [&](int i) {
                const int s = i % p.stages, col = (k_lo + i) * MID_BK;
                const uint32_t at = saddr(ring) + s * stage_bytes;
                mid_expect(&full[s], stage_bytes);
                const int row = tile * (EPI == MID_SILU ? 64 : 128);
                mid_tma(at, &w_map, col, row, &full[s]);
                mid_tma(at + MID_W_BYTES / 2, &w_map, col, EPI == MID_SILU ? p.I + row : row + 64, &full[s]);
            };
            auto ask_x = [&](int i) {
                const int s = i % p.stages;
                mid_tma(saddr(ring) + s * stage_bytes + MID_W_BYTES, &x_map, (k_lo + i) * MID_BK, 0, &full[s]);
            };
            const int early = min(p.stages, steps);
            for (int i = 0; i < early; ++i) ask_w(i);
            pdl_wait();
            asm volatile("fence.proxy.async;\n" ::: "memory");
            for (int i = 0; i < early; ++i) ask_x(i);
            for (int i = early; i < steps; ++i) {
                if (!mbar_wait(&empty[i % p.stages], ((i / p.stages) - 1) & 1)) break;
                ask_w(i);
                ask_x(i);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------------------------------------------------------- products
        if (lane == 0) {
            const uint32_t idesc = instr_desc(MID_ROWS, p.cols, false);
            for (int i = 0; i < steps; ++i) {
                const int s = i % p.stages;
                if (!mbar_wait(&full[s], (i / p.stages) & 1)) {
                    // the copies still in flight (none is asked for beyond these) must not land in what takes the ring's place
                    for (int j = i; j < min(steps, i + p.stages); ++j) mbar_wait(&full[j % p.stages], (j / p.stages) & 1);
                    break;
                }
                fence_after_sync();
                const uint32_t wa = saddr(ring) + s * stage_bytes, xa = wa + MID_W_BYTES;
#pragma unroll
                for (int kk = 0; kk < MID_BK / 16; ++kk)
                    mma_f16(tmem, smem_desc(wa + kk * 32, 16, 1024), smem_desc(xa + kk * 32, 16, 1024), idesc, i > 0 || kk > 0);
                mma_commit(&empty[s]);
            }
            mma_commit(&acc_full);
        }
        __syncwarp();
    } else if (warp >= 4) {
        // ---------------------------------------------------------------- this block's sums to shared memory (two warps
        // per 32 lanes of tensor memory, every other 32 tokens each)
        pdl_wait();
        if (p.part_in != nullptr) {
            const int n = p.K / 128;
            for (int t = tid - 128; t < p.cols; t += MID_THREADS - 128) {
                float s = 0.f;
#pragma unroll 8
                for (int b = 0; b < n; ++b) s += t < p.M ? __ldcg(p.part_in + (size_t)b * MID_PART + t) : 0.f;
                scale_of[t] = 1.0f / sqrtf(s / (float)p.K + p.eps);
            }
        }
        mbar_wait(&acc_full, 0);
        fence_after_sync();
        __syncwarp();
        const uint32_t from = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        float* to = partial + (warp & 3) * 32 + lane;
        for (int c = (warp >> 2) * 32 - 32; c < p.cols; c += 64) {
            float v[32];
            tmem_ld32(from + c, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) to[(c + i) * MID_ROWS] = v[i];
        }
        fence_before_sync();
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    fence_after_sync();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(tmem_cols));

    // ---------------------------------------------------------------- a warp per token: the sum of the parts, and what follows
    pdl_wait();
    for (int t = rank + parts * warp; t < p.M; t += parts * (MID_THREADS / 32)) {
        const uint32_t at = saddr(partial + t * MID_ROWS);
        const float s = p.part_in != nullptr ? scale_of[t] : 1.f;
        if (EPI == MID_SILU) {
            float2 g[MID_MAX_PARTS], u[MID_MAX_PARTS];
#pragma unroll
            for (int r = 0; r < MID_MAX_PARTS; ++r)
                if (r < parts) {
                    const uint32_t peer = mid_peer(at, r);
                    g[r] = mid_read2(peer + lane * 8);
                    u[r] = mid_read2(peer + 256 + lane * 8);
                }
            float2 gate = make_float2(0.f, 0.f), up = gate;
#pragma unroll
            for (int r = 0; r < MID_MAX_PARTS; ++r)
                if (r < parts) gate.x += g[r].x, gate.y += g[r].y, up.x += u[r].x, up.y += u[r].y;
            const int j = tile * 64 + lane * 2;
            if (j < p.I) {
                const float g0 = mid_round(gate.x * s), g1 = mid_round(gate.y * s), u0 = mid_round(up.x * s), u1 = mid_round(up.y * s);
                const float a0 = p.act == 1 ? gelu_tanh_f(g0) : silu_f(g0), a1 = p.act == 1 ? gelu_tanh_f(g1) : silu_f(g1);
                *reinterpret_cast<uint32_t*>((__nv_bfloat16*)p.Y + (size_t)t * p.ldy + j) = mid_pack(a0 * u0, a1 * u1);
            }
            continue;
        }
        const int n = tile * MID_ROWS + lane * 4;
        const bool in = n < p.N;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (EPI == MID_ADD && in) x = __ldcg(reinterpret_cast<const float4*>(p.resid + (size_t)t * p.N + n));
        float4 f[MID_MAX_PARTS];
#pragma unroll
        for (int r = 0; r < MID_MAX_PARTS; ++r)
            if (r < parts) f[r] = mid_read4(mid_peer(at, r) + lane * 16);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < MID_MAX_PARTS; ++r)
            if (r < parts) v.x += f[r].x, v.y += f[r].y, v.z += f[r].z, v.w += f[r].w;
        if (EPI == MID_ADD) {
            // the branch is rounded to bfloat16 first, as a separate product would store it
            x.x += mid_round(v.x * s), x.y += mid_round(v.y * s), x.z += mid_round(v.z * s), x.w += mid_round(v.w * s);
            if (in) {
                *reinterpret_cast<float4*>(p.resid + (size_t)t * p.N + n) = x;
                float w[4];
                if (p.norm_w_bf16) {
                    const uint2 b = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)p.norm_w + n);
                    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&b.x));
                    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&b.y));
                    w[0] = lo.x, w[1] = lo.y, w[2] = hi.x, w[3] = hi.y;
                } else {
                    const float4 b = *reinterpret_cast<const float4*>((const float*)p.norm_w + n);
                    w[0] = b.x, w[1] = b.y, w[2] = b.z, w[3] = b.w;
                }
                *reinterpret_cast<uint2*>(p.h + (size_t)t * p.N + n) = make_uint2(mid_pack(x.x * w[0], x.y * w[1]), mid_pack(x.z * w[2], x.w * w[3]));
            }
            const float ss = warp_sum(in ? (x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w) : 0.f);
            if (lane == 0) p.part_out[(size_t)tile * MID_PART + t] = ss;
        } else if (in) {
            if (EPI == MID_F32)
                *reinterpret_cast<float4*>((float*)p.Y + (size_t)t * p.ldy + n) = make_float4(v.x * s, v.y * s, v.z * s, v.w * s);
            else
                *reinterpret_cast<uint2*>((__nv_bfloat16*)p.Y + (size_t)t * p.ldy + n) = make_uint2(mid_pack(v.x * s, v.y * s), mid_pack(v.z * s, v.w * s));
        }
    }
    // nobody leaves while its sums are still read
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// Parts of k, of four steps of 64 at least: as many as still let the clusters of all tiles run at once (`at_once`: how many
// clusters of a size do).  A product of 6,144 rows and K = 4,096 with clusters of six, of which some have to wait for the
// first to end: 17.9 us at 24 tokens, against 12.5 with the clusters of five that this gives it.
int mid_parts(int tiles, int K, const int (&at_once)[MID_MAX_PARTS + 1]) {
    for (int parts = MID_MAX_PARTS; parts > 1; --parts)
        if (parts <= K / MID_BK / 4 && tiles <= at_once[parts]) return parts;
    return 1;
}

template <int EPI> int launch_mid(MidParams p, const void* X, int ldx, const void* W, cudaStream_t stream) {
    PL_REQUIRE(p.M >= 1 && p.M <= MID_MAX_COLS && p.N >= 1 && p.K >= MID_BK && p.K % MID_BK == 0 && ldx % 8 == 0,
               "gemm_mid: M=%d (1..%d) N=%d K=%d (a multiple of 64) ldx=%d", p.M, MID_MAX_COLS, p.N, p.K, ldx);
    PL_REQUIRE(p.part_in == nullptr || p.K % 128 == 0, "gemm_mid: a normed input of K=%d", p.K);
    struct AtOnce {
        int clusters[MID_MAX_PARTS + 1];
    };
    static PerDevice<AtOnce> found;
    constexpr size_t smem = MID_RING + 1024;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(MID_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    const AtOnce* at_once = found.get("gemm_mid", [&](AtOnce& a) {
        PL_CUDA(cudaFuncSetAttribute(gemm_mid_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        cfg.numAttrs = 1;
        for (int parts = 1; parts <= MID_MAX_PARTS; ++parts) {
            attr[0].val.clusterDim.x = parts;
            cfg.gridDim = dim3(parts);
            int n = 0;
            PL_CUDA(cudaOccupancyMaxActiveClusters(&n, gemm_mid_kernel<EPI>, &cfg));
            a.clusters[parts] = 2 * n;   // (it counts one block per SM for any kernel with tensor memory; two fit, and two run)
        }
        return 0;
    });
    if (!at_once) return 1;
    p.cols = (p.M + 31) / 32 * 32;
    const int stages = MID_RING / (MID_W_BYTES + p.cols * 128);
    p.stages = stages < MID_MAX_STAGES ? stages : MID_MAX_STAGES;
    const int w_rows = EPI == MID_SILU ? 2 * p.I : p.N;
    alignas(64) CUtensorMap x_map, w_map;
    if (!tensor_map_bf16(&x_map, X, (unsigned long long)p.M, (unsigned long long)p.K, (unsigned long long)ldx, (unsigned)p.cols) ||
        !tensor_map_bf16(&w_map, W, (unsigned long long)w_rows, (unsigned long long)p.K, (unsigned long long)p.K, 64))
        return 1;
    const int tiles = EPI == MID_SILU ? (p.I + 63) / 64 : (p.N + MID_ROWS - 1) / MID_ROWS;
    const int parts = mid_parts(tiles, p.K, at_once->clusters);
    cfg.gridDim = dim3(tiles * parts);
    attr[0].val.clusterDim.x = parts;
    static const bool no_pdl = getenv("PAGED_LLM_B200_NO_PDL") != nullptr;
    cfg.numAttrs = no_pdl ? 1 : 2;
    PL_CUDA(cudaLaunchKernelEx(&cfg, gemm_mid_kernel<EPI>, p, x_map, w_map));
    return 0;
}

}  // namespace

// Waits inside the kernel that gave up since the library was loaded (0 unless something is broken).
PL_EXPORT int pl_gemm_mid_timeouts() {
    int n = 0;
    if (cudaMemcpyFromSymbol(&n, tc::g_timeouts, sizeof(int)) != cudaSuccess) return -1;
    return n;
}

PL_EXPORT int pl_gemm_mid_max_tokens() { return MID_MAX_COLS; }

// part_in non-null: X is the h of a pl_gemm_mid_add and the product that of RMSNorm(x) * w (see the head of this file).
PL_EXPORT int pl_gemm_mid(const void* X, int ldx, const void* W, void* Y, int ldy, int M, int N, int K, int out_float32,
                          const float* part_in, float eps, cudaStream_t stream) {
    MidParams p = {};
    p.Y = Y, p.ldy = ldy, p.M = M, p.N = N, p.K = K, p.part_in = part_in, p.eps = eps;
    PL_REQUIRE(N % 4 == 0 && ldy >= N && ldy % 4 == 0 && ((uintptr_t)Y & 15) == 0, "gemm_mid: N=%d, ldy=%d and Y must allow wide stores", N, ldy);
    return out_float32 ? launch_mid<MID_F32>(p, X, ldx, W, stream) : launch_mid<MID_BF16>(p, X, ldx, W, stream);
}

// Y[M, I] = act(X Wg^T) * (X Wu^T), W = [Wg; Wu] of shape [2I, K]; act 0 SiLU, 1 the tanh form of GELU.
PL_EXPORT int pl_gemm_mid_silu(const void* X, int ldx, const void* W, void* Y, int ldy, int M, int I, int K, int act,
                               const float* part_in, float eps, cudaStream_t stream) {
    MidParams p = {};
    p.Y = Y, p.ldy = ldy, p.M = M, p.N = I, p.I = I, p.K = K, p.act = act, p.part_in = part_in, p.eps = eps;
    PL_REQUIRE(act == 0 || act == 1, "gemm_mid_silu: unknown activation %d", act);
    PL_REQUIRE(I % 2 == 0 && ldy >= I && ldy % 2 == 0 && ((uintptr_t)Y & 3) == 0, "gemm_mid_silu: I=%d, ldy=%d and Y must allow stores of pairs", I, ldy);
    return launch_mid<MID_SILU>(p, X, ldx, W, stream);
}

// resid[M, N] += bf16(X W^T) in float32; h = bf16(resid * norm_w); part_out[N / 128][256]: sums of squares of resid.
PL_EXPORT int pl_gemm_mid_add(const void* X, int ldx, const void* W, float* resid, void* h, const void* norm_w, int norm_w_dtype,
                              int M, int N, int K, float* part_out, cudaStream_t stream) {
    MidParams p = {};
    p.resid = resid, p.h = (__nv_bfloat16*)h, p.norm_w = norm_w, p.norm_w_bf16 = norm_w_dtype == PL_BF16;
    p.part_out = part_out, p.M = M, p.N = N, p.K = K;
    PL_REQUIRE(N % MID_ROWS == 0 && (((uintptr_t)resid | (uintptr_t)h | (uintptr_t)norm_w) & 15) == 0,
               "gemm_mid_add: N=%d must be a multiple of 128 and the stream, h and the norm's weight 16-byte aligned", N);
    return launch_mid<MID_ADD>(p, X, ldx, W, stream);
}
