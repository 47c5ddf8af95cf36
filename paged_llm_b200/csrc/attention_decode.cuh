// Decode attention for head sizes 64 and 128 without score modifiers, windows or chunks: what a Llama decode step runs.
//
// What bounds it should be the read of the cached keys and values; what did bound it was issue slots.  With the queries
// as the 16 rows of mma.sync (attn_bf16_kernel), a warp spent some 480 instructions on 16 keys: half of each product and
// of each softmax on rows that pad the few query heads of a kv head, the rest on the addresses of 16-byte copies and on
// masks.  Here
//   - the keys are the 16 rows and the queries the 8 columns (NT tiles of them): S^T = K Q^T and O^T += V^T P^T, so that
//     eight query heads per kv head fill the product; P^T comes out of S^T's fragments by movmatrix;
//   - a warp's tile of 16 keys is one box per 64 columns of the cache seen as a matrix of rows (page, K or V, kv head,
//     slot): TMA copies it, swizzled, into the warp's own ring (no barrier over the block; one mbarrier per stage);
//     a warp looks the pages of 32 tiles up at once, a tile per lane;
//   - the running maximum is moved only when a score exceeds it by 2^8 (probabilities stay below 256 and are
//     rounded relative to their size), so that the usual tile needs one vote and no shuffle.
// Rows of a box behind the range may hold anything: their scores are masked and their values zeroed.
#pragma once

#include "tcgen05.cuh"
#include "tensor_map.cuh"

namespace dec {

constexpr float LOG2E = 1.4426950408889634f;
constexpr int KEYS = 16;                        // keys of a warp's tile
constexpr float LAZY = 8.f;                     // how far a score may exceed the running maximum, in base-2 units

__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void box_load(uint32_t dst, const CUtensorMap* map, int col, int row, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
        "l"(map), "r"(col), "r"(row), "r"(bar)
        : "memory");
}

template <int D, int NT, int NW, int STAGES>
struct Shape {
    static constexpr int HALVES = D / 64, HALF = KEYS * 128, SIDE = HALVES * HALF, TILE = 2 * SIDE;   // bytes: K, then V
    static constexpr int BM = 8 * NT, QP = D + 8, OP = D + 4, THREADS = 32 * NW;
    static constexpr int RING = NW * STAGES * TILE, Q_BYTES = BM * QP * 2;
    static constexpr int MERGE = NW * BM * OP * 4 + NW * BM * 8 + BM * (D + 2) * 4;       // red_o, red_ml, cpart in the ring
    static_assert(MERGE <= RING && BM * 32 * 8 <= RING, "the merge reuses the ring");
    static constexpr size_t smem(bool rope) { return 1024 + RING + (rope ? TILE : 0) + Q_BYTES; }
};

// CLUSTER, ROPE: as in attn_bf16_kernel.
template <int D, int NT, int NW, int STAGES, bool CLUSTER, bool ROPE>
__global__ void __launch_bounds__(32 * NW) attn_decode_kernel(AttnParams p, const __grid_constant__ CUtensorMap kv_map) {
    using S = Shape<D, NT, NW, STAGES>;
    extern __shared__ unsigned char dec_smem[];
    __shared__ uint64_t full[NW][STAGES];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    // lengths, lists, block tables and all keys but the step's own are older than the step: they are read before the wait
    const AttnItem it = CLUSTER ? attn_cluster_item(p, blockIdx.x / (p.cluster * p.nkv), blockIdx.x % p.cluster, p.cluster)
                                : attn_decode_item(p, blockIdx.x / p.nkv, 16, 32);
    const int padding = attn_padding_from(p);
    if (!it.valid) {                                        // the same for all blocks of a cluster
        pdl_wait();
        attn_zero_padding<__nv_bfloat16>(p, padding);
        return;
    }
    unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)dec_smem + 1023) & ~(uintptr_t)1023);
    unsigned char* own = ring + S::RING;                    // (ROPE) the step's own keys and values, laid out as a tile
    __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(ring + S::RING + (ROPE ? S::TILE : 0));     // [BM][QP]
    const uint32_t ring_at = tc::saddr(ring) + warp * STAGES * S::TILE;

    const int kvh = CLUSTER ? (blockIdx.x / p.cluster) % p.nkv : blockIdx.x % p.nkv, G = p.nh / p.nkv;
    const __nv_bfloat16* q = (const __nv_bfloat16*)p.q;
    const int* bt = p.block_table + (size_t)it.seq * p.bt_stride;
    const int own_lo = it.lk - it.nq;                       // the step's own keys: written by the kernel in front, or here
    const int hi = ROPE ? min(it.key_hi, max(own_lo, it.key_lo)) : it.key_hi;      // end of the keys that come by TMA

    // ---- the warp's tiles: NW apart from one another
    const int tiles = (hi - it.key_lo + KEYS - 1) / KEYS;
    const int count = tiles > warp ? (tiles - warp + NW - 1) / NW : 0;
    auto tile_key = [&](int i) { return it.key_lo + (warp + i * NW) * KEYS; };
    auto rows_of = [&](int i0) {                            // lane l: first row of K of tile i0 + l in the cache
        const int key = tile_key(i0 + lane);
        if (key >= hi) return -KEYS;
        const int page = bt[p.ps_shift >= 0 ? key >> p.ps_shift : key / p.ps];
        const int slot = p.ps_shift >= 0 ? key & (p.ps - 1) : key % p.ps;
        return page >= 0 && page < p.num_pages ? (page * 2 * p.nkv + kvh) * p.ps + slot : -KEYS;    // (outside: reads zeros)
    };
    int rows = rows_of(0);
    const int v_rows = p.nkv * p.ps;
    auto ask = [&](int i) {                                 // all lanes of the warp
        if (i > 0 && (i & 31) == 0) rows = rows_of(i);
        const int row = __shfl_sync(0xffffffffu, rows, i & 31);
        if (lane == 0) {
            const int s = i % STAGES;
            const uint32_t bar = tc::saddr(&full[warp][s]), at = ring_at + s * S::TILE;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(S::TILE) : "memory");
#pragma unroll
            for (int h = 0; h < S::HALVES; ++h) {
                box_load(at + h * S::HALF, &kv_map, h * 64, row, bar);
                box_load(at + S::SIDE + h * S::HALF, &kv_map, h * 64, row >= 0 ? row + v_rows : row, bar);
            }
        }
    };
    if (lane == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) tc::mbar_init(&full[warp][s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        tc::fence_async_smem();
    }
    __syncwarp();
    int asked = 0;
    for (; asked < min(STAGES, count) && (ROPE || tile_key(asked) + KEYS <= own_lo); ++asked) ask(asked);

    // (ROPE) the angles of the pairs that this thread rotates first, from a constant table: chunk c8 of the first half of
    // a head with its partner in the second half
    constexpr int HC = D / 16;
    float4 angle[4];
    const int r0 = tid / HC, pos0 = it.lk - it.nq + r0 / G;
    const bool rotate = ROPE && r0 < S::BM && r0 < it.rows_total && pos0 >= 0 && pos0 < p.rope_len;
    if (rotate) {
        const float4* cs = reinterpret_cast<const float4*>(p.rope_table + (size_t)pos0 * (D / 2) + (tid % HC) * 8);
#pragma unroll
        for (int k = 0; k < 4; ++k) angle[k] = __ldg(cs + k);
    }
    pdl_wait();
    attn_zero_padding<__nv_bfloat16>(p, padding);
    if (!ROPE) {
        asm volatile("fence.proxy.async;\n" ::: "memory");        // the kernel in front wrote them by ordinary stores
        for (; asked < min(STAGES, count); ++asked) ask(asked);
    }

    // ---- queries, and the step's own keys
    if (ROPE) {
        for (int e = tid; e < S::BM * HC; e += S::THREADS) {
            const int r = e / HC, c8 = e % HC;
            uint4 lo = make_uint4(0, 0, 0, 0), hi4 = lo;
            if (r < it.rows_total) {
                const __nv_bfloat16* src = q + (size_t)(it.q0 + r / G) * p.q_stride + (kvh * G + r % G) * D + c8 * 8;
                lo = *reinterpret_cast<const uint4*>(src);
                hi4 = *reinterpret_cast<const uint4*>(src + D / 2);
                if (e != tid) rotate_pair(lo, hi4, p.rope_table, p.rope_len, it.lk - it.nq + r / G, D, c8 * 8);
                else if (rotate) rotate_by(lo, hi4, angle);
            }
            *reinterpret_cast<uint4*>(Qs + r * S::QP + c8 * 8) = lo;
            *reinterpret_cast<uint4*>(Qs + r * S::QP + D / 2 + c8 * 8) = hi4;
        }
    } else {
        for (int e = tid; e < S::BM * (D / 8); e += S::THREADS) {
            const int r = e / (D / 8), c8 = e % (D / 8);
            uint4 v = make_uint4(0, 0, 0, 0);
            if (r < it.rows_total) v = *reinterpret_cast<const uint4*>(q + (size_t)(it.q0 + r / G) * p.q_stride + (kvh * G + r % G) * D + c8 * 8);
            *reinterpret_cast<uint4*>(Qs + r * S::QP + c8 * 8) = v;
        }
    }
    // 16-byte chunk c of row r of a tile's side, as TMA's 128-byte swizzle lays it
    auto chunk_at = [](int r, int c) { return (c / 8) * S::HALF + r * 128 + (((c & 7) ^ (r & 7)) << 4); };
    const bool own_here = ROPE && it.key_hi > hi;
    if (own_here) {
        // rotated keys and values straight from the projection, also written to their page slots, by the threads behind
        // those that fetch the queries; rows without a key are zeroed
        for (int e = S::THREADS - 1 - tid; e < KEYS * HC; e += S::THREADS) {
            const int j = e / HC, c8 = e % HC;
            uint4 klo = make_uint4(0, 0, 0, 0), khi = klo, vlo = klo, vhi = klo;
            if (j < it.key_hi - hi) {
                const int n = hi + j;                                      // position of the key
                const __nv_bfloat16* row = q + (size_t)(it.q0 + n - own_lo) * p.q_stride;
                const __nv_bfloat16* ks = row + (size_t)(p.nh + kvh) * D + c8 * 8;
                const __nv_bfloat16* vs = row + (size_t)(p.nh + p.nkv + kvh) * D + c8 * 8;
                klo = *reinterpret_cast<const uint4*>(ks);
                khi = *reinterpret_cast<const uint4*>(ks + D / 2);
                vlo = *reinterpret_cast<const uint4*>(vs);
                vhi = *reinterpret_cast<const uint4*>(vs + D / 2);
                rotate_pair(klo, khi, p.rope_table, p.rope_len, n, D, c8 * 8);
                const int page = bt[n / p.ps];
                if (page >= 0 && page < p.num_pages) {
                    __nv_bfloat16* dst = (__nv_bfloat16*)p.kv + (((size_t)page * 2 * p.nkv + kvh) * p.ps + n % p.ps) * D + c8 * 8;
                    *reinterpret_cast<uint4*>(dst) = klo;
                    *reinterpret_cast<uint4*>(dst + D / 2) = khi;
                    *reinterpret_cast<uint4*>(dst + (size_t)v_rows * D) = vlo;
                    *reinterpret_cast<uint4*>(dst + (size_t)v_rows * D + D / 2) = vhi;
                }
            }
            *reinterpret_cast<uint4*>(own + chunk_at(j, c8)) = klo;
            *reinterpret_cast<uint4*>(own + chunk_at(j, HC + c8)) = khi;
            *reinterpret_cast<uint4*>(own + S::SIDE + chunk_at(j, c8)) = vlo;
            *reinterpret_cast<uint4*>(own + S::SIDE + chunk_at(j, HC + c8)) = vhi;
        }
    }
    __syncthreads();

    const int g = lane >> 2, t4 = lane & 3;
    uint32_t qf[NT][D / 16][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            const __nv_bfloat16* src = Qs + (nt * 8 + g) * S::QP + kk * 16 + 2 * t4;
            qf[nt][kk][0] = *reinterpret_cast<const uint32_t*>(src);
            qf[nt][kk][1] = *reinterpret_cast<const uint32_t*>(src + 8);
        }
    float m_run[NT][2], m_use[NT][2], l_run[NT][2], o[D / 16][NT][4];      // of columns 2 t4, 2 t4 + 1 (the maxima: the same in all lanes)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) m_run[nt][e] = -INFINITY, m_use[nt][e] = 0.f, l_run[nt][e] = 0.f;
#pragma unroll
    for (int mt = 0; mt < D / 16; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[mt][nt][e] = 0.f;
    const float scale2 = p.scale * LOG2E;
    const int row_k = (lane & 7) + ((lane >> 3) & 1) * 8, col_k = lane >> 4;        // ldmatrix: K as it lies,
    const int row_v = (lane & 7) + (lane >> 4) * 8, col_v = (lane >> 3) & 1;        // V transposed
    const uint32_t x = lane & 7;

    // the keys [key, key + 16) that lie at `at` (K, then V); those from `end` on are not there
    auto take = [&](uint32_t at, int key, int end) {
        float s[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[nt][e] = 0.f;
        const uint32_t k_at = at + row_k * 128, v_at = at + S::SIDE + row_v * 128;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            uint32_t a[4];
            ldsm(a, k_at + (kk / 4) * S::HALF + ((((kk & 3) * 2 + col_k) ^ x) << 4));
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_bf16(s[nt], a, qf[nt][kk][0], qf[nt][kk][1]);
        }
        if (key + KEYS > end || key + KEYS - 1 > own_lo) {                 // a key that some row does not see
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int n = key + g + (e >> 1) * 8, pos = own_lo + (nt * 8 + 2 * t4 + (e & 1)) / G;
                    if (n >= end || n > pos) s[nt][e] = -INFINITY;
                }
        }
        bool above = false;
        float top[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                top[nt][e] = fmaxf(s[nt][e], s[nt][2 + e]) * scale2;
                above |= top[nt][e] > m_run[nt][e] + LAZY;
            }
        if (__any_sync(0xffffffffu, above)) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float m = top[nt][e];
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
                    m = fmaxf(m, m_run[nt][e]);
                    const float alpha = m_run[nt][e] == -INFINITY ? 0.f : fast_exp2(m_run[nt][e] - m);
                    m_run[nt][e] = m;
                    m_use[nt][e] = m == -INFINITY ? 0.f : m;
                    l_run[nt][e] *= alpha;
#pragma unroll
                    for (int mt = 0; mt < D / 16; ++mt) {
                        o[mt][nt][e] *= alpha;
                        o[mt][nt][2 + e] *= alpha;
                    }
                }
        }
        uint32_t pb[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            float pr[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                pr[e] = fast_exp2(fmaf(s[nt][e], scale2, -m_use[nt][e & 1]));
                l_run[nt][e & 1] += pr[e];
            }
            pb[nt][0] = transpose8x8(pack_bf16(pr[0], pr[1]));
            pb[nt][1] = transpose8x8(pack_bf16(pr[2], pr[3]));
        }
#pragma unroll
        for (int mt = 0; mt < D / 16; ++mt) {
            uint32_t a[4];
            ldsm_trans(a, v_at + (mt / 4) * S::HALF + ((((mt & 3) * 2 + col_v) ^ x) << 4));
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_bf16(o[mt][nt], a, pb[nt][0], pb[nt][1]);
        }
    };

    if (own_here && warp == NW - 1) take(tc::saddr(own), hi, it.key_hi);       // while the first tile is still on its way
    for (int i = 0; i < count; ++i) {
        const int s = i % STAGES, key = tile_key(i);
        if (!__all_sync(0xffffffffu, tc::mbar_wait(&full[warp][s], (i / STAGES) & 1))) {
            // a copy that never arrived (counted, see kernel_timeouts): the others in flight must not land in what takes the
            // ring's place
            for (int j = i; j < asked; ++j) tc::mbar_wait(&full[warp][j % STAGES], (j / STAGES) & 1);
            break;
        }
        const uint32_t at = ring_at + s * S::TILE;
        if (key + KEYS > hi) {                              // the last tile: what lies behind the range must not be a NaN
            unsigned char* v = ring + (size_t)warp * STAGES * S::TILE + s * S::TILE + S::SIDE;
            for (int e = lane; e < (key + KEYS - hi) * (D / 8); e += 32)
                *reinterpret_cast<uint4*>(v + chunk_at(hi - key + e / (D / 8), e % (D / 8))) = make_uint4(0, 0, 0, 0);
            __syncwarp();
        }
        take(at, key, hi);
        __syncwarp();
        if (asked < count) ask(asked++);
    }

    // ---- merge
    __syncthreads();                                        // all tiles are used up: the ring is free
    float* red_o = reinterpret_cast<float*>(ring);                             // [NW][BM][OP]
    float* red_ml = red_o + NW * S::BM * S::OP;                                // [NW][BM][2]
    float* cpart = red_ml + NW * S::BM * 2;                                    // [BM][D + 2]
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float l = l_run[nt][e];
            l += __shfl_xor_sync(0xffffffffu, l, 4);
            l += __shfl_xor_sync(0xffffffffu, l, 8);
            l += __shfl_xor_sync(0xffffffffu, l, 16);
            const int r = warp * S::BM + nt * 8 + 2 * t4 + e;
            if (g == 0) {
                red_ml[r * 2] = m_run[nt][e];
                red_ml[r * 2 + 1] = l;
            }
#pragma unroll
            for (int mt = 0; mt < D / 16; ++mt) {
                red_o[r * S::OP + mt * 16 + g] = o[mt][nt][e];
                red_o[r * S::OP + mt * 16 + g + 8] = o[mt][nt][2 + e];
            }
        }
    attn_merge<D, S::BM, NW, S::THREADS, S::OP, CLUSTER>(p, it, kvh, red_ml, red_o, cpart, ring);
}

// What the kernel takes; anything else runs in attn_bf16_kernel.
inline bool takes(const AttnParams& p) {
    return (p.cluster > 0 || p.is_small) && (p.d == 64 || p.d == 128) && p.window <= 0 && p.chunk <= 0 && p.softcap <= 0.f &&
           p.slopes == nullptr && p.dist_bias == nullptr && p.keep_first <= 0 && p.scale > 0.f && p.ps % KEYS == 0 &&
           p.num_pages > 0 && (long long)p.num_pages * 2 * p.nkv * p.ps < (1ll << 31) - KEYS && p.nh / p.nkv <= 16;
}

template <int D, int NT, int NW, int STAGES, bool CLUSTER, bool ROPE>
int launch_as(const AttnParams& p, cudaStream_t stream) {
    auto kernel = attn_decode_kernel<D, NT, NW, STAGES, CLUSTER, ROPE>;
    constexpr size_t smem = Shape<D, NT, NW, STAGES>::smem(ROPE);
    static bool attr_set[kAttnMaxDevices] = {};
    int dev = 0;
    PL_CUDA(cudaGetDevice(&dev));
    PL_REQUIRE(dev >= 0 && dev < kAttnMaxDevices, "attention_decode: device index %d is out of range", dev);
    if (!attr_set[dev]) {
        PL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (CLUSTER) PL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));    // up to 16 blocks
        attr_set[dev] = true;
    }
    alignas(64) CUtensorMap map;
    if (!tensor_map_bf16(&map, p.kv, (unsigned long long)p.num_pages * 2 * p.nkv * p.ps, D, D, KEYS)) return 1;
    PL_REQUIRE(!CLUSTER || p.cluster <= 16, "attention_decode: clusters of 1 to 16 blocks, not %d", p.cluster);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.n_work * p.nkv * (CLUSTER ? p.cluster : 1));
    cfg.blockDim = dim3(32 * NW);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CLUSTER ? p.cluster : 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    static const bool no_pdl = getenv("PAGED_LLM_B200_NO_PDL") != nullptr;
    cfg.numAttrs = no_pdl ? 1 : 2;
    PL_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, map));
    return 0;
}

template <int D, int NW, int STAGES>
int launch_shape(const AttnParams& p, cudaStream_t stream) {
    const bool one = p.small_rows > 0 && p.small_rows <= 8;
    if (p.cluster > 0) {
        if (p.rope_table != nullptr) return one ? launch_as<D, 1, NW, STAGES, true, true>(p, stream) : launch_as<D, 2, NW, STAGES, true, true>(p, stream);
        return one ? launch_as<D, 1, NW, STAGES, true, false>(p, stream) : launch_as<D, 2, NW, STAGES, true, false>(p, stream);
    }
    if (p.rope_table != nullptr) return one ? launch_as<D, 1, NW, STAGES, false, true>(p, stream) : launch_as<D, 2, NW, STAGES, false, true>(p, stream);
    return one ? launch_as<D, 1, NW, STAGES, false, false>(p, stream) : launch_as<D, 2, NW, STAGES, false, false>(p, stream);
}

template <int D>
int launch(const AttnParams& p, cudaStream_t stream) {
    PL_REQUIRE(p.rope_table == nullptr || p.rope_len > 0, "attention_decode: bad rotary table");
    // Two blocks per SM of three stages in both shapes, but for steps of very many requests (below): three stages win up to 4 us
    // where blocks walk long ranges, two win up to 3 us where many blocks walk short ones.  Measured, us per layer; attn_bf16_kernel, one range per request, before:
    //                                                     before   here   two stages   the bytes at 6.45 TB/s
    //   64 requests x 641 keys, 4 kv heads of 64            14.4    9.8        11.0     6.5
    //   64 x 2,048                                          33.4   23.4        27.2    20.8
    //   27 of 131 to 3,500 keys, 8 kv heads of 64           41.9   22.0        23.9    15.6   (even ranges)
    //   131 of 70 to 777 keys, 4 kv heads of 64             27.5   17.6        14.4     8.8
    //   8 x 4,096, 4 kv heads of 64                         17.5   13.0        14.2     5.2
    //   16 x 3,000, 8 kv heads of 128                       47.3   37.0        40.3    30.5
    //   8 x 1,032 to 1,277, 8 kv heads of 128               19.3   13.2        12.9     5.9
    //   1 x 641, 4 kv heads of 64                            5.5    5.6         5.4     0.1
    // Head size 64 with four warps of four stages: 11.0 at the first, 22.5 at the third; eight warps of four stages
    // (one block per SM): 14.7 and 34.
    //
    // Steps of so many requests that blocks come and go: with two stages three blocks fit an SM (80 registers: up to eight
    // query rows), and the list is cut for as many (CudaOps._three_blocks says when).  us per layer, three stages / two, with
    // contexts all of one length, and from a quarter of it to seven quarters:
    //                             100          500         1,200        2,000         3,000         4,000
    //   112 x 8     alike      17.9  15.0   32.0  27.6   52.6  52.1   80.4  78.9   113.2 112.1   144.9 143.9
    //               mixed      18.2  15.4   30.5  27.1   53.0  48.9   78.3  73.2   108.5 104.4   140.6 137.0
    //   192 x 8     alike      26.6  21.0   48.6  41.0   82.2  78.1  124.9 120.8   179.7 174.1   234.0 228.8
    //               mixed      28.2  22.3   49.5  42.7   85.5  79.4  125.9 120.3   178.7 173.6   230.9 225.3
    //   256 x 4     alike      19.5  16.3   35.9  31.7   59.2  58.1   87.5  86.0   123.4 122.4   159.2 159.2
    //               mixed      20.5  17.4   36.9  32.3   60.9  56.8   88.1  83.4   123.4 119.2   157.7 154.1
    //    33 x 32    alike      19.1  15.9   35.8  31.7   59.9  57.8   87.3  86.3   121.6 123.1   159.0 159.5
    // Fewer pairs in a graph of as many (the rest of its requests are empty):
    //    97 x 8     alike      14.6  11.8   28.9  23.8   45.1  43.5   67.6  64.5    94.7  92.2   120.8 119.3
    //               mixed      16.1  13.2   27.9  23.6   45.0  41.0   66.1  63.0    91.6  90.6   119.3 120.3
    // A tenth of the requests with six times the keys of the others, 8 kv heads, longest context 4,800: 112 50.2 49.7, 192 80.9
    // 75.8; longest 16,000: 97 122.4 124.9, 112 140.8 142.3, 192 230.8 230.8.
    if constexpr (D == 64) {
        if (p.three_blocks && p.cluster <= 0 && p.small_rows > 0 && p.small_rows <= 8)
            return p.rope_table != nullptr ? launch_as<D, 1, 8, 2, false, true>(p, stream) : launch_as<D, 1, 8, 2, false, false>(p, stream);
    }
    if constexpr (D == 64) return launch_shape<D, 8, 3>(p, stream);
    else return launch_shape<D, 4, 3>(p, stream);
}

}  // namespace dec
