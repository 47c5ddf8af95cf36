// Paged attention in true float32 on the CUDA cores, for prefill portions and
// for decoding, and the kernel that merges split partials (used by both
// precisions).  Scores, softmax and the weighted sum are float32 with expf.
#include "attention_common.cuh"

constexpr int F32_ROWS = 16;     // query rows per block
constexpr int F32_KEYS = 32;     // keys per iteration: one per lane
constexpr int F32_STAGES = 2;

// W floats from `src`, zeros without one (`any`: an address that may be named all the same).
template <int W> __device__ __forceinline__ void f32_copy(float* dst, const float* src, const float* any) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = src != nullptr ? 4 * W : 0;
    const float* from = src != nullptr ? src : any;
    if (W == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(from), "r"(bytes));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(from), "r"(bytes));
}

// grid: (items, kv heads); 128 threads = 4 warps, each owning 4 of the 16 rows.  A tile of 32 keys is brought in by
// 16-byte asynchronous copies while the one before is worked on; the 32 keys' addresses are looked up a tile earlier
// still.  What bounds it is the issue of shared-memory loads, so four rows share each: a lane reads four elements of
// its key for four rows' dot products, and the four rows' probabilities of a key as one float4 for its two columns of
// the weighted sum.  Every sum keeps its order (over the head's elements, over the keys).
// NC: pairs of columns per lane, ceil(d / 64).  VEC: the cache starts on a 16-byte boundary (and so do all rows); copies
// of 4 bytes where it does not.
template <int NC, bool VEC>
__global__ void __launch_bounds__(128) attn_f32_kernel(AttnParams p) {
    pdl_launch_dependents();
    const int padding = attn_padding_from(p);
    pdl_wait();
    attn_zero_padding<float>(p, padding);
    const AttnItem it = attn_decode_item(p, blockIdx.x / p.nkv, F32_ROWS, F32_KEYS);
    if (!it.valid) return;
    extern __shared__ __align__(16) float smem[];
    __shared__ const float* rows[F32_STAGES][F32_KEYS];   // each key of a tile: its address, or null (nothing there)
    const int d = p.d, kvh = blockIdx.x % p.nkv, G = p.nh / p.nkv, KP = d + 4;
    float* Qs = smem;                                 // [16][d]
    float* Ps = Qs + F32_ROWS * d;                    // [4 warps][32 keys][4 rows]
    float* Ks = Ps + 4 * F32_KEYS * 4;                // [2][32][d + 4]: four words of padding, no bank conflicts
    float* Vs = Ks + F32_STAGES * F32_KEYS * KP;      // [2][32][d]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* q = (const float*)p.q;
    const float* kv = (const float*)p.kv;
    const int* bt = p.block_table + (size_t)it.seq * p.bt_stride;
    const int n_tiles = (it.key_hi - it.key_lo + F32_KEYS - 1) / F32_KEYS;
    const size_t v_off = (size_t)p.nkv * p.ps * d;

    auto find_rows = [&](int t) {                     // threads 0..31
        int n = it.key_lo + t * F32_KEYS + tid;
        const float* src = nullptr;
        if (n < it.key_hi) {
            if (n >= p.keep_first) n += it.gap;
            const int page = bt[n / p.ps];            // (ps_shift is for the bfloat16 kernels)
            if (page >= 0) src = kv + ((((size_t)page * 2) * p.nkv + kvh) * p.ps + n % p.ps) * d;
        }
        rows[t % F32_STAGES][tid] = src;
    };
    auto load_tile = [&](int t) {
        constexpr int W = VEC ? 4 : 1;
        const int st = t % F32_STAGES, chunks = d / W;
        float* kd = Ks + st * F32_KEYS * KP;
        float* vd = Vs + st * F32_KEYS * d;
        for (int e = tid; e < F32_KEYS * chunks; e += 128) {
            const int j = e / chunks, c = (e - j * chunks) * W;
            const float* src = rows[st][j];
            f32_copy<W>(kd + j * KP + c, src != nullptr ? src + c : nullptr, kv);
            f32_copy<W>(vd + j * d + c, src != nullptr ? src + v_off + c : nullptr, kv);
        }
    };
    if (tid < F32_KEYS) {
        find_rows(0);
        find_rows(1);
    }
    for (int e = tid; e < F32_ROWS * d; e += 128) {
        const int r = e / d, c = e - r * d;
        const int R = it.row_base + r;
        float v = 0.f;
        if (R < it.rows_total) v = q[(size_t)(it.q0 + R / G) * p.q_stride + (kvh * G + R % G) * d + c];
        Qs[e] = v;
    }
    int pos[4], first[4];
    float m[4], l[4], acc[4][2 * NC], slope[4];
    const float* brow[4];
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) {
        const int R = it.row_base + warp * 4 + rr;
        pos[rr] = R < it.rows_total ? it.lk - it.nq + R / G : -1;
        first[rr] = attn_first_key(p, max(pos[rr], 0));
        slope[rr] = p.slopes != nullptr && R < it.rows_total ? p.slopes[kvh * G + R % G] : 0.f;
        brow[rr] = p.dist_bias != nullptr && R < it.rows_total ? p.dist_bias + (size_t)(kvh * G + R % G) * p.dist_len : nullptr;
        m[rr] = -INFINITY;
        l[rr] = 0.f;
#pragma unroll
        for (int cc = 0; cc < 2 * NC; ++cc) acc[rr][cc] = 0.f;
    }
    __syncthreads();
    if (n_tiles > 0) load_tile(0);
    asm volatile("cp.async.commit_group;\n" ::);

    for (int t = 0; t < n_tiles; ++t) {
        if (t + 1 < n_tiles) load_tile(t + 1);
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        if (t + 2 < n_tiles && tid < F32_KEYS) find_rows(t + 2);      // the tile at hand no longer needs its addresses
        const int st = t % F32_STAGES;
        const int place = it.key_lo + t * F32_KEYS + lane, n = place + (place >= p.keep_first ? it.gap : 0);
        if (pos[0] >= 0) {                                            // (a warp's rows beyond the last come last)
            const float4* kr = reinterpret_cast<const float4*>(Ks + (st * F32_KEYS + lane) * KP);
            const float4* qr = reinterpret_cast<const float4*>(Qs + warp * 4 * d);
            float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int c = 0; c < d / 4; ++c) {
                const float4 k4 = kr[c];
#pragma unroll
                for (int rr = 0; rr < 4; ++rr) {
                    const float4 q4 = qr[rr * (d / 4) + c];
                    s[rr] = fmaf(q4.x, k4.x, s[rr]);
                    s[rr] = fmaf(q4.y, k4.y, s[rr]);
                    s[rr] = fmaf(q4.z, k4.z, s[rr]);
                    s[rr] = fmaf(q4.w, k4.w, s[rr]);
                }
            }
            float pj[4];
            unsigned live = 0u;                                       // rows that see a key of this tile (uniform per warp)
#pragma unroll
            for (int rr = 0; rr < 4; ++rr) {
                pj[rr] = 0.f;
                if (pos[rr] < 0) continue;                            // uniform per warp
                const float sc = attn_score(p, s[rr], slope[rr], n, pos[rr], brow[rr]);
                const bool vis = place < it.key_hi && n <= pos[rr] && (n >= first[rr] || n < p.keep_first);
                const float m_new = fmaxf(m[rr], warp_max(vis ? sc : -INFINITY));
                if (m_new == -INFINITY) continue;
                if (__any_sync(0xffffffffu, vis)) live |= 1u << rr;
                pj[rr] = vis ? expf(sc - m_new) : 0.f;
                const float alpha = m[rr] == -INFINITY ? 0.f : expf(m[rr] - m_new);
                l[rr] = l[rr] * alpha + warp_sum(pj[rr]);
                m[rr] = m_new;
#pragma unroll
                for (int cc = 0; cc < 2 * NC; ++cc) acc[rr][cc] *= alpha;
            }
            float4* ps = reinterpret_cast<float4*>(Ps) + warp * F32_KEYS;
            ps[lane] = make_float4(pj[0], pj[1], pj[2], pj[3]);
            __syncwarp();
            const float* vr = Vs + st * F32_KEYS * d + lane * 2;
            auto weigh = [&](int rr, float w, const float2& v, int cc) {
                acc[rr][2 * cc] = fmaf(w, v.x, acc[rr][2 * cc]);
                acc[rr][2 * cc + 1] = fmaf(w, v.y, acc[rr][2 * cc + 1]);
            };
            if (live == 15u) {
#pragma unroll 8
                for (int j = 0; j < F32_KEYS; ++j) {
                    const float4 w = ps[j];
#pragma unroll
                    for (int cc = 0; cc < NC; ++cc) {
                        if (lane * 2 + 64 * cc >= d) continue;
                        const float2 v = *reinterpret_cast<const float2*>(vr + j * d + 64 * cc);
                        weigh(0, w.x, v, cc), weigh(1, w.y, v, cc), weigh(2, w.z, v, cc), weigh(3, w.w, v, cc);
                    }
                }
            } else {
                // a row that sees no key of the tile takes no part (its zeros times a value that is not finite would be NaN)
                for (int j = 0; j < F32_KEYS; ++j) {
                    const float4 w = ps[j];
#pragma unroll
                    for (int cc = 0; cc < NC; ++cc) {
                        if (lane * 2 + 64 * cc >= d) continue;
                        const float2 v = *reinterpret_cast<const float2*>(vr + j * d + 64 * cc);
                        if (live & 1) weigh(0, w.x, v, cc);
                        if (live & 2) weigh(1, w.y, v, cc);
                        if (live & 4) weigh(2, w.z, v, cc);
                        if (live & 8) weigh(3, w.w, v, cc);
                    }
                }
            }
        }
        __syncthreads();                                              // the stage may be filled again
    }

#pragma unroll
    for (int rr = 0; rr < 4; ++rr) {
        if (pos[rr] < 0) continue;
        const int R = it.row_base + warp * 4 + rr;
        const int tok = R / G, head = kvh * G + R % G;
        float* o;
        float f = 1.f;
        if (it.splits <= 1) {
            o = (float*)p.out + (size_t)(it.q0 + tok) * p.out_stride + head * d;
            const float lsum = l[rr] + attn_sink_term(p, head, m[rr]);
            f = lsum > 0.f ? 1.0f / lsum : 0.f;
        } else {
            float* part = attn_partial(p, it.scratch_base + tok, head, it.split);
            if (lane == 0) {
                part[0] = m[rr];
                part[1] = l[rr];
            }
            o = part + 2;
        }
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
            const int c = lane * 2 + 64 * cc;
            if (c < d) {
                o[c] = acc[rr][2 * cc] * f;
                o[c + 1] = acc[rr][2 * cc + 1] * f;
            }
        }
    }
}

// Merge of split partials.  grid: (small items, heads); the block of an item's
// split 0 merges all splits of every token of its request for one head.
template <typename TO>
__global__ void attn_combine_kernel(AttnParams p) {
    pdl_launch_dependents();
    pdl_wait();
    if ((int)blockIdx.x >= p.n_work) return;
    const int4 w = p.work[blockIdx.x];
    if (w.x < 0 || w.z != 0 || w.w <= 1) return;
    const int head = blockIdx.y, splits = w.w, d = p.d;
    const int q0 = p.cu_q[w.x], nq = p.cu_q[w.x + 1] - q0;
    for (int i = 0; i < nq; ++i) {
        float M = -INFINITY;
        for (int j = 0; j < splits; ++j) M = fmaxf(M, attn_partial(p, w.y + i, head, j)[0]);
        float L = 0.f;
        for (int j = 0; j < splits; ++j) {
            const float* part = attn_partial(p, w.y + i, head, j);
            if (part[0] != -INFINITY) L += part[1] * expf(part[0] - M);
        }
        L += attn_sink_term(p, head, M);
        const float inv = L > 0.f ? 1.0f / L : 0.f;
        TO* o = (TO*)p.out + (size_t)(q0 + i) * p.out_stride + head * d;
        for (int c = threadIdx.x; c < d; c += blockDim.x) {
            float a = 0.f;
            for (int j = 0; j < splits; ++j) {
                const float* part = attn_partial(p, w.y + i, head, j);
                if (part[0] != -INFINITY) a += part[2 + c] * expf(part[0] - M);
            }
            o[c] = from_float<TO>(a * inv);
        }
    }
}

int pl_attn_check(const AttnParams& p, const char* who) {
    PL_REQUIRE(p.nh > 0 && p.nkv > 0 && p.nh % p.nkv == 0, "%s: %d query heads on %d kv heads", who, p.nh, p.nkv);
    PL_REQUIRE(p.d > 0 && p.d % 16 == 0 && p.d <= 256, "%s: head_dim=%d must be a multiple of 16 up to 256", who, p.d);
    PL_REQUIRE(p.ps > 0, "%s: page_size=%d", who, p.ps);
    PL_REQUIRE(p.window >= 0, "%s: window=%d", who, p.window);
    PL_REQUIRE(p.chunk >= 0, "%s: chunk=%d", who, p.chunk);
    PL_REQUIRE(p.keep_first == 0 || (p.keep_first > 0 && p.window > 0 && p.chunk == 0),
               "%s: keep_first=%d goes with a window (%d) and without chunks (%d)", who, p.keep_first, p.window, p.chunk);
    PL_REQUIRE(p.max_splits >= 1, "%s: max_splits=%d", who, p.max_splits);
    PL_REQUIRE(p.softcap >= 0.f, "%s: softcap=%f must not be negative", who, (double)p.softcap);
    PL_REQUIRE(p.dist_bias == nullptr || p.dist_len > 0, "%s: a bias by distance of %d entries", who, p.dist_len);
    return 0;
}

template <int NC, bool VEC> static int launch_attn_f32(const AttnParams& p, cudaStream_t stream) {
    const size_t smem = ((size_t)F32_ROWS * p.d + 4 * F32_KEYS * 4 + F32_STAGES * F32_KEYS * (2 * p.d + 4)) * sizeof(float);
    constexpr size_t most = ((size_t)F32_ROWS * 64 * NC + 4 * F32_KEYS * 4 + F32_STAGES * F32_KEYS * (2 * 64 * NC + 4)) * sizeof(float);
    static PerDevice<char> ready;
    if (!ready.get("attention_f32", [&](char&) {
            PL_CUDA(cudaFuncSetAttribute(attn_f32_kernel<NC, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
            return 0;
        }))
        return 1;
    PL_CUDA(launch_pdl(attn_f32_kernel<NC, VEC>, dim3(p.n_work * p.nkv), dim3(128), smem, stream, p));
    return 0;
}

template <bool VEC> static int dispatch_attn_f32(const AttnParams& p, cudaStream_t stream) {
    return p.d <= 64 ? launch_attn_f32<1, VEC>(p, stream) : p.d <= 128 ? launch_attn_f32<2, VEC>(p, stream) : launch_attn_f32<4, VEC>(p, stream);
}

PL_EXPORT int pl_attention_f32(const AttnParams* params, cudaStream_t stream) {
    AttnParams p = *params;
    if (p.n_work == 0) return 0;
    if (int rc = pl_attn_check(p, "attention_f32")) return rc;
    return ((uintptr_t)p.kv & 15) == 0 ? dispatch_attn_f32<true>(p, stream) : dispatch_attn_f32<false>(p, stream);
}

PL_EXPORT int pl_attention_combine(const AttnParams* params, int out_dtype, cudaStream_t stream) {
    AttnParams p = *params;
    if (p.n_work == 0) return 0;
    if (int rc = pl_attn_check(p, "attention_combine")) return rc;
    const int threads = p.d <= 64 ? 64 : (p.d <= 128 ? 128 : 256);
    if (out_dtype == PL_F32)
        PL_CUDA(launch_pdl(attn_combine_kernel<float>, dim3(p.n_work, p.nh), dim3(threads), 0, stream, p));
    else if (out_dtype == PL_BF16)
        PL_CUDA(launch_pdl(attn_combine_kernel<__nv_bfloat16>, dim3(p.n_work, p.nh), dim3(threads), 0, stream, p));
    else
        return pl_fail("attention_combine: unknown dtype %d", out_dtype);
    return 0;
}
