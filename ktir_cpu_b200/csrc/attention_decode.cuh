// Attention of a few query rows over a long context (decode), head_dim 128; part of attention_fwd.cu.
//
// What the kernel above does per query head it does here per K/V head and per piece of the context: the query rows that
// share a K/V head (tokens x group, at most 32) form one tile of 16 or 32 rows, and the context is cut into pieces so
// that every SM streams a part of K and V once.  Reading K and V is all that bounds it: with one CTA per query head
// and the whole context walked by each, 64 of 148 SMs were busy and K/V crossed L2 once per query head.
//
// A CTA takes one piece of one K/V head in steps of 64 positions.  Warp 4 streams K and V through a ring of 32 KB slots
// by TMA (page ids from the block table); warps 0-3 each own 16 positions of every step and run the online softmax on
// them by themselves: scores by mma.sync (16 query rows fill its tile; a tcgen05 tile would be 7/8 padding), P rounded
// to f16 in registers as the A operand of P V, f32 running maximum, sum and accumulator.  At the end the four are
// merged through shared memory, then the pieces of a cluster through distributed shared memory, each CTA taking a slice
// of the rows.  With several clusters per head a CTA leaves its slice in scratch and the last one to finish that slice
// (a counter that wraps to zero by itself) merges it.  No CTA waits for another outside its cluster.
// 1 token, 64 / 8 heads, 8192 positions f16 (33.5 MB): 15.8 us (5.1 at the measured copy rate), 88 with
// a CTA per query head; 2 tokens, 128 / 32 heads, 16002 positions (264 MB): 47.2 (40.9), 169 before.  Measured: clusters of
// 8 do not all fit at once (26 us), of 2 leave more to the last merge (22.6 against 18.1 at 32 rows), two CTAs per SM
// with half the ring each 22.0.
#pragma once
#include <cooperative_groups.h>

#define AD_ROWS 64                       // positions per step
#define AD_SLOTS 6
#define AD_SLOT_BYTES (2 * AD_ROWS * AT_D * 2)
#define AD_BLK (AD_ROWS * 128)           // one [64 positions x 64 dims] block, 128-byte swizzled
#define AD_CLUSTER 4
#define AD_MAX_ROWS 32
#define AD_THREADS 160
#define AD_SMEM (AD_SLOTS * AD_SLOT_BYTES + AD_MAX_ROWS * 256 + 1024 + 256)

static __device__ __forceinline__ void ad_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
static __device__ __forceinline__ void ad_ldm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
static __device__ __forceinline__ void ad_ldm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// Scratch: a counter per K/V head and slice, then per head, cluster and group of four dims the partial O, then its
// (max, sum).  The counters outlive a launch, so where they end depends on the heads that the scratch is laid out for
// and not on those of the launch: parts of a statement share one scratch with the whole of it.
static __host__ __device__ __forceinline__ size_t ad_counter_bytes(int heads) { return ((size_t)heads * 32 + 255) & ~(size_t)255; }
static int64_t ad_scratch_bytes(const ktb_attn_args& a, int group) {
    const int heads = a.heads / group;
    return (int64_t)ad_counter_bytes(a.scratch_heads ? a.scratch_heads : heads) + (int64_t)heads * a.splits * a.seq_q * group * 32 * 24;
}

template <int MT>                        // tiles of 16 query rows
__global__ void __launch_bounds__(AD_THREADS, 1)
ktb_attention_decode_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const ktb_attn_args a,
                            int group, int box_rows, int steps, int cluster, ktb_status* st) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sQ = ring + AD_SLOTS * AD_SLOT_BYTES;                   // [MT * 16 rows][256 bytes], chunks swizzled like K
    uint64_t* full = reinterpret_cast<uint64_t*>(sQ + AD_MAX_ROWS * 256);
    uint64_t* empty = full + AD_SLOTS;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + AD_SLOTS);
    int* is_last = const_cast<int*>(abort_flag) + 1;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int kv_head = blockIdx.x / a.splits, piece = blockIdx.x - kv_head * a.splits;
    const int u0 = (int)((int64_t)steps * piece / a.splits), u1 = (int)((int64_t)steps * (piece + 1) / a.splits);
    const int n = u1 - u0, rows = a.seq_q * group;
    if (threadIdx.x == 0) {
        for (int i = 0; i < AD_SLOTS; ++i) {
            tc_mbar_init(&full[i], 1);
            tc_mbar_init(&empty[i], 4);
        }
        *abort_flag = 0;
        tc_fence_barrier_init();
    }
    __syncthreads();

    if (warp == 4) {
        if (lane == 0) {
            tc_prefetch_tmap(&map_k);
            tc_prefetch_tmap(&map_v);
        }
        const int32_t* bt32 = reinterpret_cast<const int32_t*>(a.arena) + a.bt_off;
        const int64_t* bt64 = reinterpret_cast<const int64_t*>(a.arena) + a.bt_off;
        const int boxes = AD_ROWS / box_rows;                        // per step
        long long pages = 0;                                         // lane i: page of box i of the current 32
        for (int x = 0; x < n * boxes; ++x) {
            if ((x & 31) == 0 && x + lane < n * boxes) {             // the table is read 32 entries at a time, ahead of use
                int64_t j = ((int64_t)u0 * AD_ROWS + (int64_t)(x + lane) * box_rows) / a.page;
                if (j >= a.num_tiles) j = a.num_tiles - 1;           // past the table: any page, its scores are hidden below
                pages = a.bt_dtype == KTB_I64 ? bt64[j] : (long long)bt32[j];
                if (pages < 0) {
                    if (atomicExch(&st->negative_index, 1) == 0) st->bad_index_value = (int32_t)pages;
                    pages = 0;
                }
            }
            const int page = (int)__shfl_sync(0xffffffffu, pages, x & 31);
            const int s = x / boxes, r = (x - s * boxes) * box_rows, slot = s % AD_SLOTS;
            const int y = (int)(((int64_t)(u0 + s) * AD_ROWS + r) % a.page);
            bool ok = true;
            if (lane == 0) {
                if (r == 0) {
                    ok = tc_mbar_wait(&empty[slot], ((s / AD_SLOTS) & 1) ^ 1, abort_flag, st, 41);
                    if (ok) tc_mbar_expect_tx(&full[slot], AD_SLOT_BYTES);
                }
                uint8_t* k = ring + slot * AD_SLOT_BYTES;
                for (int d = 0; d < 2 && ok; ++d) {
                    at_tma_load_4d(k + d * AD_BLK + r * 128, &map_k, &full[slot], d * 64, kv_head, y, page);
                    at_tma_load_4d(k + (2 + d) * AD_BLK + r * 128, &map_v, &full[slot], d * 64, kv_head, y, page);
                }
            }
            if (!__shfl_sync(0xffffffffu, (int)ok, 0)) break;
        }
    } else {
        for (int e = threadIdx.x; e < MT * 16 * 16; e += 128) {   // 16-byte chunks; rows past the last are zeros
            const int row = e >> 4, c = e & 15, tok = row / group, head = kv_head * group + row - tok * group;
            uint4 q = make_uint4(0, 0, 0, 0);
            if (row < rows)
                q = *reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(a.arena) + a.q_off + (int64_t)tok * a.q_row_stride +
                                                    (int64_t)head * a.q_head_stride + c * 8);
            *reinterpret_cast<uint4*>(sQ + row * 256 + ((c ^ (row & 7)) << 4)) = q;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");               // (the four softmax warps)
    }

    // accumulators of this warp: rows lane / 4 and lane / 4 + 8 of each tile, columns 8 i + 2 (lane % 4) + {0, 1}
    const int q4 = lane >> 2, c2 = (lane & 3) * 2;
    float O[MT][16][4], m[MT][2], l[MT][2];
    if (warp < 4) {
        int64_t limit[MT][2];                                        // last visible position of the thread's rows
        const int64_t n_kv = (int64_t)a.num_tiles * a.page;
#pragma unroll
        for (int t = 0; t < MT; ++t) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) O[t][i][e] = 0.f;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int tok = (t * 16 + h * 8 + q4) / group;
                limit[t][h] = n_kv - 1;
                if (a.causal && (int64_t)tok + a.causal_delta < limit[t][h]) limit[t][h] = (int64_t)tok + a.causal_delta;
                // the initial maximum and sum count once per row: in warp 0 of the first piece
                const bool first = piece == 0 && warp == 0;
                m[t][h] = first ? a.m_init * 1.4426950408889634f : -INFINITY;
                l[t][h] = first && (lane & 3) == 0 ? a.l_init : 0.f;
            }
        }
        const float sl = a.scale * 1.4426950408889634f;
        const uint32_t ring0 = tc_smem_u32(ring), q0 = tc_smem_u32(sQ);
        const int k_row = warp * 16 + (lane & 7), v_row = k_row + ((lane >> 3) & 1) * 8;
        for (int s = 0; s < n; ++s) {
            const int slot = s % AD_SLOTS;
            if (!__all_sync(0xffffffffu, tc_mbar_wait(&full[slot], (s / AD_SLOTS) & 1, abort_flag, st, 42))) break;
            const uint32_t base = ring0 + slot * AD_SLOT_BYTES;
            float S[MT][2][4];
#pragma unroll
            for (int t = 0; t < MT; ++t)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[t][j][e] = 0.f;
#pragma unroll
            for (int kc = 0; kc < 4; ++kc) {                         // 32 dims: four 16-byte chunks of a row
                uint32_t b[2][4];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int r = k_row + j * 8, chunk = (kc & 1) * 4 + (lane >> 3);
                    ad_ldm4(base + (kc >> 1) * AD_BLK + r * 128 + ((chunk ^ (r & 7)) << 4), b[j]);
                }
#pragma unroll
                for (int t = 0; t < MT; ++t)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int r = t * 16 + (lane & 15), chunk = kc * 4 + h * 2 + (lane >> 4);
                        uint32_t q[4];
                        ad_ldm4(q0 + r * 256 + ((chunk ^ (r & 7)) << 4), q);
                        ad_mma(S[t][0], q, b[0][h * 2], b[0][h * 2 + 1]);
                        ad_mma(S[t][1], q, b[1][h * 2], b[1][h * 2 + 1]);
                    }
            }
            const int64_t p0 = (int64_t)(u0 + s) * AD_ROWS + warp * 16;      // first position of this warp
            uint32_t P[MT][4];
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                float alpha[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    // (scores in the log2 domain; hidden positions are -inf and become exact zeros)
                    float mx = -INFINITY;
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            float& x = S[t][j][h * 2 + e];
                            x = p0 + j * 8 + c2 + e <= limit[t][h] ? x * sl : -INFINITY;
                            mx = fmaxf(mx, x);
                        }
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                    const float mn = fmaxf(m[t][h], mx), mz = mn == -INFINITY ? 0.f : mn;
                    alpha[h] = at_ex2(m[t][h] - mz);                 // (0 while nothing has been seen)
                    m[t][h] = mn;
                    float sum = 0.f;
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            float& x = S[t][j][h * 2 + e];
                            x = at_ex2(x - mz);
                            sum += x;
                        }
                    l[t][h] = l[t][h] * alpha[h] + sum;
                }
                if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        O[t][i][0] *= alpha[0];
                        O[t][i][1] *= alpha[0];
                        O[t][i][2] *= alpha[1];
                        O[t][i][3] *= alpha[1];
                    }
                }
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const __half2 p = __floats2half2_rn(S[t][j][h * 2], S[t][j][h * 2 + 1]);
                        P[t][j * 2 + h] = *reinterpret_cast<const uint32_t*>(&p);
                    }
            }
#pragma unroll
            for (int i = 0; i < 16; i += 2) {                        // two column tiles of 8 dims
                const int chunk = (i & 7) + (lane >> 4);
                uint32_t b[4];
                ad_ldm4t(base + (2 + (i >> 3)) * AD_BLK + v_row * 128 + ((chunk ^ (v_row & 7)) << 4), b);
#pragma unroll
                for (int t = 0; t < MT; ++t) {
                    ad_mma(O[t][i], P[t], b[0], b[1]);
                    ad_mma(O[t][i + 1], P[t], b[2], b[3]);
                }
            }
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(&empty[slot]);
        }
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                l[t][h] += __shfl_xor_sync(0xffffffffu, l[t][h], 1);
                l[t][h] += __shfl_xor_sync(0xffffffffu, l[t][h], 2);
            }
    }
    __syncthreads();                     // every load has landed and been read: the ring is free
    float* sO = reinterpret_cast<float*>(ring);                      // [4 warps][MT * 16 rows][128 + 4]
    float* sM = sO + 4 * MT * 16 * (AT_D + 4);                       // [4][MT * 16] maxima, then sums
    float* sL = sM + 4 * MT * 16;
    if (warp < 4) {
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = (warp * MT + t) * 16 + h * 8 + q4;
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    *reinterpret_cast<float2*>(sO + row * (AT_D + 4) + i * 8 + c2) = make_float2(O[t][i][h * 2], O[t][i][h * 2 + 1]);
                if ((lane & 3) == 0) {
                    sM[row] = m[t][h];
                    sL[row] = l[t][h];
                }
            }
    }
    __syncthreads();
    // Merge the four warps; thread = (row, four dims).  A row's O scaled to its maximum, the maximum and the sum beside it.
    auto store = [&](int row, int d, float4 o, float sum) {
        const int tok = row / group, head = kv_head * group + row - tok * group;
        const float inv = 1.0f / sum;
        __half2 h[2] = {__floats2half2_rn(o.x * inv, o.y * inv), __floats2half2_rn(o.z * inv, o.w * inv)};
        *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(a.arena) + a.o_off + (int64_t)tok * a.o_row_stride +
                                  (int64_t)head * a.o_head_stride + d) = *reinterpret_cast<uint2*>(h);
    };
    const bool whole = *abort_flag == 0;
    float4* mO = reinterpret_cast<float4*>(sL + 4 * MT * 16);        // [rows][32]
    float2* mML = reinterpret_cast<float2*>(mO + MT * 16 * 32);      // [rows]
    for (int e = threadIdx.x; e < rows * 32; e += AD_THREADS) {
        const int row = e >> 5, d = (e & 31) * 4;
        float mx = -INFINITY;
#pragma unroll
        for (int w = 0; w < 4; ++w) mx = fmaxf(mx, sM[w * MT * 16 + row]);
        const float mz = mx == -INFINITY ? 0.f : mx;
        float sum = 0.f;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float f = at_ex2(sM[w * MT * 16 + row] - mz);
            const float4 x = *reinterpret_cast<const float4*>(sO + (w * MT * 16 + row) * (AT_D + 4) + d);
            sum += sL[w * MT * 16 + row] * f;
            o.x += x.x * f; o.y += x.y * f; o.z += x.z * f; o.w += x.w * f;
        }
        if (a.splits == 1) {
            if (whole) store(row, d, o, sum);
            continue;
        }
        mO[e] = o;
        if (d == 0) mML[row] = make_float2(mx, sum);
    }
    if (a.splits == 1) return;
    // the pieces of the cluster, a slice of the rows' elements per CTA
    const int rank = piece % cluster, clusters = a.splits / cluster, kv_heads = gridDim.x / a.splits;
    const int per = (rows * 32 + cluster - 1) / cluster;
    const int e0 = rank * per, e1 = e0 + per < rows * 32 ? e0 + per : rows * 32;
    float4* part_o = reinterpret_cast<float4*>(reinterpret_cast<uint8_t*>(a.dev_scratch) + ad_counter_bytes(a.scratch_heads ? a.scratch_heads : kv_heads));
    float2* part_ml = reinterpret_cast<float2*>(part_o + (size_t)a.splits / cluster * kv_heads * rows * 32);
    auto merge = [&](int n_parts, auto ml_of, auto o_of, float4& o, float& mx, float& sum) {
        mx = -INFINITY;
        for (int p = 0; p < n_parts; ++p) mx = fmaxf(mx, ml_of(p).x);
        const float mz = mx == -INFINITY ? 0.f : mx;
        sum = 0.f;
        o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int p = 0; p < n_parts; ++p) {
            const float2 ml = ml_of(p);
            const float f = at_ex2(ml.x - mz);
            const float4 x = o_of(p);
            sum += ml.y * f;
            o.x += x.x * f; o.y += x.y * f; o.z += x.z * f; o.w += x.w * f;
        }
    };
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();                                           // every CTA's merged rows are in its shared memory
    const size_t mine = ((size_t)kv_head * clusters + piece / cluster) * rows * 32;
    for (int e = e0 + threadIdx.x; e < e1; e += AD_THREADS) {
        float4 o;
        float mx, sum;
        merge(cluster, [&](int p) { return *cl.map_shared_rank(mML + (e >> 5), p); }, [&](int p) { return *cl.map_shared_rank(mO + e, p); }, o, mx, sum);
        if (clusters == 1) {
            if (whole) store(e >> 5, (e & 31) * 4, o, sum);
            continue;
        }
        part_o[mine + e] = o;
        part_ml[mine + e] = make_float2(mx, sum);
    }
    if (clusters > 1) {
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0)            // (wraps to zero with the last cluster: the next launch finds it so)
            *is_last = atomicInc(reinterpret_cast<unsigned*>(a.dev_scratch) + kv_head * cluster + rank, (unsigned)clusters - 1) ==
                       (unsigned)clusters - 1;
        __syncthreads();
        if (*is_last) {
            __threadfence();
            const size_t base = (size_t)kv_head * clusters * rows * 32;
            for (int e = e0 + threadIdx.x; e < e1; e += AD_THREADS) {
                float4 o;
                float mx, sum;
                merge(clusters, [&](int p) { return __ldcg(part_ml + base + (size_t)p * rows * 32 + e); },
                      [&](int p) { return __ldcg(part_o + base + (size_t)p * rows * 32 + e); }, o, mx, sum);
                if (whole) store(e >> 5, (e & 31) * 4, o, sum);
            }
        }
    }
    cl.sync();                                           // peers may still read this CTA's shared memory
}

static int launch_attn_decode(ktb_ctx* ctx, const ktb_attn_args& a, const CUtensorMap& mk, const CUtensorMap& mv, int group, int box_rows) {
    const int kv_heads = a.heads / group, rows = a.seq_q * group;
    int64_t seen = (int64_t)a.num_tiles * a.page;                    // positions that some row sees
    if (a.causal && (int64_t)a.seq_q + a.causal_delta < seen) seen = (int64_t)a.seq_q + a.causal_delta;
    const int64_t least = (seen + AD_ROWS - 1) / AD_ROWS, most = ((int64_t)a.num_tiles * a.page + AD_ROWS - 1) / AD_ROWS;
    if (a.steps != 0 && (a.steps < least || a.steps > most))
        return ktb_fail(ctx, KTB_E_ARG, "attention_fwd", "steps must cover the positions that the rows see, within the context");
    const int steps = a.steps ? a.steps : (int)least;
    // the largest cluster that the pieces fill
    int cluster = 1;
    while (cluster < AD_CLUSTER && a.splits % (cluster * 2) == 0) cluster *= 2;
    auto k = rows <= 16 ? ktb_attention_decode_kernel<1> : ktb_attention_decode_kernel<2>;
    KTB_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, AD_SMEM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kv_heads * a.splits);
    cfg.blockDim = dim3(AD_THREADS);
    cfg.dynamicSmemBytes = AD_SMEM;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = cluster;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    KTB_CUDA(ctx, cudaLaunchKernelEx(&cfg, k, mk, mv, a, group, box_rows, steps, cluster, ctx->dev_status));
    KTB_CHECK_LAUNCH(ctx, "ktb_attention_decode_kernel");
    return KTB_OK;
}
