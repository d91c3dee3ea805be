// Row reductions in the pairing order of the reference's linalg.reduce, shared by the row kernels.
//
// A row of cols = T * 8 * NV elements is held by a group of T threads (thread t owns the 16-byte vectors
// j * T + t, j < NV).  row_fold combines x[i] (op) x[i + h] for h = cols/2 ... 1 — the halving order of
// _tree_fold (ktir_cpu/dialects/linalg_ops.py:86-133) when cols is a power of two: first across a thread's
// own vectors, then across the warps of the group (one shared-memory exchange, combined in the same
// pairing), then by warp shuffle, then across the 8 elements of the remaining vector.
#pragma once
#include "common.cuh"

template <bool MAXNUM>
static __device__ __forceinline__ float sm_max(float a, float b) {
    if (!MAXNUM && (a != a || b != b)) return __int_as_float(0x7fc00000);
    return fmaxf(a, b);
}

template <int OP, bool MAXNUM, bool R16>
static __device__ __forceinline__ float sm_comb(float a, float b) {
    if (OP == 0) return sm_max<MAXNUM>(a, b);
    const float r = a + b;
    return R16 ? ktb_round16(r) : r;
}

// How a row of any length is dealt out: whole warps, `nv` chunks of 8 elements per thread.  The fewest warps that hold
// the row (and the partial chunks at its two ends) with `max_nv` chunks per thread, then as few chunks as those need;
// rows of one warp share a CTA of 256 threads eight at a time and need no block barrier, rows of two warps four at
// a time.  With less than 512 threads per SM from all rows together a row gets more threads, which shortens its chain.
struct rg_split {
    int threads, nv, groups;
};
static inline rg_split rg_choose(int cols, bool aligned, int64_t rows, int sm_count, int max_nv, int max_threads) {
    const int vecs = (cols + (aligned ? 7 : 14)) / 8;
    rg_split s;
    int nv = max_nv;
    auto threads = [&](int n) { return (vecs + 32 * n - 1) / (32 * n) * 32; };
    while (nv > 1 && rows * threads(nv) < (int64_t)sm_count * 512 && threads(nv / 2) <= max_threads) nv /= 2;
    s.threads = threads(nv);
    s.nv = (vecs + s.threads - 1) / s.threads;
    s.groups = s.threads == 32 ? 8 : 256 / s.threads > 4 ? 4 : 256 / s.threads < 1 ? 1 : 256 / s.threads;
    return s;
}

// Named barrier of one row group (ids 1..4 as literals so only those are reserved).
static __device__ __forceinline__ void group_barrier(int id, int threads) {
    switch (id) {
        case 1: asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); break;
        case 2: asm volatile("bar.sync 2, %0;" ::"r"(threads) : "memory"); break;
        case 3: asm volatile("bar.sync 3, %0;" ::"r"(threads) : "memory"); break;
        default: asm volatile("bar.sync 4, %0;" ::"r"(threads) : "memory"); break;
    }
}

// Pairing of the cross-warp levels: value(base, stride, n) = value(base, 2*stride, n/2)
// (op) value(base + stride, 2*stride, n/2), leaves are the per-warp partials.
template <int OP, bool MAXNUM, bool R16>
static __device__ __forceinline__ float warp_tree(const float* p, int n_warps, int lane_slot_stride) {
    // p[w * lane_slot_stride] is the partial of warp w for this (lane, slot)
    float o[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) o[w] = w < n_warps ? p[w * lane_slot_stride] : 0.f;
    if (n_warps == 8) {
        const float a = sm_comb<OP, MAXNUM, R16>(sm_comb<OP, MAXNUM, R16>(o[0], o[4]), sm_comb<OP, MAXNUM, R16>(o[2], o[6]));
        const float b = sm_comb<OP, MAXNUM, R16>(sm_comb<OP, MAXNUM, R16>(o[1], o[5]), sm_comb<OP, MAXNUM, R16>(o[3], o[7]));
        return sm_comb<OP, MAXNUM, R16>(a, b);
    }
    if (n_warps == 4)
        return sm_comb<OP, MAXNUM, R16>(sm_comb<OP, MAXNUM, R16>(o[0], o[2]), sm_comb<OP, MAXNUM, R16>(o[1], o[3]));
    return sm_comb<OP, MAXNUM, R16>(o[0], o[1]);
}

// Fold of the T*8*NV values of a row; every thread of the group gets the result.
template <int NV, int OP, bool MAXNUM, bool R16>
static __device__ __forceinline__ float row_fold(const float (&x)[NV][8], int T, int t, int group,
                                                 float* xchg /* [256][8] */, float* bcast /* [256/32] */) {
    float v[8];
    if (NV == 1) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = x[0][k];
    } else {
        constexpr int H = NV / 2 > 0 ? NV / 2 : 1;
        float w[H][8];
#pragma unroll
        for (int j = 0; j < H; ++j)
#pragma unroll
            for (int k = 0; k < 8; ++k) w[j][k] = sm_comb<OP, MAXNUM, R16>(x[j][k], x[j + H][k]);
#pragma unroll
        for (int m = H / 2; m >= 1; m >>= 1)
#pragma unroll
            for (int j = 0; j < m; ++j)
#pragma unroll
                for (int k = 0; k < 8; ++k) w[j][k] = sm_comb<OP, MAXNUM, R16>(w[j][k], w[j + m][k]);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = w[0][k];
    }
    if (T > 32) {
        const int n_warps = T >> 5;
        float* mine = xchg + (size_t)threadIdx.x * 8;
#pragma unroll
        for (int k = 0; k < 8; ++k) mine[k] = v[k];
        group_barrier(1 + group, T);
        if (t < 32) {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = warp_tree<OP, MAXNUM, R16>(mine + k, n_warps, 32 * 8);
        }
    }
    const int w = T < 32 ? T : 32;
    for (int d = w >> 1; d >= 1; d >>= 1) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float o = __shfl_down_sync(0xffffffffu, v[k], d, w);
            v[k] = sm_comb<OP, MAXNUM, R16>(v[k], o);
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = sm_comb<OP, MAXNUM, R16>(v[k], v[k + 4]);
    v[0] = sm_comb<OP, MAXNUM, R16>(v[0], v[2]);
    v[1] = sm_comb<OP, MAXNUM, R16>(v[1], v[3]);
    v[0] = sm_comb<OP, MAXNUM, R16>(v[0], v[1]);
    if (T > 32) {
        if (t == 0) bcast[group] = v[0];
        group_barrier(1 + group, T);
        return bcast[group];
    }
    return __shfl_sync(0xffffffffu, v[0], 0, w);
}


// ---- rows of any length ---------------------------------------------------------------------------------
static __device__ __forceinline__ void rg_barrier(int group, int T) {
    if (T == 32) __syncwarp();
    else group_barrier(1 + group, T);
}

// A row that starts `mis` elements (0..7) after a boundary of 8 is walked in the memory's own 8-element chunks: chunk
// c holds elements 8 c - mis ... 8 c - mis + 7, of which the first and the last chunk may have fewer.  Whole chunks
// move as 16-byte vectors whatever the row's start; only the elements of the edge chunks go one by one.
static __device__ __forceinline__ bool rg_whole(int c, int mis, int cols) { return c * 8 >= mis && c * 8 - mis + 8 <= cols; }
static __device__ __forceinline__ bool rg_any(int c, int mis, int cols) { return c * 8 - mis < cols; }

// Chunk c of an f16 row as packed halves; what lies outside the row keeps what `raw` held.
static __device__ __forceinline__ void rg_load_h(const __half* row, int mis, int cols, int c, uint4& raw) {
    const __half* p = row + (c * 8 - mis);
    if (rg_whole(c, mis, cols)) {
        raw = __ldcs(reinterpret_cast<const uint4*>(p));
    } else if (rg_any(c, mis, cols)) {
        __half* e = reinterpret_cast<__half*>(&raw);
#pragma unroll
        for (int v = 0; v < 8; ++v)
            if (c * 8 + v >= mis && c * 8 + v - mis < cols) e[v] = p[v];
    }
}
// ... of a row whose own start lies elsewhere between boundaries than `mis` (chunks laid out for another row).
static __device__ __forceinline__ void rg_load_h_apart(const __half* row, int mis, int cols, int c, uint4& raw) {
    const __half* p = row + (c * 8 - mis);
    __half* e = reinterpret_cast<__half*>(&raw);
#pragma unroll
    for (int v = 0; v < 8; ++v)
        if (c * 8 + v >= mis && c * 8 + v - mis < cols) e[v] = p[v];
}
// `same`: the destination row starts at the same offset from a boundary as the row whose chunks these are.
static __device__ __forceinline__ void rg_store_h(__half* row, int mis, int cols, int c, bool same, const uint4& raw) {
    __half* p = row + (c * 8 - mis);
    if (same && rg_whole(c, mis, cols)) {
        __stcs(reinterpret_cast<uint4*>(p), raw);
    } else if (rg_any(c, mis, cols)) {
        const __half* e = reinterpret_cast<const __half*>(&raw);
#pragma unroll
        for (int v = 0; v < 8; ++v)
            if (c * 8 + v >= mis && c * 8 + v - mis < cols) p[v] = e[v];
    }
}
// The same as f32 values for an f16 or f32 tile whose row starts at element `off`; `same` as above (a weight row,
// say, may start elsewhere).
static __device__ __forceinline__ void rg_load8(const void* arena, int64_t off, int dtype, int mis, int cols, int c, bool same,
                                                float (&x)[8]) {
    const int64_t at = off + (c * 8 - mis);
    if (same && rg_whole(c, mis, cols)) {
        if (dtype == KTB_F16) {
            const uint4 raw = *reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(arena) + at);
            const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = __half22float2(h[i]);
                x[2 * i] = f.x;
                x[2 * i + 1] = f.y;
            }
        } else {
            const float4 lo = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(arena) + at);
            const float4 hi = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(arena) + at + 4);
            x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w;
            x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
        }
    } else if (rg_any(c, mis, cols)) {
#pragma unroll
        for (int v = 0; v < 8; ++v)
            if (c * 8 + v >= mis && c * 8 + v - mis < cols)
                x[v] = dtype == KTB_F16 ? __half2float(reinterpret_cast<const __half*>(arena)[at + v])
                                        : reinterpret_cast<const float*>(arena)[at + v];
    }
}
static __device__ __forceinline__ void rg_store8(void* arena, int64_t off, int dtype, int mis, int cols, int c, bool same,
                                                 const float (&x)[8]) {
    if (dtype == KTB_F16) {
        uint4 raw;
        __half2* h = reinterpret_cast<__half2*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(x[2 * i], x[2 * i + 1]);
        rg_store_h(reinterpret_cast<__half*>(arena) + off, mis, cols, c, same, raw);
        return;
    }
    float* p = reinterpret_cast<float*>(arena) + off + (c * 8 - mis);
    if (same && rg_whole(c, mis, cols)) {
        __stcs(reinterpret_cast<float4*>(p), make_float4(x[0], x[1], x[2], x[3]));
        __stcs(reinterpret_cast<float4*>(p + 4), make_float4(x[4], x[5], x[6], x[7]));
    } else if (rg_any(c, mis, cols)) {
#pragma unroll
        for (int v = 0; v < 8; ++v)
            if (c * 8 + v >= mis && c * 8 + v - mis < cols) p[v] = x[v];
    }
}
// Chunk c of the values to be folded, to shared memory; the row then begins at buf + mis.
static __device__ __forceinline__ void rg_park8(float* buf, int mis, int cols, int c, const float (&x)[8]) {
    if (!rg_any(c, mis, cols)) return;
    reinterpret_cast<float4*>(buf + c * 8)[0] = make_float4(x[0], x[1], x[2], x[3]);
    reinterpret_cast<float4*>(buf + c * 8)[1] = make_float4(x[4], x[5], x[6], x[7]);
}

// Three levels of the reference's fold at once: of n values, level one leaves n - n / 2 — value i is x(i) (op)
// x(i + n / 2), and an odd last one is carried along (ktir_cpu/dialects/linalg_ops.py:86-133).  For all but the last
// few i (none of them carried) this is eight values in a fixed pairing.
template <typename F, typename C>
static __device__ __forceinline__ auto rg_level3(F x, C op, int n, int i) {
    const int h0 = n >> 1, n1 = n - h0, h1 = n1 >> 1, n2 = n1 - h1, h2 = n2 >> 1;
    if (i < h2 && i + h2 < h1 && i + h2 + h1 < h0) {
        const auto p = op(op(x(i), x(i + h0)), op(x(i + h1), x(i + h1 + h0)));
        const auto q = op(op(x(i + h2), x(i + h2 + h0)), op(x(i + h2 + h1), x(i + h2 + h1 + h0)));
        return op(p, q);
    }
    // the general form, as a loop over the eight places: those that do not exist are left out of their pair
    auto s2 = x(0);                                      // (both are set before they are read)
    auto s1 = s2;
#pragma unroll 1
    for (int e2 = 0; e2 < (i < h2 ? 2 : 1); ++e2) {
        const int j = i < h2 ? i + e2 * h2 : i + h2;
#pragma unroll 1
        for (int e1 = 0; e1 < (j < h1 ? 2 : 1); ++e1) {
            const int k = j < h1 ? j + e1 * h1 : j + h1;
            const auto v = k < h0 ? op(x(k), x(k + h0)) : x(k + h0);
            s1 = e1 ? op(s1, v) : v;
        }
        s2 = e2 ? op(s2, s1) : s1;
    }
    return s2;
}
static __host__ __device__ __forceinline__ int rg_after3(int n) {
    n -= n >> 1;
    n -= n >> 1;
    return n - (n >> 1);
}

// Elements (of the row's dtype, or floats) that the chunks of a row take in shared memory, and the floats that its fold
// takes beside them: an eighth of the values, an eighth of those, the result.
static __host__ __device__ __forceinline__ int rg_chunk_elems(int cols) { return (cols + 14) & ~7; }
static __host__ __device__ __forceinline__ int rg_fold_floats(int cols) {
    const int n1 = rg_after3(cols);
    return ((n1 + 3) & ~3) + ((rg_after3(n1) + 3) & ~3) + 4;
}

// Fold of value(0) .. value(cols - 1), which the T threads of the group have put where `value` finds them, in the
// reference's order for any length, with `op` on values of type V; every thread gets the result, and what `value`
// reads is left alone.  Three levels per barrier (every value is read once, an eighth of that again); the last 32 by
// shuffles in the first warp.  `first_wide(dst)` may do the first three levels itself (whole vectors) and return true.
template <typename V, typename F, typename C, typename W>
static __device__ __forceinline__ V rg_fold_with(F value, C op, W first_wide, float* tmp, int cols, int T, int t, int group) {
    V* dst = reinterpret_cast<V*>(tmp);
    V* other = reinterpret_cast<V*>(tmp + ((rg_after3(cols) + 3) & ~3));
    V* result = reinterpret_cast<V*>(tmp + rg_fold_floats(cols) - 4);
    rg_barrier(group, T);
    int n = cols;
    V v = V();
    if (n > 256) {
        const int m = rg_after3(n);
        if (!first_wide(dst))
            for (int i = t; i < m; i += T) dst[i] = rg_level3(value, op, n, i);
        n = m;
        rg_barrier(group, T);
        while (n > 256) {
            const int k = rg_after3(n);
            const V* src = dst;
            for (int i = t; i < k; i += T) other[i] = rg_level3([&](int q) { return src[q]; }, op, n, i);
            rg_barrier(group, T);
            V* o = dst;
            dst = other;
            other = o;
            n = k;
        }
        if (t < 32 && t < rg_after3(n)) v = rg_level3([&](int q) { return dst[q]; }, op, n, t);
    } else if (t < 32 && t < rg_after3(n)) {
        v = rg_level3(value, op, n, t);
    }
    if (t < 32) {
        for (n = rg_after3(n); n > 1;) {
            const int h = n >> 1;
            const V o = __shfl_down_sync(0xffffffffu, v, h);
            v = t < h ? op(v, o) : o;
            n -= h;
        }
        if (t == 0) *result = v;
    }
    rg_barrier(group, T);
    return *result;
}
template <int OP, bool MAXNUM, bool R16, typename F>
static __device__ __forceinline__ float rg_fold(F value, float* tmp, int cols, int T, int t, int group) {
    return rg_fold_with<float>(value, [](float a, float b) { return sm_comb<OP, MAXNUM, R16>(a, b); },
                               [](float*) { return false; }, tmp, cols, T, t, group);
}

// Two f32 values in one 64-bit register: fma / add / mul on such a pair are ONE instruction here, each half rounded like
// the scalar op.
static __device__ __forceinline__ uint64_t sm_pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
static __device__ __forceinline__ void sm_unpack2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
static __device__ __forceinline__ uint64_t sm_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
static __device__ __forceinline__ uint64_t sm_add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
static __device__ __forceinline__ uint64_t sm_mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The same fold of a sum whose every add rounds to f16, on packed halves: an f16 add of two f16 values is
// the f32 add rounded to f16 (24 >= 2 * 11 + 2 significand bits: the double rounding cannot show), so the
// results are those of row_fold<NV, 1, false, true> at an eighth of the conversions.  x[j][q] holds elements
// 2q, 2q + 1 of vector j.
static __device__ __forceinline__ __half2 warp_tree_h(const __half2* p, int n_warps, int stride) {
    __half2 o[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) o[w] = w < n_warps ? p[w * stride] : __half2();
    if (n_warps == 8)
        return __hadd2_rn(__hadd2_rn(__hadd2_rn(o[0], o[4]), __hadd2_rn(o[2], o[6])),
                          __hadd2_rn(__hadd2_rn(o[1], o[5]), __hadd2_rn(o[3], o[7])));
    if (n_warps == 4) return __hadd2_rn(__hadd2_rn(o[0], o[2]), __hadd2_rn(o[1], o[3]));
    return __hadd2_rn(o[0], o[1]);
}

template <int NV>
static __device__ __forceinline__ float row_fold_h(const __half2 (&x)[NV][4], int T, int t, int group,
                                                   float* xchg /* [256][8] */, float* bcast /* [256/32] */) {
    __half2 v[4];
    if (NV == 1) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = x[0][k];
    } else {
        constexpr int H = NV / 2 > 0 ? NV / 2 : 1;
        __half2 w[H][4];
#pragma unroll
        for (int j = 0; j < H; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) w[j][k] = __hadd2_rn(x[j][k], x[j + H][k]);
#pragma unroll
        for (int m = H / 2; m >= 1; m >>= 1)
#pragma unroll
            for (int j = 0; j < m; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k) w[j][k] = __hadd2_rn(w[j][k], w[j + m][k]);
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = w[0][k];
    }
    if (T > 32) {
        const int n_warps = T >> 5;
        __half2* mine = reinterpret_cast<__half2*>(xchg) + (size_t)threadIdx.x * 4;
#pragma unroll
        for (int k = 0; k < 4; ++k) mine[k] = v[k];
        group_barrier(1 + group, T);
        if (t < 32) {
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = warp_tree_h(mine + k, n_warps, 32 * 4);
        }
    }
    const int w = T < 32 ? T : 32;
    for (int d = w >> 1; d >= 1; d >>= 1) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = __hadd2_rn(v[k], __shfl_down_sync(0xffffffffu, v[k], d, w));
    }
    v[0] = __hadd2_rn(v[0], v[2]);                       // elements k and k + 4
    v[1] = __hadd2_rn(v[1], v[3]);
    v[0] = __hadd2_rn(v[0], v[1]);                       // 0 + 2, 1 + 3
    const float r = __half2float(__hadd_rn(__low2half(v[0]), __high2half(v[0])));
    if (T > 32) {
        if (t == 0) bcast[group] = r;
        group_barrier(1 + group, T);
        return bcast[group];
    }
    return __shfl_sync(0xffffffffu, r, 0, w);
}
