// Row programs over rows of any length and alignment (part of row_program.cu).  How such a row is cut into chunks of 8
// elements and folded: row_fold.cuh.  The rows' order of summation and every rounding are those of the kernels for
// 2^n columns.

// A row-value program that passes ONE value from op to op — sum, * 1/n, + eps, 1/sqrt — which is what the means and
// scales of normalisations are.  Every thread evaluates it on registers; the general evaluator's operands go through
// memory, one thread runs it and the others wait.
#define RP_CHAIN_OPS 6
struct rp_chain {
    int n, red;                    // ops, and the reduction result they start from; n < 0: no chain
    int32_t code[RP_CHAIN_OPS];    // opcode with its KTB_VM_ROUND16 / IMM flags
    float imm[RP_CHAIN_OPS];
};

static rp_chain rp_make_chain(const ktb_vm_program& p, int n_red) {
    rp_chain c = {};
    c.n = -1;
    if (p.n_ops > RP_CHAIN_OPS) return c;
    int cur = -1, red = p.n_ops == 0 ? p.result_reg : -1;
    for (int i = 0; i < p.n_ops; ++i) {
        const ktb_vm_op& o = p.ops[i];
        int from;
        switch (o.opcode & 0xff) {
            case KTB_VM_ADD: case KTB_VM_SUB: case KTB_VM_MUL: case KTB_VM_DIV:
                if (!(o.opcode & (KTB_VM_IMM_A | KTB_VM_IMM_B))) return c;
                from = (o.opcode & KTB_VM_IMM_A) ? o.b : o.a;
                break;
            case KTB_VM_MOV: case KTB_VM_NEG: case KTB_VM_ABS: case KTB_VM_SQRT: case KTB_VM_RSQRT:
                if (o.opcode & (KTB_VM_IMM_A | KTB_VM_IMM_B)) return c;
                from = o.a;
                break;
            default: return c;
        }
        if (i == 0) red = from;
        else if (from != cur) return c;
        cur = o.dst;
        c.code[i] = o.opcode;
        c.imm[i] = o.imm;
    }
    if (red < 0 || red >= n_red || (p.n_ops && p.result_reg != cur)) return c;
    c.n = p.n_ops;
    c.red = red;
    return c;
}

static __device__ __forceinline__ float rp_run_chain(const rp_chain& c, float v) {
    for (int i = 0; i < c.n; ++i) {
        const int code = c.code[i];
        const float imm = c.imm[i];
        const float a = (code & KTB_VM_IMM_A) ? imm : v, b = (code & KTB_VM_IMM_A) ? v : imm;
        switch (code & 0xff) {
            case KTB_VM_ADD: v = a + b; break;
            case KTB_VM_SUB: v = a - b; break;
            case KTB_VM_MUL: v = a * b; break;
            case KTB_VM_DIV: v = a / b; break;
            case KTB_VM_NEG: v = -a; break;
            case KTB_VM_ABS: v = fabsf(a); break;
            case KTB_VM_SQRT: v = sqrtf(a); break;
            case KTB_VM_RSQRT: v = 1.0f / sqrtf(a); break;
            default: break;                              // MOV
        }
        if (code & KTB_VM_ROUND16) v = ktb_round16(v);
    }
    return v;
}

// Shared words of a row group for the general evaluator: its registers, its result, the reduction results and the row
// scalars it is given (in memory from the start: as local arrays they were a stack frame of every thread).
#define RG_VM_RESULT KTB_VM_REGS
#define RG_VM_RED (KTB_VM_REGS + 4)
#define RG_VM_SCAL (KTB_VM_REGS + 8)
#define RG_VM_BAR (KTB_VM_REGS + 12)                     // the mbarrier of the row's bulk copy (8 bytes)
#define RG_VM_FLOATS (KTB_VM_REGS + 16)
static_assert(KTB_RP_MAX_RED <= 4 && KTB_RP_MAX_SCAL <= 4, "row group words");

// Row value `prog` for the whole group: as a chain by every thread, else by the first one through shared memory.
static __device__ __forceinline__ float rg_row_value(const ktb_vm_program& prog, const rp_chain& c, float red0, float red1, float* vmr,
                                                     int T, int t, int group) {
    if (c.n >= 0) return rp_run_chain(c, c.red ? red1 : red0);
    if (t == 0) {
        vmr[RG_VM_RED] = red0;
        vmr[RG_VM_RED + 1] = red1;
        vmr[RG_VM_RESULT] = rp_vm1(prog, vmr + RG_VM_RED, vmr, 1);
    }
    rg_barrier(group, T);
    const float v = vmr[RG_VM_RESULT];
    rg_barrier(group, T);                                // (before the slot is written again)
    return v;
}

// One thread per 64 elements of a row, in whole warps; more where the rows are few.
static rg_split rg_choose_norm(int64_t elems, int64_t rows, int sm_count, int most) {
    rg_split s = {};
    int T = (int)((elems + 2047) / 2048) * 32;
    while (T < most && rows * T < (int64_t)sm_count * 512 && T * 8 < elems) T *= 2;
    s.threads = T > most ? most : T;
    s.groups = s.threads == 32 ? 8 : s.threads <= 64 ? 4 : 1;
    return s;
}

// Arithmetic of a normalisation on eight values at once and on one: f32 (pairs in 64-bit registers), f32 with every op
// rounded to f16, and packed halves for f16 tiles whose every op rounds — an f16 add, subtract or multiply of f16
// values IS the f32 op rounded (24 >= 2 * 11 + 2 significand bits: the double rounding cannot show).
template <bool R16>
struct rg_f32 {
    using V = float;
    struct W { uint64_t p[4]; };
    static __device__ __forceinline__ float rnd(float x) { return R16 ? ktb_round16(x) : x; }
    static __device__ __forceinline__ V of(float x) { return x; }
    static __device__ __forceinline__ float back(V x) { return x; }
    static __device__ __forceinline__ V add(V a, V b) { return rnd(a + b); }
    static __device__ __forceinline__ V sub(V a, V b) { return rnd(a - b); }
    static __device__ __forceinline__ V mul(V a, V b) { return rnd(a * b); }
    static __device__ __forceinline__ uint64_t rnd2(uint64_t x) {
        if (!R16) return x;
        float a, b;
        sm_unpack2(x, a, b);
        return sm_pack2(ktb_round16(a), ktb_round16(b));
    }
    static __device__ __forceinline__ W splat(float x) { const uint64_t q = sm_pack2(x, x); return W{{q, q, q, q}}; }
    static __device__ __forceinline__ W add(W a, W b) {
#pragma unroll
        for (int i = 0; i < 4; ++i) a.p[i] = rnd2(sm_add2(a.p[i], b.p[i]));
        return a;
    }
    static __device__ __forceinline__ W sub(W a, W b) {          // a - b = a + (-b), exactly
#pragma unroll
        for (int i = 0; i < 4; ++i) a.p[i] = rnd2(sm_add2(a.p[i], b.p[i] ^ 0x8000000080000000ull));
        return a;
    }
    // (one by one: a packed multiply that feeds a packed add came out as one packed fma, rounded once — measured, a
    // last place of the sum in one row of thirty — and the reference rounds twice)
    static __device__ __forceinline__ W mul(W a, W b) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float a0, a1, b0, b1;
            sm_unpack2(a.p[i], a0, a1);
            sm_unpack2(b.p[i], b0, b1);
            a.p[i] = rnd2(sm_pack2(__fmul_rn(a0, b0), __fmul_rn(a1, b1)));
        }
        return a;
    }
    static __device__ __forceinline__ W load(const __half* x) { return halves(*reinterpret_cast<const uint4*>(x)); }
    static __device__ __forceinline__ W halves(const uint4& raw) {
        const __half2* h = reinterpret_cast<const __half2*>(&raw);
        W w;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h[i]);
            w.p[i] = sm_pack2(f.x, f.y);
        }
        return w;
    }
    static __device__ __forceinline__ W load(const float* x) { return from(reinterpret_cast<const float4*>(x)[0], reinterpret_cast<const float4*>(x)[1]); }
    static __device__ __forceinline__ W from(float4 a, float4 b) {
        return W{{sm_pack2(a.x, a.y), sm_pack2(a.z, a.w), sm_pack2(b.x, b.y), sm_pack2(b.z, b.w)}};
    }
    static __device__ __forceinline__ W from(const float (&f)[8]) {
        return W{{sm_pack2(f[0], f[1]), sm_pack2(f[2], f[3]), sm_pack2(f[4], f[5]), sm_pack2(f[6], f[7])}};
    }
    static __device__ __forceinline__ uint4 to_halves(const W& w) {
        uint4 raw;
        __half2* h = reinterpret_cast<__half2*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float a, b;
            sm_unpack2(w.p[i], a, b);
            h[i] = __floats2half2_rn(a, b);
        }
        return raw;
    }
    static __device__ __forceinline__ void put(V* dst, const W& w) {
        *reinterpret_cast<ulonglong2*>(dst) = make_ulonglong2(w.p[0], w.p[1]);
        *reinterpret_cast<ulonglong2*>(dst + 4) = make_ulonglong2(w.p[2], w.p[3]);
    }
    static __device__ __forceinline__ void floats(const W& w, float (&f)[8]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) sm_unpack2(w.p[i], f[2 * i], f[2 * i + 1]);
    }
};
struct rg_f16 {
    using V = __half;
    struct __align__(16) W { __half2 p[4]; };
    static __device__ __forceinline__ V of(float x) { return __float2half_rn(x); }
    static __device__ __forceinline__ float back(V x) { return __half2float(x); }
    static __device__ __forceinline__ V add(V a, V b) { return __hadd_rn(a, b); }
    static __device__ __forceinline__ V sub(V a, V b) { return __hsub_rn(a, b); }
    static __device__ __forceinline__ V mul(V a, V b) { return __hmul_rn(a, b); }
    static __device__ __forceinline__ W splat(float x) { const __half2 q = __float2half2_rn(x); return W{{q, q, q, q}}; }
    static __device__ __forceinline__ W add(W a, W b) {
#pragma unroll
        for (int i = 0; i < 4; ++i) a.p[i] = __hadd2_rn(a.p[i], b.p[i]);
        return a;
    }
    static __device__ __forceinline__ W sub(W a, W b) {
#pragma unroll
        for (int i = 0; i < 4; ++i) a.p[i] = __hsub2_rn(a.p[i], b.p[i]);
        return a;
    }
    static __device__ __forceinline__ W mul(W a, W b) {
#pragma unroll
        for (int i = 0; i < 4; ++i) a.p[i] = __hmul2_rn(a.p[i], b.p[i]);
        return a;
    }
    static __device__ __forceinline__ W load(const __half* x) { return halves(*reinterpret_cast<const uint4*>(x)); }
    static __device__ __forceinline__ uint4 to_halves(const W& w) { return *reinterpret_cast<const uint4*>(&w); }
    static __device__ __forceinline__ W halves(const uint4& raw) {
        W w;
        w.p[0] = *reinterpret_cast<const __half2*>(&raw.x);
        w.p[1] = *reinterpret_cast<const __half2*>(&raw.y);
        w.p[2] = *reinterpret_cast<const __half2*>(&raw.z);
        w.p[3] = *reinterpret_cast<const __half2*>(&raw.w);
        return w;
    }
    static __device__ __forceinline__ W from(const float (&f)[8]) {
        return W{{__floats2half2_rn(f[0], f[1]), __floats2half2_rn(f[2], f[3]), __floats2half2_rn(f[4], f[5]), __floats2half2_rn(f[6], f[7])}};
    }
    static __device__ __forceinline__ void put(V* dst, const W& w) { *reinterpret_cast<W*>(dst) = w; }
    static __device__ __forceinline__ void floats(const W& w, float (&f)[8]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 q = __half22float2(w.p[i]);
            f[2 * i] = q.x;
            f[2 * i + 1] = q.y;
        }
    }
};

// The normalisation skeletons (rp_norm) of rows of any length, column blocks included.  The row is parked in shared
// memory in its own dtype (all blocks, one read of HBM); the sums read their terms from there — term and block
// accumulation are evaluated as the first fold level reads them, on whole vectors where the length is a multiple of
// 64 and the row starts on a boundary — and so does the output.  No row in registers, no block barrier beyond those
// of the fold: eight rows or more per SM are in flight, which is what covers the chain of each.
// FAST, the common case: f16 tiles, every row on a boundary, the blocks end to end — row and blocks are one run of whole
// chunks and nothing is looked at chunk by chunk.
// Bound by the latency of a row's chain next to HBM: rms norm f16[2048, 5120] 16.5 us (849 in 61 steps; 6.5 at the
// measured copy rate), layer norm f16[2048, 8192] 28.9, blocked f16[4096, 8 x 1024] 59.2 (41.6).  Without FAST: rms
// norm f16[2048, 5001] 26.7.  Tried: five and six CTAs per SM (spills: 75 and 80 us blocked), weights and biases
// copied to shared memory with the row (71: four rows per SM instead of eight), prefetched to L2 (no change).
// Copy of whole 16-byte words, both ends on a 16-byte boundary, counted by `bar`.
static __device__ __forceinline__ void rg_bulk_load(void* smem_dst, const void* src, int bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(tc_smem_u32(smem_dst)), "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(tc_smem_u32(bar))
                 : "memory");
}
// Bounded wait (about a second of SM clocks) for the copies behind `bar`.  If they never land the status word says so and
// the thread goes on: the group's barriers still meet, and the host discards the result.
static __device__ __forceinline__ void rg_wait(uint64_t* bar, ktb_status* st, int site) {
    if (tc_mbar_try_wait(bar, 0)) return;
    const long long start = clock64();
    while (clock64() - start < 2000000000ll)
        if (tc_mbar_try_wait(bar, 0)) return;
    if (atomicExch(&st->wait_timeout, 1) == 0) st->wait_site = site;
}
// Shared memory of one row: evaluator words, fold, accumulated blocks, the row.
static __host__ __device__ __forceinline__ int rg_norm_bytes(int cols, int nb, int x_bytes, int v_bytes, bool blocked) {
    return 4 * (RG_VM_FLOATS + rg_fold_floats(cols)) + rg_chunk_elems(cols) * (nb * x_bytes + (blocked ? v_bytes : 0));
}
template <typename XT, typename A, int MODE, bool BLOCKED, bool FAST>
__global__ void __launch_bounds__(FAST ? 256 : 512, FAST ? 4 : 2)
ktb_row_norm_any_kernel(const __grid_constant__ ktb_rowprog_args a, const __grid_constant__ rp_norm m,
                        const __grid_constant__ rp_chain c_mean, const __grid_constant__ rp_chain c_scale, int T, int64_t total_rows,
                        ktb_status* st) {
    using V = typename A::V;
    using W = typename A::W;
    extern __shared__ __align__(16) float rg_smem[];
    const int group = threadIdx.x / T;
    const int t = threadIdx.x - group * T;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x / T) + group;
    if (row >= total_rows) return;                       // whole row groups: the barriers are per group
    const int cols = a.cols, nb = BLOCKED ? a.n_blocks : 1, pitch = rg_chunk_elems(cols);
    constexpr int XF = sizeof(XT);                       // bytes per parked element
    float* vmr = rg_smem + (size_t)group * (rg_norm_bytes(cols, nb, XF, sizeof(V), BLOCKED) / 4);
    float* tmp = vmr + RG_VM_FLOATS;
    V* acc = reinterpret_cast<V*>(tmp + rg_fold_floats(cols));                           // BLOCKED: the accumulated blocks
    XT* xs = reinterpret_cast<XT*>(acc + (BLOCKED ? pitch : 0));
    const int64_t item = (uint32_t)row / (uint32_t)a.rows_per_item;
    const int64_t r = row - item * a.rows_per_item;
    const int64_t* offs = a.dev_item_offsets + item * (a.n_in + 1 + a.n_side);
    const int64_t x_off = offs[m.x] + r * a.row_stride[m.x];
    const int mis = FAST ? 0 : (int)(x_off & 7), chunks = (cols + mis + 7) >> 3;
    const int64_t y_off = offs[a.n_in] + r * a.row_stride[a.n_in];
    const int64_t w_off = m.has_w ? offs[m.w] + r * a.row_stride[m.w] : 0;
    const int64_t b_off = m.has_b ? offs[m.b] + r * a.row_stride[m.b] : 0;
    const int n8 = nb * cols >> 3;                       // chunks of that run
    const int step = FAST ? cols : pitch;                // elements from block to block in `xs`

    if constexpr (FAST) {
        // one thread asks for the row as one copy into shared memory: nothing passes through registers
        uint64_t* bar = reinterpret_cast<uint64_t*>(vmr + RG_VM_BAR);
        if (t == 0) {
            tc_mbar_init(bar, 1);
            tc_fence_barrier_init();
            tc_fence_proxy_async();
            tc_mbar_expect_tx(bar, n8 * 16);
            rg_bulk_load(xs, reinterpret_cast<const __half*>(a.arena) + x_off, n8 * 16, bar);
        }
        rg_barrier(group, T);
        rg_wait(bar, st, 21);
    }
    else
    for (int jb = 0; jb < nb; ++jb) {
        const int64_t at = x_off + jb * a.blk_stride[m.x];
        const bool same = (at & 7) == mis;
        XT* dst = xs + jb * pitch;
        for (int c0 = t; c0 < chunks; c0 += 4 * T) {
            if constexpr (XF == 2) {
                const __half* p = reinterpret_cast<const __half*>(a.arena) + at;
                uint4 raw[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    raw[u] = make_uint4(0, 0, 0, 0);
                    if (same) rg_load_h(p, mis, cols, c0 + u * T, raw[u]);
                    else rg_load_h_apart(p, mis, cols, c0 + u * T, raw[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (c0 + u * T < chunks) *reinterpret_cast<uint4*>(dst + (c0 + u * T) * 8) = raw[u];
            } else {
                float v[4][8];
#pragma unroll
                for (int u = 0; u < 4; ++u) rg_load8(a.arena, at, KTB_F32, mis, cols, c0 + u * T, same, v[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (c0 + u * T < chunks) rg_park8(reinterpret_cast<float*>(dst), mis, cols, c0 + u * T, v[u]);
            }
        }
    }
    const XT* x0 = xs + mis;
    const bool wide = mis == 0 && cols % 64 == 0;        // every eighth of the row is whole chunks
    auto elem = [&](const XT* p) {
        if constexpr (sizeof(V) == 2) return *p;
        else return (float)*p;
    };
    // sum over the row of term(x), which works on V and W alike; the column blocks are accumulated first, a chunk of
    // columns per thread
    auto sum_of = [&](auto term) {
        if (BLOCKED) {
            rg_barrier(group, T);                        // the row is parked
            for (int c = t; c < chunks; c += T) {
                W s = A::splat(m.acc_init);
#pragma unroll 4
                for (int jb = 0; jb < nb; ++jb) s = A::add(s, term(A::load(xs + jb * step + c * 8)));
                A::put(acc + c * 8, s);
            }
        }
        auto value = [&](int k) { return BLOCKED ? acc[mis + k] : term(elem(x0 + k)); };
        auto wide8 = [&](int k) {
            if constexpr (BLOCKED) return A::load(acc + k);
            else return term(A::load(xs + k));
        };
        auto first_wide = [&](V* dst) {
            if (!wide) return false;
            const int q = cols >> 3;                     // an eighth
            for (int i = t * 8; i < q; i += T * 8) {
                const W e0 = A::add(A::add(wide8(i), wide8(i + 4 * q)), A::add(wide8(i + 2 * q), wide8(i + 6 * q)));
                const W e1 = A::add(A::add(wide8(i + q), wide8(i + 5 * q)), A::add(wide8(i + 3 * q), wide8(i + 7 * q)));
                A::put(dst + i, A::add(e0, e1));
            }
            return true;
        };
        return A::back(rg_fold_with<V>(value, [](V p, V q) { return A::add(p, q); }, first_wide, tmp, cols, T, t, group));
    };
    float red0 = 0.f, red1 = 0.f, mean = 0.f;
    if (MODE != RP_RMS) red0 = sum_of([](auto x) { return x; });
    if (MODE == RP_LAYER) {
        mean = rg_row_value(a.scal[m.s_mean].prog, c_mean, red0, red1, vmr, T, t, group);
        const V mv = A::of(mean);
        const W mw = A::splat(mean);
        auto centre = [&](auto x) {
            if constexpr (sizeof(x) == sizeof(V)) {
                const V d = A::sub(x, mv);
                return A::mul(d, d);
            } else {
                const W d = A::sub(x, mw);
                return A::mul(d, d);
            }
        };
        red1 = sum_of(centre);
    }
    if (MODE == RP_RMS) red0 = sum_of([](auto x) { return A::mul(x, x); });
    if (a.out_per_row) {
        if (t == 0) {
            vmr[RG_VM_RED] = red0;
            vmr[RG_VM_RED + 1] = red1;
            const float o = rp_vm1(a.out.prog, vmr + RG_VM_RED, vmr, 1);
            const int64_t go = offs[a.n_in] + r * a.row_stride[a.n_in];
            if (a.dtype[a.n_in] == KTB_F16) reinterpret_cast<__half*>(a.arena)[go] = __float2half_rn(o);
            else reinterpret_cast<float*>(a.arena)[go] = o;
        }
        return;
    }
    if (MODE == RP_MEAN) return;                         // (a mean without an output tile is a per-row result)
    const float scale = rg_row_value(a.scal[m.s_scale].prog, c_scale, red0, red1, vmr, T, t, group);
    if (a.n_side && t == 0) {
        vmr[RG_VM_RED] = red0;
        vmr[RG_VM_RED + 1] = red1;
        if (MODE == RP_LAYER) vmr[RG_VM_SCAL + m.s_mean] = mean;
        vmr[RG_VM_SCAL + m.s_scale] = scale;
        rp_store_sides(a, row, vmr + RG_VM_RED, vmr, 1, vmr + RG_VM_SCAL, m.side_scal);
    }
    const W mw = A::splat(mean), sw = A::splat(scale);
    if constexpr (FAST) {
        const __half* base = reinterpret_cast<const __half*>(a.arena);
        const uint4* pw = reinterpret_cast<const uint4*>(base + w_off);
        const uint4* pb = reinterpret_cast<const uint4*>(base + b_off);
        const uint4* px = reinterpret_cast<const uint4*>(xs);
        uint4* py = reinterpret_cast<uint4*>(reinterpret_cast<__half*>(a.arena) + y_off);
        constexpr int U = 4;                             // chunks on their way per thread
        for (int i = t; i < n8; i += U * T) {
            uint4 w[U], b[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i + u * T < n8) {
                    if (m.has_w) w[u] = pw[i + u * T];
                    if (m.has_b) b[u] = pb[i + u * T];
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i + u * T < n8) {
                    W q = A::halves(px[i + u * T]);
                    if (MODE == RP_LAYER) q = A::sub(q, mw);
                    q = A::mul(q, sw);
                    if (m.has_w) q = A::mul(q, A::halves(w[u]));
                    if (m.has_b) q = A::add(q, A::halves(b[u]));
                    __stcs(py + i + u * T, A::to_halves(q));             // (a final rounding to f16 is this one)
                }
        }
    } else
    for (int jb = 0; jb < nb; ++jb) {
        const int64_t ya = y_off + jb * a.blk_stride[a.n_in];
        const int64_t wa = m.has_w ? w_off + jb * a.blk_stride[m.w] : 0, ba = m.has_b ? b_off + jb * a.blk_stride[m.b] : 0;
        const bool wsame = (wa & 7) == mis, bsame = (ba & 7) == mis, ysame = (ya & 7) == mis;
#pragma unroll 2
        for (int c = t; c < chunks; c += T) {
            float w[8], b[8], y[8];
            if (m.has_w) rg_load8(a.arena, wa, a.dtype[m.w], mis, cols, c, wsame, w);
            if (m.has_b) rg_load8(a.arena, ba, a.dtype[m.b], mis, cols, c, bsame, b);
            W q = A::load(xs + jb * pitch + c * 8);
            if (MODE == RP_LAYER) q = A::sub(q, mw);
            q = A::mul(q, sw);
            if (m.has_w) q = A::mul(q, A::from(w));
            if (m.has_b) q = A::add(q, A::from(b));
            A::floats(q, y);
            if (m.out_round16) {
#pragma unroll
                for (int v = 0; v < 8; ++v) y[v] = ktb_round16(y[v]);
            }
            rg_store8(a.arena, ya, a.dtype[a.n_in], mis, cols, c, ysame, y);
        }
    }
}

// Any other row program on rows of any length: the phases one after the other, each chunk through the interpreter, its
// values parked as floats for the fold.
__global__ void __launch_bounds__(256)
ktb_row_program_any_kernel(const __grid_constant__ ktb_rowprog_args a, int T, int64_t total_rows) {
    extern __shared__ __align__(16) float rg_smem[];
    float* regs = rg_smem + threadIdx.x;                 // the interpreter's registers, [register][element][thread]
    const int group = threadIdx.x / T;
    const int t = threadIdx.x - group * T;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x / T) + group;
    if (row >= total_rows) return;                       // whole row groups: the barriers are per group
    const int cols = a.cols;
    float* vmr = rg_smem + RP_REGS_BYTES / 4 + (size_t)group * (RG_VM_FLOATS + rg_fold_floats(cols) + rg_chunk_elems(cols));
    float* tmp = vmr + RG_VM_FLOATS;
    float* vals = tmp + rg_fold_floats(cols);
    const int64_t item = (uint32_t)row / (uint32_t)a.rows_per_item;
    const int64_t r = row - item * a.rows_per_item;
    int64_t off[KTB_VM_MAX_IN + 1];
#pragma unroll
    for (int k = 0; k <= KTB_VM_MAX_IN; ++k)
        off[k] = k <= a.n_in ? a.dev_item_offsets[item * (a.n_in + 1 + a.n_side) + k] + r * a.row_stride[k] : 0;
    const int mis = (int)(off[0] & 7), chunks = (cols + mis + 7) >> 3;
    float* red = vmr + RG_VM_RED;                        // written by the group's first thread, who alone reads them
    float scal[KTB_RP_MAX_SCAL] = {0.f, 0.f, 0.f, 0.f};
    if (t == 0) red[0] = red[1] = red[2] = 0.f;
    int scal_done = 0;
    for (int p = 0; p <= a.n_red; ++p) {
        if (p == a.n_red && a.out_per_row) {
            if (t == 0) {
                const float o = rp_vm1(a.out.prog, red, vmr, 1);
                if (a.dtype[a.n_in] == KTB_F16) reinterpret_cast<__half*>(a.arena)[off[a.n_in]] = __float2half_rn(o);
                else reinterpret_cast<float*>(a.arena)[off[a.n_in]] = o;
            }
            break;
        }
        if (p == a.n_red && a.n_side && t == 0) rp_store_sides(a, row, red, vmr, 1);
        if (p == a.n_red && a.n_side) rg_barrier(group, T);
        for (; scal_done < a.n_scal && a.scal[scal_done].ready_after < p; ++scal_done)
        {
            if (t == 0) vmr[RG_VM_RESULT] = rp_vm1(a.scal[scal_done].prog, red, vmr, 1);
            rg_barrier(group, T);
            const float v = vmr[RG_VM_RESULT];
#pragma unroll
            for (int q = 0; q < KTB_RP_MAX_SCAL; ++q)
                if (q == scal_done) scal[q] = v;
            rg_barrier(group, T);                        // (before the slot is written again)
        }
        const ktb_rp_phase& ph = p < a.n_red ? a.red[p] : a.out;
        const int nb = ph.blocked ? a.n_blocks : 1;
#pragma unroll
        for (int s = 0; s < KTB_RP_MAX_SCAL; ++s)
            if (s < a.n_scal && a.n_in + s < KTB_VM_REGS) {
#pragma unroll
                for (int v = 0; v < 8; ++v) regs[RP_REG(a.n_in + s, v)] = scal[s];
            }
        for (int jb = 0; jb < nb; ++jb)
            for (int c = t; c < chunks; c += T) {
#pragma unroll
                for (int k = 0; k < KTB_VM_MAX_IN; ++k)
                    if (k < a.n_in && (((ph.load_mask >> k) & 1) || (ph.prog.n_ops == 0 && ph.prog.result_reg == k))) {
                        const int64_t at = off[k] + jb * a.blk_stride[k];
                        float in[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                        rg_load8(a.arena, at, a.dtype[k], mis, cols, c, (at & 7) == mis, in);
#pragma unroll
                        for (int v = 0; v < 8; ++v) regs[RP_REG(k, v)] = in[v];
                    }
                if (ph.prog.n_ops) rp_vm8(ph.prog, regs);
                float val[8];
#pragma unroll
                for (int v = 0; v < 8; ++v) val[v] = regs[RP_REG(ph.prog.result_reg, v)];
                if (p == a.n_red) {
                    const int64_t at = off[a.n_in] + jb * a.blk_stride[a.n_in];
                    rg_store8(a.arena, at, a.dtype[a.n_in], mis, cols, c, (at & 7) == mis, val);
                    continue;
                }
                if (ph.blocked) {
#pragma unroll
                    for (int v = 0; v < 8; ++v) {
                        const float s = (jb == 0 ? ph.acc_init : vals[c * 8 + v]) + val[v];
                        val[v] = ph.acc_round16 ? ktb_round16(s) : s;
                    }
                }
                rg_park8(vals, mis, cols, c, val);
            }
        if (p < a.n_red) {
            const float* first = vals + mis;
            auto value = [=](int i) { return first[i]; };
            const float f = ph.op == KTB_RP_ADD ? (ph.round16 ? rg_fold<1, false, true>(value, tmp, cols, T, t, group)
                                                       : rg_fold<1, false, false>(value, tmp, cols, T, t, group))
                     : ph.op == KTB_RP_MAXNUM ? rg_fold<0, true, false>(value, tmp, cols, T, t, group)
                                              : rg_fold<0, false, false>(value, tmp, cols, T, t, group);
            if (t == 0) red[p] = f;
        }
    }
}

// Largest dynamic shared memory of a CTA on this architecture.
#define RG_SMEM_MOST (227 * 1024)

// The skeleton kernel, if the rows (all their blocks) fit shared memory; false if not.
static bool rp_try_norm_any(ktb_ctx* ctx, const ktb_rowprog_args& a, const rp_norm& m, int64_t total_rows, int* rc) {
    const int nb = m.blocked ? a.n_blocks : 1;
    const bool f16 = a.dtype[m.x] == KTB_F16;
    // halves only where every tile is f16: an f32 weight tile of an f16-rounding kernel needs f32 operands
    const bool wb16 = (!m.has_w || a.dtype[m.w] == KTB_F16) && (!m.has_b || a.dtype[m.b] == KTB_F16);
    const bool halves = f16 && m.r16 && wb16;
    if ((int64_t)nb * a.cols > (1 << 20)) return false;
    bool fast = f16 && wb16 && a.aligned && (a.out_per_row || a.dtype[a.n_in] == KTB_F16) && a.cols % 8 == 0;
    for (int q = 0; nb > 1 && q <= a.n_in; ++q)
        if (q == m.x || (q == a.n_in && !a.out_per_row) || (m.has_w && q == m.w) || (m.has_b && q == m.b)) fast = fast && a.blk_stride[q] == a.cols;
    const int row_bytes = rg_norm_bytes(a.cols, nb, f16 ? 2 : 4, halves ? 2 : 4, m.blocked);
    rg_split s = rg_choose_norm((int64_t)nb * a.cols, total_rows, ctx->sm_count, 256);
    while (s.groups > 1 && s.groups * row_bytes > RG_SMEM_MOST) s.groups /= 2;
    if (s.groups * row_bytes > RG_SMEM_MOST) return false;
    rp_chain none = {};
    none.n = -1;
    const rp_chain mean = m.s_mean >= 0 ? rp_make_chain(a.scal[m.s_mean].prog, a.n_red) : none;
    const rp_chain scale = m.s_scale >= 0 ? rp_make_chain(a.scal[m.s_scale].prog, a.n_red) : none;
    using kernel = void (*)(const ktb_rowprog_args, const rp_norm, const rp_chain, const rp_chain, int, int64_t, ktb_status*);
    kernel k = nullptr;
#define RG_PICK(MODE, BLK)                                                                                        \
    if (m.mode == MODE && (m.blocked != 0) == BLK)                                                                \
        k = fast ? (halves  ? ktb_row_norm_any_kernel<__half, rg_f16, MODE, BLK, true>                            \
                    : m.r16 ? ktb_row_norm_any_kernel<__half, rg_f32<true>, MODE, BLK, true>                      \
                            : ktb_row_norm_any_kernel<__half, rg_f32<false>, MODE, BLK, true>)                    \
            : halves ? ktb_row_norm_any_kernel<__half, rg_f16, MODE, BLK, false>                                  \
            : f16  ? (m.r16 ? ktb_row_norm_any_kernel<__half, rg_f32<true>, MODE, BLK, false>                     \
                            : ktb_row_norm_any_kernel<__half, rg_f32<false>, MODE, BLK, false>)                   \
                   : (m.r16 ? ktb_row_norm_any_kernel<float, rg_f32<true>, MODE, BLK, false>                      \
                            : ktb_row_norm_any_kernel<float, rg_f32<false>, MODE, BLK, false>);
    RG_PICK(RP_RMS, false) RG_PICK(RP_MEAN, false) RG_PICK(RP_LAYER, false)
    RG_PICK(RP_RMS, true) RG_PICK(RP_MEAN, true) RG_PICK(RP_LAYER, true)
#undef RG_PICK
    const size_t smem = (size_t)(s.groups * row_bytes);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) {
            *rc = ktb_fail(ctx, KTB_E_CUDA, "row_program_any", cudaGetErrorString(e));
            return true;
        }
    }
    const unsigned blocks = (unsigned)((total_rows + s.groups - 1) / s.groups);
    k<<<blocks, s.threads * s.groups, smem, ctx->stream>>>(a, m, mean, scale, s.threads, total_rows, ctx->dev_status);
    const cudaError_t e = cudaGetLastError();
    *rc = e == cudaSuccess ? KTB_OK : ktb_fail(ctx, KTB_E_CUDA, "ktb_row_norm_any_kernel", cudaGetErrorString(e));
    if (*rc == KTB_OK) ctx->launches++;
    return true;
}

static int rp_launch_any(ktb_ctx* ctx, const ktb_rowprog_args& a, int64_t total_rows) {
    rg_split s = rg_choose_norm(a.cols, total_rows, ctx->sm_count, 256);
    const int64_t row_bytes = 4ll * (RG_VM_FLOATS + rg_fold_floats(a.cols) + rg_chunk_elems(a.cols));
    while (s.groups > 1 && (int64_t)RP_REGS_BYTES + s.groups * row_bytes > RG_SMEM_MOST) s.groups /= 2;
    const size_t smem = RP_REGS_BYTES + (size_t)(s.groups * row_bytes);
    KTB_CUDA(ctx, cudaFuncSetAttribute(ktb_row_program_any_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const unsigned blocks = (unsigned)((total_rows + s.groups - 1) / s.groups);
    ktb_row_program_any_kernel<<<blocks, s.threads * s.groups, smem, ctx->stream>>>(a, s.threads, total_rows);
    KTB_CHECK_LAUNCH(ctx, "ktb_row_program_any_kernel");
    return KTB_OK;
}
