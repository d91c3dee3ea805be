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

// Row value `prog` for the whole group: as a chain by every thread, else by the first one through shared memory.
static __device__ __forceinline__ float rg_row_value(const ktb_vm_program& prog, const rp_chain& c, const float* red, float* vmr,
                                                     int T, int t, int group) {
    if (c.n >= 0) return rp_run_chain(c, red[c.red]);
    if (t == 0) vmr[KTB_VM_REGS] = rp_vm1(prog, red, vmr, 1);
    rg_barrier(group, T);
    const float v = vmr[KTB_VM_REGS];
    rg_barrier(group, T);                                // (before the slot is written again)
    return v;
}
#define RG_VM_FLOATS (KTB_VM_REGS + 4)

// One thread per about 40 elements of a row, in whole warps; more where the rows are few.
static rg_split rg_choose_norm(int64_t elems, int64_t rows, int sm_count, int most) {
    rg_split s = {};
    int T = (int)((elems + 1279) / 1280) * 32;
    while (T < most && rows * T < (int64_t)sm_count * 512 && T * 8 < elems) T *= 2;
    s.threads = T > most ? most : T;
    s.groups = s.threads == 32 ? 8 : s.threads <= 64 ? 4 : s.threads <= 128 ? 2 : 1;
    return s;
}

// The normalisation skeletons (rp_norm) of rows of any length, column blocks included.  The row is parked in shared
// memory in its own dtype (all blocks, one read of HBM); the sums read their terms from there — term and block
// accumulation are evaluated as the first fold level reads them — and so does the output.  No row values in
// registers: 16 rows or so per SM are in flight.  Bound by issue (about 25 instructions per element and sum with
// f16 rounding, 8 without) next to HBM.  rms norm with weights and 1/rms
// stored, f16[2048, 5120]: 849 us in 61 steps, 28.7 us here (6.5 at the measured copy rate).
template <typename XT, bool R16>
__global__ void __launch_bounds__(512)
ktb_row_norm_any_kernel(const __grid_constant__ ktb_rowprog_args a, const __grid_constant__ rp_norm m,
                        const __grid_constant__ rp_chain c_mean, const __grid_constant__ rp_chain c_scale, int T, int64_t total_rows) {
    extern __shared__ __align__(16) float rg_smem[];
    const int group = threadIdx.x / T;
    const int t = threadIdx.x - group * T;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x / T) + group;
    if (row >= total_rows) return;                       // whole row groups: the barriers are per group
    const int cols = a.cols, nb = m.blocked ? a.n_blocks : 1, pitch = rg_chunk_elems(cols);
    constexpr int XF = sizeof(XT);                       // bytes per parked element
    float* vmr = rg_smem + (size_t)group * (RG_VM_FLOATS + rg_fold_floats(cols) + nb * pitch * XF / 4);
    float* tmp = vmr + RG_VM_FLOATS;
    XT* xs = reinterpret_cast<XT*>(tmp + rg_fold_floats(cols));
    const int64_t item = (uint32_t)row / (uint32_t)a.rows_per_item;
    const int64_t r = row - item * a.rows_per_item;
    const int64_t* offs = a.dev_item_offsets + item * (a.n_in + 1 + a.n_side);
    const int64_t x_off = offs[m.x] + r * a.row_stride[m.x];
    const int mis = (int)(x_off & 7), chunks = (cols + mis + 7) >> 3;
    auto rnd = [](float v) { return R16 ? ktb_round16(v) : v; };

    for (int jb = 0; jb < nb; ++jb) {
        const int64_t at = x_off + jb * a.blk_stride[m.x];
        const bool same = (at & 7) == mis;
        XT* dst = xs + jb * pitch;
        for (int c0 = t; c0 < chunks; c0 += 4 * T) {     // four chunks on their way per thread
            if constexpr (XF == 2) {
                uint4 raw[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    raw[u] = make_uint4(0, 0, 0, 0);
                    if (same) rg_load_h(reinterpret_cast<const __half*>(a.arena) + at, mis, cols, c0 + u * T, raw[u]);
                    else rg_load_h_apart(reinterpret_cast<const __half*>(a.arena) + at, mis, cols, c0 + u * T, raw[u]);
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
    auto elem = [&](int jb, int k) {
        if constexpr (XF == 2) return __half2float(x0[jb * pitch + k]);
        else return (float)x0[jb * pitch + k];
    };
    float red[KTB_RP_MAX_RED] = {0.f, 0.f, 0.f};
    float mean = 0.f;
    if (m.mode != RP_RMS) {
        red[0] = rg_fold<1, false, R16>([&](int k) {
            if (!m.blocked) return elem(0, k);
            float s = m.acc_init;
            for (int jb = 0; jb < nb; ++jb) s = rnd(s + elem(jb, k));
            return s;
        }, tmp, cols, T, t, group);
        if (m.mode == RP_LAYER) mean = rg_row_value(a.scal[m.s_mean].prog, c_mean, red, vmr, T, t, group);
    }
    if (m.mode != RP_MEAN) {
        const bool centred = m.mode == RP_LAYER;
        const float sq = rg_fold<1, false, R16>([&](int k) {
            auto term = [&](float x) {
                const float d = centred ? rnd(x - mean) : x;
                return rnd(d * d);
            };
            if (!m.blocked) return term(elem(0, k));
            float s = m.acc_init;
            for (int jb = 0; jb < nb; ++jb) s = rnd(s + term(elem(jb, k)));
            return s;
        }, tmp, cols, T, t, group);
        if (centred) red[1] = sq;
        else red[0] = sq;
    }
    if (a.out_per_row) {
        if (t == 0) {
            const float o = rp_vm1(a.out.prog, red, vmr, 1);
            const int64_t go = offs[a.n_in] + r * a.row_stride[a.n_in];
            if (a.dtype[a.n_in] == KTB_F16) reinterpret_cast<__half*>(a.arena)[go] = __float2half_rn(o);
            else reinterpret_cast<float*>(a.arena)[go] = o;
        }
        return;
    }
    const float scale = rg_row_value(a.scal[m.s_scale].prog, c_scale, red, vmr, T, t, group);
    if (a.n_side && t == 0) {
        float scal[KTB_RP_MAX_SCAL] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < KTB_RP_MAX_SCAL; ++q) scal[q] = q == m.s_scale ? scale : q == m.s_mean ? mean : 0.f;
        rp_store_sides(a, row, red, vmr, 1, scal, m.side_scal);
    }
    const int64_t y_off = offs[a.n_in] + r * a.row_stride[a.n_in];
    const int64_t w_off = m.has_w ? offs[m.w] + r * a.row_stride[m.w] : 0;
    const int64_t b_off = m.has_b ? offs[m.b] + r * a.row_stride[m.b] : 0;
    for (int jb = 0; jb < nb; ++jb) {
        const int64_t ya = y_off + jb * a.blk_stride[a.n_in];
        const int64_t wa = m.has_w ? w_off + jb * a.blk_stride[m.w] : 0, ba = m.has_b ? b_off + jb * a.blk_stride[m.b] : 0;
        for (int c = t; c < chunks; c += T) {
            float w[8], b[8], y[8];
            if (m.has_w) rg_load8(a.arena, wa, a.dtype[m.w], mis, cols, c, (wa & 7) == mis, w);
            if (m.has_b) rg_load8(a.arena, ba, a.dtype[m.b], mis, cols, c, (ba & 7) == mis, b);
            if constexpr (XF == 2) {
                const uint4 raw = *reinterpret_cast<const uint4*>(xs + jb * pitch + c * 8);
                const __half* h = reinterpret_cast<const __half*>(&raw);
#pragma unroll
                for (int v = 0; v < 8; ++v) y[v] = __half2float(h[v]);
            } else {
                const float* p = reinterpret_cast<const float*>(xs) + jb * pitch + c * 8;
                const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 4);
                y[0] = lo.x; y[1] = lo.y; y[2] = lo.z; y[3] = lo.w;
                y[4] = hi.x; y[5] = hi.y; y[6] = hi.z; y[7] = hi.w;
            }
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                float q = m.mode == RP_LAYER ? rnd(y[v] - mean) : y[v];
                q = rnd(q * scale);
                if (m.has_w) q = rnd(q * w[v]);
                if (m.has_b) q = rnd(q + b[v]);
                y[v] = m.out_round16 ? ktb_round16(q) : q;
            }
            rg_store8(a.arena, ya, a.dtype[a.n_in], mis, cols, c, (ya & 7) == mis, y);
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
    rp_chain none = {};
    none.n = -1;

    float red[KTB_RP_MAX_RED] = {0.f, 0.f, 0.f};
    float scal[KTB_RP_MAX_SCAL] = {0.f, 0.f, 0.f, 0.f};
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
            scal[scal_done] = rg_row_value(a.scal[scal_done].prog, none, red, vmr, T, t, group);
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
            red[p] = ph.op == KTB_RP_ADD ? (ph.round16 ? rg_fold<1, false, true>(value, tmp, cols, T, t, group)
                                                       : rg_fold<1, false, false>(value, tmp, cols, T, t, group))
                     : ph.op == KTB_RP_MAXNUM ? rg_fold<0, true, false>(value, tmp, cols, T, t, group)
                                              : rg_fold<0, false, false>(value, tmp, cols, T, t, group);
        }
    }
}

// Largest dynamic shared memory of a CTA on this architecture.
#define RG_SMEM_MOST (227 * 1024)

// The skeleton kernel, if the rows (all their blocks) fit shared memory; false if not.
static bool rp_try_norm_any(ktb_ctx* ctx, const ktb_rowprog_args& a, const rp_norm& m, int64_t total_rows, int* rc) {
    const int nb = m.blocked ? a.n_blocks : 1;
    const bool f16 = a.dtype[m.x] == KTB_F16;
    rg_split s = rg_choose_norm((int64_t)nb * a.cols, total_rows, ctx->sm_count, 512);
    const int64_t row_bytes = 4ll * (RG_VM_FLOATS + rg_fold_floats(a.cols)) + (int64_t)nb * rg_chunk_elems(a.cols) * (f16 ? 2 : 4);
    while (s.groups > 1 && s.groups * row_bytes > RG_SMEM_MOST) s.groups /= 2;
    if (s.groups * row_bytes > RG_SMEM_MOST) return false;
    rp_chain none = {};
    none.n = -1;
    const rp_chain mean = m.s_mean >= 0 ? rp_make_chain(a.scal[m.s_mean].prog, a.n_red) : none;
    const rp_chain scale = m.s_scale >= 0 ? rp_make_chain(a.scal[m.s_scale].prog, a.n_red) : none;
    auto k = f16 ? (m.r16 ? ktb_row_norm_any_kernel<__half, true> : ktb_row_norm_any_kernel<__half, false>)
                 : (m.r16 ? ktb_row_norm_any_kernel<float, true> : ktb_row_norm_any_kernel<float, false>);
    const size_t smem = (size_t)(s.groups * row_bytes);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) {
            *rc = ktb_fail(ctx, KTB_E_CUDA, "row_program_any", cudaGetErrorString(e));
            return true;
        }
    }
    const unsigned blocks = (unsigned)((total_rows + s.groups - 1) / s.groups);
    k<<<blocks, s.threads * s.groups, smem, ctx->stream>>>(a, m, mean, scale, s.threads, total_rows);
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
