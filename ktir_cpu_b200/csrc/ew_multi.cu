// Several elementwise stores over the same tiles in one launch.
//
// A loop body that stores a handful of tiles computed from the same loads (ktir_cpu/interpreter.py:196-281 runs every
// op of it by itself) reads each input once here; every output is a short register program over the loaded values.
// Programs of one op work on registers; longer ones run on registers in shared memory, [register][element][thread].
// Bound by issue (the transcendentals) next to HBM.  add, mul, exp, tanh, erf, select and an f32 add of f16[2^22]:
// 682 us as 41 launches (erf 31, select 5), 33 here (11.7 at the measured copy rate);
// blocks of 333 elements that start anywhere, f16[3196800]: 30.8.
#include "row_fold.cuh"
#include "vm.cuh"

// A predicate is the set of outcomes it holds for: less, equal, greater, unordered.
static __device__ __forceinline__ bool em_cmp(int pred, float a, float b) {
    const int outcome = a < b ? KTB_CMP_LT : a == b ? KTB_CMP_EQ : a > b ? KTB_CMP_GT : KTB_CMP_UNORDERED;
    return (pred & outcome) != 0;
}

static __device__ __forceinline__ float em_sign(float a) { return a > 0.f ? 1.f : a < 0.f ? -1.f : a == 0.f ? 0.f : a; }

// Abramowitz & Stegun 7.1.26 in the reference's order of ops, each rounded to f32 ...
static __device__ __forceinline__ float em_erf32(float x) {
    const float a = fabsf(x);
    const float t = 1.0f / (1.0f + 0.3275911f * a);
    float p = t * 1.061405429f;
    p = t * (-1.453152027f + p);
    p = t * (1.421413741f + p);
    p = t * (-0.284496736f + p);
    p = t * (0.254829592f + p);
    const float e = expf(-a * a);
    return em_sign(x) * (1.0f - p * e);
}
// ... and for two f16 values with every op rounded to f16: adds and products of halves are the rounded f32 ops, the
// quotient and the exponential go through f32.
static __device__ __forceinline__ __half2 em_erf16(__half2 x) {
    auto c = [](float v) { return __float2half2_rn(v); };
    const __half2 a = __habs2(x);
    const float2 s = __half22float2(__hadd2_rn(c(1.0f), __hmul2_rn(c(0.3275911f), a)));
    const __half2 t = __floats2half2_rn(1.0f / s.x, 1.0f / s.y);
    __half2 p = __hmul2_rn(t, c(1.061405429f));
    p = __hmul2_rn(t, __hadd2_rn(c(-1.453152027f), p));
    p = __hmul2_rn(t, __hadd2_rn(c(1.421413741f), p));
    p = __hmul2_rn(t, __hadd2_rn(c(-0.284496736f), p));
    p = __hmul2_rn(t, __hadd2_rn(c(0.254829592f), p));
    const float2 q = __half22float2(__hmul2_rn(__hneg2(a), a));
    const __half2 e = __floats2half2_rn(expf(q.x), expf(q.y));
    const float2 f = __half22float2(x);
    return __hmul2_rn(__floats2half2_rn(em_sign(f.x), em_sign(f.y)), __hsub2_rn(c(1.0f), __hmul2_rn(p, e)));
}

// The longer ops, four values at a time and out of line: inlined in the switch below, the compiler computed every op and
// selected one (181 instructions per element for an exp), and the argument reduction of sin and cos wants a stack,
// which dragged the values into memory.
#define EM_FN(NAME, EXPR)                                                    \
    static __device__ __noinline__ float4 NAME(float4 A) {                   \
        auto f = [](float a) { return EXPR; };                               \
        return make_float4(f(A.x), f(A.y), f(A.z), f(A.w));                  \
    }
EM_FN(em_exp, expf(a))
EM_FN(em_log, logf(a))
EM_FN(em_log2, log2f(a))
EM_FN(em_sqrt, sqrtf(a))
EM_FN(em_rsqrt, 1.0f / sqrtf(a))
EM_FN(em_rsqrt16, 1.0f / ktb_round16(sqrtf(a)))
EM_FN(em_tanh, tanhf(a))
EM_FN(em_sin, sinf(a))
EM_FN(em_cos, cosf(a))
EM_FN(em_erf, em_erf32(a))
static __device__ __noinline__ float4 em_erf_f16(float4 A) {
    const float2 lo = __half22float2(em_erf16(__floats2half2_rn(A.x, A.y))), hi = __half22float2(em_erf16(__floats2half2_rn(A.z, A.w)));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
#define EM_FN2(NAME, EXPR)                                                              \
    static __device__ __noinline__ float4 NAME(float4 A, float4 B) {                    \
        auto f = [](float a, float b) { return EXPR; };                                 \
        return make_float4(f(A.x, B.x), f(A.y, B.y), f(A.z, B.z), f(A.w, B.w));         \
    }
EM_FN2(em_div, a / b)
EM_FN2(em_max, (a >= b || a != a) ? a : b)
EM_FN2(em_maxnum, (a >= b || b != b) ? a : b)
EM_FN2(em_min, (a <= b || a != a) ? a : b)
EM_FN2(em_minnum, (a <= b || b != b) ? a : b)

#define EM_LANES(EXPR)                                     \
    {                                                      \
        _Pragma("unroll") for (int v = 0; v < 8; ++v) {    \
            const float a = A[v];                          \
            (void)a;                                       \
            R[v] = (EXPR);                                 \
        }                                                  \
    }                                                      \
    break;
#define EM_LANES2(EXPR)                                    \
    {                                                      \
        _Pragma("unroll") for (int v = 0; v < 8; ++v) {    \
            const float a = A[v], b = B[v];                \
            R[v] = (EXPR);                                 \
        }                                                  \
    }                                                      \
    break;
#define EM_CALL(FN)                                                        \
    {                                                                      \
        em_split(R, FN(make_float4(A[0], A[1], A[2], A[3])), 0);           \
        em_split(R, FN(make_float4(A[4], A[5], A[6], A[7])), 4);           \
    }                                                                      \
    break;
#define EM_CALL2(FN)                                                                                                        \
    {                                                                                                                       \
        em_split(R, FN(make_float4(A[0], A[1], A[2], A[3]), make_float4(B[0], B[1], B[2], B[3])), 0);                       \
        em_split(R, FN(make_float4(A[4], A[5], A[6], A[7]), make_float4(B[4], B[5], B[6], B[7])), 4);                       \
    }                                                                                                                       \
    break;
static __device__ __forceinline__ void em_split(float (&R)[8], float4 q, int at) {
    R[at] = q.x; R[at + 1] = q.y; R[at + 2] = q.z; R[at + 3] = q.w;
}

// One op on eight values; get(r, X) fetches register r.  `round`: apply the op's own final rounding (not needed where
// the result is stored as f16 at once).
template <typename G>
static __device__ __forceinline__ void em_op(const ktb_vm_op& op, G get, bool round, float (&R)[8]) {
    const int code = op.opcode & 0xff;
    const bool r16 = (op.opcode & KTB_VM_ROUND16) != 0;
    float A[8];
    get(op.a, A);
    if (code >= KTB_VM_ADD && code <= KTB_VM_MINNUM) {
        float B[8];
        get(op.b, B);
        switch (code) {
            case KTB_VM_ADD: EM_LANES2(a + b)
            case KTB_VM_SUB: EM_LANES2(a - b)
            case KTB_VM_MUL: EM_LANES2(a * b)
            case KTB_VM_DIV: EM_CALL2(em_div)
            case KTB_VM_MAX: EM_CALL2(em_max)
            case KTB_VM_MAXNUM: EM_CALL2(em_maxnum)
            case KTB_VM_MIN: EM_CALL2(em_min)
            default: EM_CALL2(em_minnum)
        }
    } else {
        switch (code) {
            case KTB_VM_MOV: EM_LANES(a)
            case KTB_VM_CONST: EM_LANES(op.imm)
            case KTB_VM_NEG: EM_LANES(-a)
            case KTB_VM_ABS: EM_LANES(fabsf(a))
            case KTB_VM_EXP: EM_CALL(em_exp)
            case KTB_VM_LOG: EM_CALL(em_log)
            case KTB_VM_LOG2: EM_CALL(em_log2)
            case KTB_VM_SQRT: EM_CALL(em_sqrt)
            case KTB_VM_RSQRT: EM_CALL(em_rsqrt)
            case KTB_VM_TANH: EM_CALL(em_tanh)
            case KTB_VM_SIN: EM_CALL(em_sin)
            case KTB_VM_COS: EM_CALL(em_cos)
            case KTB_VM_FMA: {
                float B[8], C[8];
                get(op.b, B);
                get(op.c, C);
#pragma unroll
                for (int v = 0; v < 8; ++v) R[v] = __fadd_rn(__fmul_rn(A[v], B[v]), C[v]);
                break;
            }
            case KTB_VM_CSEL: {
                const int pred = (int)op.imm >> 3;
                float B[8];
                get(op.b, B);
                uint32_t take = 0;
#pragma unroll
                for (int v = 0; v < 8; ++v) take |= (em_cmp(pred, A[v], B[v]) ? 1u : 0u) << v;
                get(op.c, A);
                get((int)op.imm & 7, B);
#pragma unroll
                for (int v = 0; v < 8; ++v) R[v] = (take >> v) & 1 ? A[v] : B[v];
                break;
            }
            case KTB_VM_RSQRT_STEPS:
                if (r16) {
                    EM_CALL(em_rsqrt16)
                } else {
                    EM_CALL(em_rsqrt)
                }
            default:                                       // KTB_VM_ERF
                if (r16) {
                    EM_CALL(em_erf_f16)
                } else {
                    EM_CALL(em_erf)
                }
        }
    }
    if (r16 && round) {
#pragma unroll
        for (int v = 0; v < 8; ++v) R[v] = ktb_round16(R[v]);
    }
}

// A program of several ops on registers in shared memory; the inputs are there already.  (Out of line: one copy.)
#define EM_REG(q, v) (((q) * 8 + (v)) * 256)
static __device__ __noinline__ void em_run(const ktb_vm_program& p, float* regs) {
    for (int i = 0; i < p.n_ops; ++i) {
        const ktb_vm_op op = p.ops[i];
        float R[8];
        em_op(op, [&](int r, float (&X)[8]) {
#pragma unroll
            for (int v = 0; v < 8; ++v) X[v] = regs[EM_REG(r, v)];
        }, true, R);
#pragma unroll
        for (int v = 0; v < 8; ++v) regs[EM_REG(op.dst, v)] = R[v];
    }
}

// Where chunk `at` of the launch lies: item, row of the tile, chunk of the row.
struct em_place {
    const int64_t* offs;
    uint32_t row, chunk;
    __device__ __forceinline__ em_place(const ktb_ew_multi_args& a, uint32_t per_row, uint32_t per_item, uint64_t at) {
        const uint32_t item = at < (1ull << 32) ? (uint32_t)at / per_item : (uint32_t)(at / per_item);
        const uint32_t rem = (uint32_t)(at - (uint64_t)item * per_item);
        row = rem / per_row;
        chunk = rem - row * per_row;
        offs = a.dev_item_offsets + (int64_t)item * (a.n_in + a.n_out);
    }
    // first element of operand k's row (inputs, then outputs)
    __device__ __forceinline__ int64_t at(const ktb_ew_multi_args& a, int k) const { return offs[k] + (int64_t)row * a.row_stride[k]; }
};

template <int NIN>
static __device__ __forceinline__ void em_pick(const float (&x)[NIN][8], int r, float (&o)[8]) {
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        o[v] = x[0][v];
#pragma unroll
        for (int k = 1; k < NIN; ++k) o[v] = r == k ? x[k][v] : o[v];
    }
}

// All programs over the eight values of each input; store(o, R) takes the result of output o.
template <int NIN, typename S>
static __device__ __forceinline__ void em_outputs(const ktb_ew_multi_args& a, const float (&x)[NIN][8], float* regs, S store) {
    for (int o = 0; o < a.n_out; ++o) {
        const ktb_vm_program& p = a.program[o];
        float R[8];
        if (p.n_ops == 0) {
            em_pick<NIN>(x, p.result_reg, R);
        } else if (p.n_ops == 1) {
            em_op(p.ops[0], [&](int r, float (&X)[8]) { em_pick<NIN>(x, r, X); }, a.dtype[a.n_in + o] != KTB_F16, R);
        } else {
#pragma unroll
            for (int k = 0; k < NIN; ++k)
                if (k < a.n_in) {
#pragma unroll
                    for (int v = 0; v < 8; ++v) regs[EM_REG(k, v)] = x[k][v];
                }
            em_run(p, regs);
#pragma unroll
            for (int v = 0; v < 8; ++v) R[v] = regs[EM_REG(p.result_reg, v)];
        }
        store(o, R);
    }
}

// Whole chunks on 16-byte boundaries.  A thread takes `per_thread` (up to U) chunks 256 apart and asks for all their
// vectors before it works on the first: one chunk per thread left the kernel waiting (exp f32[2^24] 78 us).  `H`:
// every input is f16 (one vector per chunk and input, else two).
template <int NIN, bool H>
__global__ void __launch_bounds__(256, 4) ktb_ew_multi_kernel(const __grid_constant__ ktb_ew_multi_args a, uint32_t per_row, uint32_t per_item,
                                                              uint64_t total, int per_thread) {
    constexpr int U = H && NIN <= 2 ? 4 : NIN == 1 || H ? 2 : 1, L = H ? 1 : 2;
    extern __shared__ float em_regs[];
    const uint64_t first = (uint64_t)blockIdx.x * (256 * per_thread) + threadIdx.x;
    if (first >= total) return;
    uint4 raw[U][NIN][L];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint64_t at = first + u * 256;
        if (u < per_thread && at < total) {
            const em_place p(a, per_row, per_item, at);
#pragma unroll
            for (int k = 0; k < NIN; ++k)
                if (k < a.n_in) {
                    const int64_t e = p.at(a, k) + p.chunk * 8;
                    if (H || a.dtype[k] == KTB_F16) {
                        raw[u][k][0] = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(a.arena) + e));
                    } else {
                        raw[u][k][0] = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(a.arena) + e));
                        raw[u][k][L - 1] = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(a.arena) + e + 4));
                    }
                }
        }
    }
#pragma unroll 1
    for (int u = 0; u < per_thread; ++u) {
        const uint64_t at = first + (uint64_t)u * 256;
        if (at >= total) return;
        const em_place p(a, per_row, per_item, at);
        float x[NIN][8];
#pragma unroll
        for (int k = 0; k < NIN; ++k)
            if (k < a.n_in) {
                if (H || a.dtype[k] == KTB_F16) {
                    const __half2* h = reinterpret_cast<const __half2*>(&raw[0][k][0]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __half22float2(h[i]);
                        x[k][2 * i] = f.x;
                        x[k][2 * i + 1] = f.y;
                    }
                } else {
                    const float* f = reinterpret_cast<const float*>(&raw[0][k][0]);
                    const float* g = reinterpret_cast<const float*>(&raw[0][k][L - 1]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[k][i] = f[i], x[k][4 + i] = g[i];
                }
            }
        // the next chunk's vectors move up: the loop stays one copy of the code and `raw` in registers
#pragma unroll
        for (int w = 0; w + 1 < U; ++w)
#pragma unroll
            for (int k = 0; k < NIN; ++k)
#pragma unroll
                for (int l = 0; l < L; ++l) raw[w][k][l] = raw[w + 1][k][l];
        em_outputs<NIN>(a, x, em_regs + threadIdx.x, [&](int o, const float (&R)[8]) {
            ktb_store_vec<8>(a.arena, p.at(a, a.n_in + o) + p.chunk * 8, a.dtype[a.n_in + o], R);
        });
    }
}

// Rows of any length that start anywhere: chunks are laid out on the first input's boundaries (row_fold.cuh), whole
// ones move as vectors where the other tiles lie the same way, the ends element by element.
template <int NIN>
__global__ void __launch_bounds__(256, 4) ktb_ew_multi_any_kernel(const __grid_constant__ ktb_ew_multi_args a, uint32_t per_row,
                                                                  uint32_t per_item, uint64_t total) {
    extern __shared__ float em_regs[];
    const uint64_t at = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    if (at >= total) return;
    const em_place p(a, per_row, per_item, at);
    const int mis = (int)(p.at(a, 0) & 7), c = (int)p.chunk, cols = a.cols;
    if (!rg_any(c, mis, cols)) return;
    float x[NIN][8];
#pragma unroll
    for (int k = 0; k < NIN; ++k) {
#pragma unroll
        for (int v = 0; v < 8; ++v) x[k][v] = 0.f;
        if (k < a.n_in) {
            const int64_t off = p.at(a, k);
            rg_load8(a.arena, off, a.dtype[k], mis, cols, c, (off & 7) == mis, x[k]);
        }
    }
    em_outputs<NIN>(a, x, em_regs + threadIdx.x, [&](int o, const float (&R)[8]) {
        const int64_t off = p.at(a, a.n_in + o);
        rg_store8(a.arena, off, a.dtype[a.n_in + o], mis, cols, c, (off & 7) == mis, R);
    });
}

// Registers that an op reads, as bits.
static uint32_t em_reads(const ktb_vm_op& op) {
    const int code = op.opcode & 0xff;
    if (code == KTB_VM_CONST) return 0;
    uint32_t r = 1u << op.a;
    if ((code >= KTB_VM_ADD && code <= KTB_VM_MINNUM) || code == KTB_VM_FMA || code == KTB_VM_CSEL) r |= 1u << op.b;
    if (code == KTB_VM_FMA || code == KTB_VM_CSEL) r |= 1u << op.c;
    if (code == KTB_VM_CSEL) r |= 1u << ((int)op.imm & 7);
    return r;
}

extern "C" int ktb_launch_ew_multi(ktb_ctx* ctx, const ktb_ew_multi_args* args) {
    if (!ctx || !args) return KTB_E_ARG;
    const ktb_ew_multi_args& a = *args;
    if (a.n_in < 1 || a.n_in > KTB_VM_MAX_IN || a.n_out < 1 || a.n_out > KTB_EW_MAX_OUT)
        return ktb_fail(ctx, KTB_E_ARG, "ew_multi", "bad operand counts");
    int regs = 0;                                        // shared registers that the longer programs use
    for (int o = 0; o < a.n_out; ++o) {
        const ktb_vm_program& p = a.program[o];
        if (p.n_in != a.n_in || p.n_ops < 0 || p.n_ops > KTB_VM_MAX_OPS || p.result_reg < 0 || p.result_reg >= KTB_VM_REGS ||
            (p.n_ops == 0 && p.result_reg >= a.n_in))
            return ktb_fail(ctx, KTB_E_ARG, "ew_multi", "bad program header");
        uint32_t held = (1u << a.n_in) - 1;              // registers that hold a value: the inputs, then what has been written
        for (int i = 0; i < p.n_ops; ++i) {
            const ktb_vm_op& op = p.ops[i];
            const int code = op.opcode & 0xff;
            if (code >= KTB_VM_ALL_OPS || (op.opcode & ~(0xff | KTB_VM_ROUND16)) || op.dst < 0 || op.dst >= KTB_VM_REGS || op.a < 0 ||
                op.a >= KTB_VM_REGS || op.b < 0 || op.b >= KTB_VM_REGS || op.c < 0 || op.c >= KTB_VM_REGS)
                return ktb_fail(ctx, KTB_E_ARG, "ew_multi", "bad program op");
            if (code == KTB_VM_CSEL && !(op.imm >= 0.f && op.imm < 8.f * 16))
                return ktb_fail(ctx, KTB_E_ARG, "ew_multi", "bad comparison");
            if (em_reads(op) & ~held) return ktb_fail(ctx, KTB_E_ARG, "ew_multi", "bad program op: it reads a register that holds nothing");
            held |= 1u << op.dst;
            // (a single op's result is stored from registers: nothing else can be asked for)
            if (p.n_ops == 1 && p.result_reg != op.dst) return ktb_fail(ctx, KTB_E_ARG, "ew_multi", "bad program header: not the op's result");
            if (p.n_ops > 1) {
                int top = op.dst > op.a ? op.dst : op.a;
                top = top > op.b ? top : op.b;
                top = top > op.c ? top : op.c;
                if (code == KTB_VM_CSEL && ((int)op.imm & 7) > top) top = (int)op.imm & 7;
                if (top + 1 > regs) regs = top + 1;
            }
        }
        if (!((held >> p.result_reg) & 1)) return ktb_fail(ctx, KTB_E_ARG, "ew_multi", "bad program header: a result that nothing wrote");
        if (p.n_ops > 1) {
            if (p.result_reg + 1 > regs) regs = p.result_reg + 1;
            if (a.n_in > regs) regs = a.n_in;
        }
    }
    for (int k = 0; k < a.n_in + a.n_out; ++k)
        if (a.dtype[k] != KTB_F16 && a.dtype[k] != KTB_F32)
            return ktb_fail(ctx, KTB_E_UNSUPPORTED, "ew_multi", "operand dtype must be f16 or f32");
    if (a.n_items <= 0 || a.rows <= 0 || a.cols <= 0) return KTB_OK;
    bool vec = a.vector_ok && a.cols % 8 == 0;
    for (int k = 0; k < a.n_in + a.n_out; ++k) vec = vec && (a.rows == 1 || a.row_stride[k] % 8 == 0);
    const uint32_t per_row = vec ? a.cols / 8 : (a.cols + 14) / 8;
    const uint64_t per_item = (uint64_t)per_row * a.rows;
    if (per_item >= (1ull << 31) || a.n_items >= (1ll << 32)) return ktb_fail(ctx, KTB_E_UNSUPPORTED, "ew_multi", "tile too large");
    const uint64_t total = per_item * (uint64_t)a.n_items;
    bool half = true;
    for (int k = 0; k < a.n_in; ++k) half = half && a.dtype[k] == KTB_F16;
    // as many chunks per thread as the kernel holds, fewer where that would leave less than four blocks for an SM
    int per_thread = !vec ? 1 : half && a.n_in <= 2 ? 4 : a.n_in == 1 || half ? 2 : 1;
    while (per_thread > 1 && total < 256ull * per_thread * 4 * ctx->sm_count) per_thread /= 2;
    const uint64_t blocks = (total + 256 * per_thread - 1) / (256 * per_thread);
    if (blocks >= (1ull << 31)) return ktb_fail(ctx, KTB_E_UNSUPPORTED, "ew_multi", "too many elements");
    const size_t smem = (size_t)regs * 8 * 256 * sizeof(float);
    if (vec) {
        auto k = a.n_in == 1   ? (half ? ktb_ew_multi_kernel<1, true> : ktb_ew_multi_kernel<1, false>)
                 : a.n_in == 2 ? (half ? ktb_ew_multi_kernel<2, true> : ktb_ew_multi_kernel<2, false>)
                               : (half ? ktb_ew_multi_kernel<4, true> : ktb_ew_multi_kernel<4, false>);
        if (smem > 48 * 1024) KTB_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<(unsigned)blocks, 256, smem, ctx->stream>>>(a, per_row, (uint32_t)per_item, total, per_thread);
    } else {
        auto k = a.n_in == 1 ? ktb_ew_multi_any_kernel<1> : a.n_in == 2 ? ktb_ew_multi_any_kernel<2> : ktb_ew_multi_any_kernel<4>;
        if (smem > 48 * 1024) KTB_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<(unsigned)blocks, 256, smem, ctx->stream>>>(a, per_row, (uint32_t)per_item, total);
    }
    KTB_CHECK_LAUNCH(ctx, "ktb_ew_multi_kernel");
    return KTB_OK;
}
