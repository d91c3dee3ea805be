"""The measured work of this backend: KTIR kernels run through the interpreter's public entry points.

A program of this framework either calls ``execute_function`` with host arrays (parse once, call often), or plans a
function once with ``session`` and runs it with ``Session.run`` on tensors that stay in device memory.  The cases
``call_*`` are the first form; all others the second, on arenas whose tensors are filled on the GPU.
"""
import math

import numpy as np
import torch

from ktir_cpu_b200 import KTIRInterpreter, kernels

F16, F32, I32 = np.dtype(np.float16), np.dtype(np.float32), np.dtype(np.int32)
TORCH = {F16: torch.float16, F32: torch.float32, I32: torch.int32}
EPS = 1e-6


def listed():
    return [
        # the smallest call: the reference's vector-add example, host arrays in and out; launch and call latency
        dict(name="call_add_4096", kind="call_add", n=4096, block=128, cores=32),
        # the headline kernel end to end: 64 MiB up, 64 MiB down over the host link
        dict(name="call_softmax", kind="call_softmax", rows=8192, cols=4096, cores=32, step=8, f32=True),
        # the tile operations of an activation, one output tensor each (the elementwise suite of the tests)
        dict(name="elementwise_f16", kind="elementwise", ops="add mul exp tanh erf", n=1 << 22, block=4096, cores=32,
             dtype="f16"),
        # attention scores / logits of a model: the headline kernel
        dict(name="softmax_8192x4096", kind="softmax", rows=8192, cols=4096, cores=32, step=8, f32=True),
        # scores of a width that is no power of two (a context of 3000 positions, nothing padded)
        dict(name="softmax_3000", kind="softmax", rows=4096, cols=3000, cores=32, step=4, f32=True),
        # layer norm as the reference's example writes it: f16 throughout, a row in eight column blocks
        dict(name="layernorm_blocked", kind="layernorm", rows=4096, block=1024, blocks=8, cores=32),
        # the norm of a decoder layer over a prefill batch: f32 statistics, weight row, 1/rms stored
        dict(name="rmsnorm_2048x5120", kind="rmsnorm", rows=2048, cols=5120, cores=32, step=4),
        # embedding-gradient style update: gather rows, scale, accumulate into rows in core order
        dict(name="gather_scatter", kind="scatter", table=65536, cols=128, entries=262144, tile=64, cores=64),
        # a square product at the size where the tensor cores bound it
        dict(name="matmul_4096", kind="matmul", m=64, n=64, k=64, bm=64, bn=64, bk=64, cores=32, f32=True),
        # one projection of a decode batch of 64 rows: reading B bounds it; f16 accumulator form of the reference
        dict(name="matmul_decode", kind="matmul", m=1, n=90, k=45, bm=64, bn=64, bk=64, cores=30, f32=False),
        # prefill: causal attention, a batch of 8 with 32 heads folded into the heads
        dict(name="attention_prefill", kind="attention", tokens=2048, before=0, heads=256, kv_heads=256, page=128, q=128),
        # decode: one new token after a long context, grouped heads, pages in any order
        dict(name="attention_decode", kind="attention", tokens=1, before=8191, heads=64, kv_heads=8, page=64, q=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call_add", "call_softmax", "elementwise", "softmax", "softmax", "layernorm", "rmsnorm",
                       "scatter", "matmul", "matmul", "attention", "attention"])
    cores = rng.choice([4, 8, 30, 32, 48])
    if kind == "call_add":
        block = _log(rng, 16, 4096)
        return dict(kind=kind, n=block * cores * _log(rng, 1, 32), block=block, cores=cores)
    if kind in ("softmax", "call_softmax"):
        cols = _log(rng, 64, 16384)
        if rng.random() < 0.35:
            cols = 1 << int(round(math.log2(cols)))
        step = rng.choice([1, 2, 4]) if cols <= 4096 else 1
        rows = cores * step * _log(rng, 1, max(1, (1 << 24) // (cols * cores * step)))
        return dict(kind=kind, rows=rows, cols=cols, cores=cores, step=step, f32=rng.random() < 0.7)
    if kind == "elementwise":
        ops = rng.sample(["add", "sub", "mul", "div", "maximum", "minnum", "neg", "abs", "sqrt", "exp", "log", "tanh",
                          "rsqrt", "erf"], rng.randint(1, 5))
        block = _log(rng, 64, 8192)
        n = block * cores * _log(rng, 1, max(1, (1 << 23) // (block * cores)))
        return dict(kind=kind, ops=" ".join(ops), n=n, block=block, cores=cores, dtype=rng.choice(["f16", "f16", "f32"]))
    if kind == "layernorm":
        block = rng.choice([64, 128, 256, 512, 1024]) if rng.random() < 0.7 else _log(rng, 48, 1500)
        blocks = rng.randint(1, 8)
        return dict(kind=kind, rows=_log(rng, 32, max(64, (1 << 24) // (block * blocks))), block=block, blocks=blocks,
                    cores=rng.choice([8, 30, 32]))
    if kind == "rmsnorm":
        cols = 128 * _log(rng, 1, 64) if rng.random() < 0.6 else _log(rng, 64, 8192)
        step = rng.choice([1, 2, 4])
        return dict(kind=kind, rows=cores * step * _log(rng, 1, max(1, (1 << 24) // (cols * cores * step))), cols=cols,
                    cores=cores, step=step)
    if kind == "scatter":
        tile = rng.choice([16, 32, 64])
        return dict(kind=kind, table=_log(rng, 64, 65536), cols=rng.choice([64, 128, 128, 256]),
                    entries=tile * 32 * _log(rng, 1, 64), tile=tile, cores=rng.choice([8, 16, 32]))
    if kind == "matmul":
        bm, bn, bk = rng.choice([16, 32, 64, 64]), rng.choice([32, 64, 64]), rng.choice([32, 64, 64])
        m, n, k = (max(1, _log(rng, lo, 4096) // b) for lo, b in ((16, bm), (128, bn), (64, bk)))
        cores = next(c for c in (32, 30, 24, 16, 12, 9, 8, 7, 6, 5, 4, 3, 2, 1) if m * n % c == 0)
        return dict(kind=kind, m=m, n=n, k=k, bm=bm, bn=bn, bk=bk, cores=cores, f32=rng.random() < 0.6)
    page, group, kv = rng.choice([32, 64, 128]), rng.choice([1, 4, 8]), rng.choice([4, 8, 32])
    if rng.random() < 0.5:          # decode, or a few tokens at a time
        q = rng.choice([1, 1, 2, 4])
        return dict(kind="attention", tokens=q, before=_log(rng, 64, 16384), heads=kv * group, kv_heads=kv, page=page, q=q)
    q = 128 // group
    before = rng.choice([0, 0, _log(rng, 64, 2048)])
    return dict(kind="attention", tokens=q * _log(rng, 1, 2048 // q), before=before, heads=kv * group, kv_heads=kv,
                page=page, q=q)


# ---- a case as KTIR text, function name, tensors (name -> shape, dtype), scalars, names of what it writes --------
def _pages(c):
    return -(-(c["before"] + c["tokens"]) // c["page"])


def _kernel(c):
    kind = c["kind"].replace("call_", "")
    if kind == "add":
        t = {k: ((c["n"],), F16) for k in ("x_ptr", "y_ptr", "output_ptr")}
        return (kernels.vector_add(c["n"], c["block"], c["cores"]), "add_kernel", t, dict(BLOCK_SIZE=c["block"]),
                ["output_ptr"])
    if kind == "softmax":
        t = {k: ((c["rows"], c["cols"]), F16) for k in ("output_ptr", "input_ptr")}
        return (kernels.softmax_rows(c["rows"], c["cols"], c["cores"], c["step"], c["f32"]), "softmax_kernel", t, {},
                ["output_ptr"])
    if kind == "elementwise":
        dt = F16 if c["dtype"] == "f16" else F32
        outs = [f"out_{o}_ptr" for o in c["ops"].split()] + ["out_select_ptr"]
        outs += ["out_ext_add_ptr"] if dt == F16 else []
        t = {k: ((c["n"],), dt) for k in ["x_ptr", "y_ptr"] + outs}
        return (kernels.elementwise_suite(c["ops"].split(), c["n"], c["block"], c["cores"], c["dtype"], "olt"),
                "elementwise_kernel", t, {}, outs)
    if kind == "layernorm":
        rows, cols = c["rows"], c["block"] * c["blocks"]
        t = {k: ((rows, cols), F16) for k in ("X", "Y", "W", "B")}
        t.update(Mean=((rows,), F16), Rstd=((rows,), F16))
        return (kernels.layernorm_blocked(rows, cols, c["block"], c["cores"]), "_layer_norm_fwd_fused", t,
                dict(N=cols, eps=np.float16(1e-5), BLOCK_SIZE=c["block"]), ["Y", "Mean", "Rstd"])
    if kind == "rmsnorm":
        s = (c["rows"], c["cols"])
        t = dict(x_ptr=(s, F16), w_ptr=(s[1:], F16), y_ptr=(s, F16), rstd_ptr=(s[:1], F32))
        return (kernels.rmsnorm_rows(s[0], s[1], c["cores"], c["step"], EPS, weight=True), "rmsnorm_kernel", t, {},
                ["y_ptr", "rstd_ptr"])
    if kind == "scatter":
        t = dict(table_ptr=((c["table"], c["cols"]), F16), idx_ptr=((c["entries"],), I32),
                 out_ptr=((c["table"], c["cols"]), F16))
        return (kernels.gather_scale_scatter(c["table"], c["cols"], c["entries"], c["tile"], c["cores"]),
                "gather_scale_scatter", t, {}, ["out_ptr"])
    if kind == "matmul":
        M, N, K = c["m"] * c["bm"], c["n"] * c["bn"], c["k"] * c["bk"]
        t = dict(a_ptr=((M, K), F16), b_ptr=((K, N), F16), c_ptr=((M, N), F16))
        return (kernels.tiled_matmul(M, N, K, c["bm"], c["bn"], c["bk"], c["cores"], c["f32"]), "matmul_kernel", t, {},
                ["c_ptr"])
    T, total, nb, D = c["tokens"], c["before"] + c["tokens"], _pages(c), 128
    cache = ((nb, c["page"], c["kv_heads"], D), F16)
    t = dict(output_ptr=((T, c["heads"], D), F16), query_ptr=((T, c["heads"], D), F16), key_cache_ptr=cache,
             value_cache_ptr=cache, block_tables_ptr=((1, nb), I32))
    return (kernels.paged_attention(T, total, c["heads"], c["kv_heads"], D, c["page"], c["q"]), "paged_attention_kernel",
            t, dict(cur_batch_start_index=0, block_table_offset=0, num_tiles=nb, context_len=c["before"],
                    scale=np.float32(1.0 / math.sqrt(D))), ["output_ptr"])


def _inputs(c, seed):
    """name -> device tensor for every tensor the kernel reads, from the seed alone."""
    _, _, tensors, _, _ = _kernel(c)
    gen = torch.Generator("cuda").manual_seed(seed)

    def normal(name, scale=1.0):
        shape, dt = tensors[name]
        return (torch.randn(shape, generator=gen, device="cuda") * scale).to(TORCH[dt])

    kind = c["kind"].replace("call_", "")
    if kind == "add":
        return dict(x_ptr=normal("x_ptr"), y_ptr=normal("y_ptr"))
    if kind == "softmax":
        return dict(input_ptr=normal("input_ptr", 2.0))
    if kind == "elementwise":         # positive where a root or a logarithm is taken, away from a zero divisor
        x, y = normal("x_ptr"), normal("y_ptr")
        if any(o in ("sqrt", "rsqrt", "log", "log2") for o in c["ops"].split()):
            x = x.abs() + 0.01
        return dict(x_ptr=x, y_ptr=torch.where(y.abs() < 0.01, torch.full_like(y, 0.01), y))
    if kind == "layernorm":
        return dict(X=normal("X"), W=normal("W", 0.1) + 1, B=normal("B", 0.1))
    if kind == "rmsnorm":
        return dict(x_ptr=normal("x_ptr"), w_ptr=normal("w_ptr", 0.1) + 1)
    if kind == "scatter":
        idx = torch.randint(0, c["table"], (c["entries"],), generator=gen, device="cuda", dtype=torch.int32)
        return dict(table_ptr=normal("table_ptr"), idx_ptr=idx, out_ptr=torch.zeros_like(normal("out_ptr")))
    if kind == "matmul":
        return {k: (torch.rand(tensors[k][0], generator=gen, device="cuda") * 2 - 1).half() for k in ("a_ptr", "b_ptr")}
    table = torch.randperm(_pages(c), generator=gen, device="cuda").int().reshape(1, -1)
    return dict(query_ptr=normal("query_ptr"), key_cache_ptr=normal("key_cache_ptr"),
                value_cache_ptr=normal("value_cache_ptr"), block_tables_ptr=table)


class _DeviceTensor:
    """Lets torch see a session's tensor, which lies in the backend's own device memory.  Holds the interpreter: it
    frees its sessions' memory when it goes, and an output may outlive the state that it came from."""

    def __init__(self, interp, session, name, shape, dtype):
        self.interp = interp
        self.__cuda_array_interface__ = dict(shape=shape, typestr=dtype.str, data=(session.device_ptr(name), False), version=3)


def prepare(case, seed):
    source, func, tensors, scalars, outs = _kernel(case)
    interp = KTIRInterpreter()
    interp.load(source)
    data = _inputs(case, seed)
    if case["kind"].startswith("call_"):
        arrays = {k: data[k].cpu().numpy() if k in data else np.zeros(*v) for k, v in tensors.items()}
        return dict(interp=interp, func=func, kwargs={**arrays, **scalars}, outs=outs)
    shapes = {k: np.empty(*v) for k, v in tensors.items()}           # never touched: a session is planned from shapes
    session, _ = interp.session(func, **shapes, **scalars)
    views = {k: torch.as_tensor(_DeviceTensor(interp, session, k, *v), device="cuda") for k, v in tensors.items()}
    for k, v in views.items():
        if k in data:
            v.copy_(data[k])
        else:
            v.zero_()
    torch.cuda.synchronize()
    return dict(interp=interp, session=session, outputs={k: views[k] for k in outs})


def run(state):
    if "session" in state:
        state["session"].run()
        return state["outputs"]
    result = state["interp"].execute_function(state["func"], **state["kwargs"])
    return {k: result[k] for k in state["outs"]}


def _visible(c):
    """Pairs of a query position and a key position that it sees, in one head."""
    return c["tokens"] * c["before"] + c["tokens"] * (c["tokens"] + 1) // 2


def work(case):
    _, _, tensors, _, outs = _kernel(case)
    size = {k: int(np.prod(s)) * d.itemsize for k, (s, d) in tensors.items()}
    total = sum(size.values())
    kind = case["kind"].replace("call_", "")
    if kind == "scatter":        # every entry reads an index and a table row, reads and writes a destination row
        return dict(bytes=case["entries"] * (4 + 3 * 2 * case["cols"]), flops=2 * case["entries"] * case["cols"])
    if kind == "matmul":
        return dict(bytes=total, flops=2 * case["m"] * case["bm"] * case["n"] * case["bn"] * case["k"] * case["bk"])
    if kind == "attention":
        return dict(bytes=total, flops=4 * case["heads"] * 128 * _visible(case))
    elements = int(np.prod(next(iter(tensors.values()))[0]))
    return dict(bytes=total, flops=elements * {"add": 1, "elementwise": len(outs), "softmax": 5, "layernorm": 8, "rmsnorm": 4}[kind])


def tolerance(case):
    """Adds, products, gathers and ordered updates round at stated points and come back to the bit.  Elsewhere two
    correct implementations differ in the order of f32 sums and in the last place of exp, which now and then
    moves an f16 result by one step (2^-11 of the value): 3e-4 at most in the 2-norm.  The blocked layer norm
    rounds its sums themselves to f16, and attention rounds its weights; both carry that through."""
    kind = case["kind"].replace("call_", "")
    if kind in ("add", "scatter"):
        return "exact"
    if kind == "elementwise":
        return {"rel": 1e-3, "max": 1e-2} if case["dtype"] == "f16" else {"rel": 4e-6, "max": 1e-4}
    return {"rel": {"softmax": 1.5e-3, "layernorm": 4e-3, "rmsnorm": 1e-3, "matmul": 1e-3, "attention": 2e-3}[kind],
            "max": 0.05}


def exact(case, seed):
    data = {k: v if v.dtype == torch.int32 else v.double() for k, v in _inputs(case, seed).items()}
    kind = case["kind"].replace("call_", "")
    if kind == "add":
        return dict(output_ptr=data["x_ptr"] + data["y_ptr"])
    if kind == "softmax":
        return dict(output_ptr=torch.softmax(data["input_ptr"], 1))
    if kind == "elementwise":
        x, y = data["x_ptr"], data["y_ptr"]
        fn = dict(add=x.add, sub=x.sub, mul=x.mul, div=x.div, maximum=x.maximum, minnum=x.fmin)
        outs = {}
        for o in case["ops"].split():
            outs[f"out_{o}_ptr"] = fn[o](y) if o in fn else getattr(torch, o)(x)
        if "out_erf_ptr" in outs:
            outs["out_erf_ptr"] = None        # the specified polynomial, not the function, is what comes back
        outs["out_select_ptr"] = torch.where(x < y, x, y)
        if case["dtype"] == "f16":
            outs["out_ext_add_ptr"] = x + y
        return outs
    if kind == "layernorm":
        x, eps = data["X"], float(np.float16(1e-5))
        mean, var = x.mean(1), x.var(1, unbiased=False)
        rstd = 1 / torch.sqrt(var + eps)
        return dict(Y=(x - mean[:, None]) * rstd[:, None] * data["W"] + data["B"], Mean=None, Rstd=rstd)
    if kind == "rmsnorm":
        x = data["x_ptr"]
        rstd = 1 / torch.sqrt((x * x).mean(1) + EPS)
        return dict(y_ptr=x * rstd[:, None] * data["w_ptr"], rstd_ptr=rstd)
    if kind == "scatter":
        # entries of one tile that name the same row all write the same value: a row moves once per tile
        idx = data["idx_ptr"].long()
        tile = torch.arange(idx.numel(), device="cuda") // case["tile"]
        rows = torch.unique(tile * case["table"] + idx) % case["table"]
        count = torch.bincount(rows, minlength=case["table"]).double()
        return dict(out_ptr=data["out_ptr"] + 0.5 * data["table_ptr"] * count[:, None])
    if kind == "matmul":
        return dict(c_ptr=data["a_ptr"] @ data["b_ptr"])
    group, T = case["heads"] // case["kv_heads"], case["tokens"]
    table = data["block_tables_ptr"][0].long()
    out = torch.empty((T, case["heads"], 128), dtype=torch.float64, device="cuda")
    mask = torch.arange(len(table) * case["page"], device="cuda") > case["before"] + torch.arange(T, device="cuda")[:, None]
    for h in range(case["heads"]):
        k, v = (data[n][table, :, h // group].reshape(-1, 128) for n in ("key_cache_ptr", "value_cache_ptr"))
        s = (data["query_ptr"][:, h] @ k.T) / math.sqrt(128)
        out[:, h] = torch.softmax(s.masked_fill(mask, -math.inf), 1) @ v
    return dict(output_ptr=out)
