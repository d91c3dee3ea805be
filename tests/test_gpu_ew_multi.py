"""Several elementwise stores in one launch (``ktb_launch_ew_multi``) against the step-by-step path, bit for bit, and
which stores join."""
import numpy as np
import pytest

from ktir_cpu_b200 import KTIRInterpreter, kernels as K, runtime as R
from ktir_cpu_b200.interpreter import Session
from ktir_cpu_b200.parser import KTIRParser


def _run(src, kw, fused):
    it = KTIRInterpreter(fused_kernels=fused)
    it.load(src)
    got = it.execute_function("elementwise_kernel", **kw)
    kinds = [(s.kind, getattr(s, "symbol", "")) for sess in it._sessions.values() for s in sess.plan.statements]
    it.close()
    return got, kinds


def _args(ops, n, dtype, pred, seed=0):
    dt = np.float16 if dtype == "f16" else np.float32
    rng = np.random.default_rng(seed)
    x, y = (rng.standard_normal(n) * 3).astype(dt), rng.standard_normal(n).astype(dt)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -1.0], dt)     # every pair of them, and tiny values
    m = min(n, 49)
    x[:m], y[:m] = np.repeat(special, 7)[:m], np.tile(special, 7)[:m]
    x[m:m + 8] = np.finfo(dt).tiny / 4
    names = [f"out_{o}_ptr" for o in ops] + (["out_select_ptr"] if pred else []) + (["out_ext_add_ptr"] if dtype == "f16" else [])
    return dict(x_ptr=x, y_ptr=y, **{k: np.full(n, 7, dt) for k in names})


ALL = list(K.ELEMENTWISE_OPS)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f16", "f32"])
@pytest.mark.parametrize("n,block,cores", [(64 * 8, 64, 4), (8192 * 3, 8192, 3), (333 * 8, 333, 4), (8, 1, 8)])
def test_every_op_gives_the_bits_of_the_step_by_step_path(n, block, cores, dtype, build_lib):
    """All ops of the suite (19 and select: three launches), whole chunks and blocks that start anywhere.  The device
    functions are the same ones, so sin or exp agree to the bit too."""
    src = K.elementwise_suite(ALL, n, block, cores, dtype, "olt")
    kw = _args(ALL, n, dtype, "olt")
    got, kinds = _run(src, kw, True)
    assert set(kinds) == {("ew_stream", "ktb_launch_ew_multi")} and len(kinds) == 3
    want, _ = _run(src, kw, False)
    for k in want:
        np.testing.assert_array_equal(got[k].view(np.uint8), want[k].view(np.uint8), err_msg=k)


@pytest.mark.gpu
@pytest.mark.parametrize("pred", sorted(R.CMP))
def test_select_on_every_comparison(pred, build_lib):
    src = K.elementwise_suite(["mul"], 1024, 128, 4, "f16", pred)
    kw = _args(["mul"], 1024, "f16", pred)
    got, kinds = _run(src, kw, True)
    assert len(kinds) == 1
    want, _ = _run(src, kw, False)
    for k in want:
        np.testing.assert_array_equal(got[k].view(np.uint16), want[k].view(np.uint16), err_msg=k)


@pytest.mark.gpu
def test_programs_of_several_ops(build_lib):
    """A chain with constants and more live values than inputs: shared registers instead of direct ones."""
    src = K.elementwise_suite(["add", "div"], 4000, 1000, 4, "f16", "oge").replace(
        "%r_div = arith.divf %x, %y", "%q0 = arith.mulf %x, %x : tensor<1000xf16>\n      %q1 = math.exp %y : tensor<1000xf16>\n"
        "      %q2 = arith.subf %q0, %q1 : tensor<1000xf16>\n      %q3 = math.erf %q2 : tensor<1000xf16>\n      %r_div = arith.divf %q3, %q1")
    kw = _args(["add", "div"], 4000, "f16", "oge")
    got, kinds = _run(src, kw, True)
    assert kinds == [("ew_stream", "ktb_launch_ew_multi")]
    want, _ = _run(src, kw, False)
    for k in want:
        np.testing.assert_array_equal(got[k].view(np.uint16), want[k].view(np.uint16), err_msg=k)


def _plan(src, fn, tensors, arena=None):
    return Session(R.PlanOnlyDevice(), KTIRParser().parse_module(src).get_function(fn), tensors, {}, arena_ptr=0).plan.statements


def test_which_stores_join():
    f16 = np.dtype(np.float16)
    t = [(k, (4096,), f16) for k in ("x_ptr", "y_ptr", "out_add_ptr", "out_mul_ptr", "out_ext_add_ptr")]
    src = K.elementwise_suite(["add", "mul"], 4096, 128, 4, "f16")
    st, = _plan(src, "elementwise_kernel", t)
    assert (st.args.n_in, st.args.n_out) == (2, 3) and st.table.shape == (32, 5)
    assert [p.n_ops for p in list(st.args.program)[:3]] == [1, 1, 1]              # the final rounding joined the f32 add
    # a store into a tile that the others read goes last (they need what it overwrites) and stays a launch of its own
    src2 = src.replace("%out_add_view = ktdp.construct_memory_view %out_add_ptr", "%out_add_view = ktdp.construct_memory_view %y_ptr")
    kinds = [(s.kind, s.args.n_out if hasattr(s.args, "n_out") else 1) for s in _plan(src2, "elementwise_kernel", t)]
    assert kinds == [("ew_stream", 2), ("ew_stream", 1)]
    # one op keeps the kernel compiled for it
    one, = _plan(K.elementwise_suite(["add"], 4096, 128, 4, "f32"), "elementwise_kernel",
                 [(k, (4096,), np.dtype(np.float32)) for k in ("x_ptr", "y_ptr", "out_add_ptr")])
    assert one.symbol == "ktb_launch_ew_stream"


def _chain(n, block, dtype, ops):
    """x (op) y (op) y ..., one store."""
    src, prev, text = K.vector_add(n, block, 4, dtype), "%x", ""
    for i, op in enumerate(ops):
        text += f"%q{i} = math.{op} {prev}" if op in ("exp", "sqrt") else f"%q{i} = arith.{op} {prev}, %y"
        text, prev = text + f" : tensor<{block}x{dtype}>\n    ", f"%q{i}"
    at = src.index("%output = arith.addf")
    return src[:at] + text.rstrip() + src[src.index("\n", at):].replace("ktdp.store %output,", f"ktdp.store {prev},")


# (elements, block, dtype, ops) and whether the kernel for several stores takes it
ROUTES = [(8192, 128, "f32", ["mulf", "addf"], False), (8192, 128, "f32", ["minnumf"], False), (8192, 128, "f32", ["exp"], True),
          (8192, 128, "f16", ["mulf", "addf"], True), (8192, 128, "f16", ["mulf"], False), (333 * 12, 333, "f16", ["mulf", "exp", "divf"], False),
          (333 * 12, 333, "f32", ["mulf", "sqrt"], False), (333 * 12, 333, "f32", ["exp"], True), (1025 * 128, 1025, "f16", ["mulf", "addf"], True)]


@pytest.mark.parametrize("n,block,dtype,ops,multi", ROUTES)
def test_which_kernel_takes_one_store(n, block, dtype, ops, multi):
    t = [(k, (n,), np.dtype(np.float16 if dtype == "f16" else np.float32)) for k in ("x_ptr", "y_ptr", "output_ptr")]
    func = KTIRParser().parse_module(_chain(n, block, dtype, ops)).get_function("add_kernel")
    st, = Session(R.PlanOnlyDevice(), func, t, dict(BLOCK_SIZE=block), arena_ptr=0).plan.statements
    assert st.kind == "ew_stream" and st.symbol == ("ktb_launch_ew_multi" if multi else "ktb_launch_ew_stream")


@pytest.mark.gpu
@pytest.mark.parametrize("n,block,dtype,ops,multi", ROUTES)
def test_one_store_gives_the_bits_of_the_step_by_step_path(n, block, dtype, ops, multi, build_lib):
    a = _args([], n, dtype, None)
    kw = dict(x_ptr=a["x_ptr"], y_ptr=a["y_ptr"], output_ptr=np.full_like(a["x_ptr"], 7), BLOCK_SIZE=block)
    got = []
    for fused in (True, False):
        it = KTIRInterpreter(fused_kernels=fused)
        it.load(_chain(n, block, dtype, ops))
        got.append(it.execute_function("add_kernel", **kw)["output_ptr"].view(np.uint8))
        it.close()
    np.testing.assert_array_equal(got[0], got[1])
