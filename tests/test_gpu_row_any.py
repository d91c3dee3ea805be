"""Row kernels for rows of any length and alignment (``ktb_launch_row_softmax_any``, ``ktb_launch_row_program_any``) against
the oracle."""
import re

import numpy as np
import pytest

from ktir_cpu_b200 import KTIRInterpreter, kernels as K
from oracle.numpy_interp import OracleInterpreter

pytestmark = pytest.mark.gpu


def _both(src, fn, kw):
    gpu = KTIRInterpreter()
    gpu.load(src)
    got = gpu.execute_function(fn, **kw)
    stmts = [s for sess in gpu._sessions.values() for s in sess.plan.statements]
    kinds, symbols = [s.kind for s in stmts], [getattr(s, "symbol", "") for s in stmts]
    gpu.close()
    ora = OracleInterpreter()
    ora.load(src)
    return got, ora.execute_function(fn, **kw), kinds, symbols


# one warp per row (up to 1024) with 1, 2 and 4 vectors per thread, 64 threads, one CTA per row, few rows (more
# threads each); whole vectors and single elements; the edges of each
SOFTMAX = [(64, 1, 4, 2), (96, 3, 4, 4), (32, 24, 4, 1), (64, 250, 4, 4), (640, 264, 4, 4), (640, 511, 4, 4), (1280, 1000, 5, 4),
           (1280, 1023, 5, 4), (640, 1025, 4, 2), (640, 2040, 4, 2), (640, 2049, 4, 2), (1200, 3000, 4, 2), (37, 5001, 37, 1),
           (8, 16376, 4, 1), (320, 16377, 32, 1)]


@pytest.mark.parametrize("f32", [True, False])
@pytest.mark.parametrize("rows,cols,cores,step", SOFTMAX)
def test_softmax_rows_of_any_length(rows, cols, cores, step, f32, build_lib):
    """f16 results: half a step of rounding (2^-11) from the f32 value in both, plus the device's exp — 2e-3; with
    f16 arithmetic exp, the sum and the quotient each round, as the power-of-two test has it."""
    x = (np.random.default_rng(cols).standard_normal((rows, cols)) * 3).astype(np.float16)
    x[0] = 0
    if cols > 2:
        x[1, cols - 1] = 60000          # the last element takes everything
        x[2, 1:] = -np.inf
    got, want, kinds, symbols = _both(K.softmax_rows(rows, cols, cores, step, f32), "softmax_kernel",
                                      dict(output_ptr=np.full_like(x, 9), input_ptr=x))
    assert kinds == ["row_softmax"] and symbols == ["ktb_launch_row_softmax_any"]
    np.testing.assert_allclose(got["output_ptr"].astype(np.float32), want["output_ptr"].astype(np.float32),
                               rtol=2e-3 if f32 else 1e-2, atol=2e-6 if f32 else 1e-5)
    np.testing.assert_array_equal(got["input_ptr"].view(np.uint16), x.view(np.uint16))


@pytest.mark.parametrize("stride", [67, 72, 130])
def test_softmax_rows_that_start_anywhere(stride, build_lib):
    """Power-of-two rows inside a wider tensor: a row stride that is no multiple of 8 elements goes to the kernel for
    any alignment, and the columns between the rows keep what they held."""
    rows, cols = 64, 64
    src = K.softmax_rows(rows, cols, 4, 4, True).replace(f"strides: [{cols}, 1]", f"strides: [{stride}, 1]")
    x = np.random.default_rng(1).standard_normal((rows, stride)).astype(np.float16)
    got, want, kinds, symbols = _both(src, "softmax_kernel", dict(output_ptr=np.full_like(x, 9), input_ptr=x))
    assert kinds == ["row_softmax"] and symbols == ["ktb_launch_row_softmax" + ("" if stride == 72 else "_any")]
    np.testing.assert_allclose(got["output_ptr"].astype(np.float32), want["output_ptr"].astype(np.float32), rtol=2e-3, atol=2e-6)
    np.testing.assert_array_equal(got["output_ptr"][:, cols:], 9)


def _bits(got, want, names):
    for k in names:
        u = np.uint16 if want[k].dtype == np.float16 else np.uint32
        np.testing.assert_array_equal(got[k].view(u), want[k].view(u), err_msg=k)


# a row per warp, several warps, one CTA; one to four fold rounds; odd lengths (every row starts elsewhere), even, whole vectors
NORM = [(24, 71, 4, 2), (24, 257, 4, 1), (64, 300, 4, 4), (40, 1000, 5, 8), (36, 1290, 3, 4), (24, 2049, 3, 1), (12, 5120, 3, 2),
        (6, 9999, 3, 1), (4, 16383, 2, 1), (600, 264, 4, 2), (4, 512, 2, 1)]


@pytest.mark.parametrize("rows,cols,cores,step", NORM)
def test_rmsnorm_rows_of_any_length(rows, cols, cores, step, build_lib):
    """The sum in the reference's fold order, every op rounded where the reference rounds: its bits."""
    rng = np.random.default_rng(cols)
    kw = dict(x_ptr=(rng.standard_normal((rows, cols)) * 2).astype(np.float16), w_ptr=rng.standard_normal(cols).astype(np.float16),
              y_ptr=np.full((rows, cols), 9, np.float16), rstd_ptr=np.zeros(rows, np.float32))
    got, want, kinds, symbols = _both(K.rmsnorm_rows(rows, cols, cores, step, weight=True), "rmsnorm_kernel", kw)
    assert kinds == ["row_program"] and symbols == ["ktb_launch_row_program" + ("" if cols == 512 else "_any")]
    _bits(got, want, ("y_ptr", "rstd_ptr"))


# (many rows of whole vectors: a product and a sum rounded together show in a few rows of a hundred)
@pytest.mark.parametrize("rows,cols,cores", [(24, 257, 4), (40, 1000, 5), (24, 2049, 3), (96, 5120, 3), (96, 1024, 3), (4, 16383, 2)])
def test_layernorm_rows_of_any_length(rows, cols, cores, build_lib):
    rng = np.random.default_rng(cols)
    kw = dict(x_ptr=(rng.standard_normal((rows, cols)) * 3 + 1).astype(np.float16), w_ptr=rng.standard_normal(cols).astype(np.float16),
              b_ptr=rng.standard_normal(cols).astype(np.float16), y_ptr=np.zeros((rows, cols), np.float16), mean_ptr=np.zeros(rows, np.float32))
    got, want, kinds, _ = _both(K.layernorm_rows(rows, cols, cores), "layernorm_kernel", kw)
    assert kinds == ["row_program"]
    _bits(got, want, ("y_ptr", "mean_ptr"))


@pytest.mark.parametrize("rows,block,blocks,cores", [(11, 53, 7, 3), (37, 1024, 3, 32), (9, 361, 6, 4), (12, 256, 5, 5), (5, 1500, 8, 2),
                                                     (6, 448, 1, 3), (3, 2048, 8, 2)])
def test_column_blocked_layernorm_of_any_length(rows, block, blocks, cores, build_lib):
    """f16 throughout: every add of the block accumulation and of the fold rounds, in the reference's order.  (One
    block too: the loop of one trip is a chain of one term, and Mean and Rstd leave with the launch.)"""
    rng = np.random.default_rng(block)
    rc = (rows, block * blocks)
    kw = dict(X=rng.standard_normal(rc).astype(np.float16), Y=np.zeros(rc, np.float16), W=rng.standard_normal(rc).astype(np.float16),
              B=rng.standard_normal(rc).astype(np.float16), Mean=np.zeros(rows, np.float16), Rstd=np.zeros(rows, np.float16), N=rc[1],
              eps=np.float16(1e-5), BLOCK_SIZE=block)
    got, want, kinds, _ = _both(K.layernorm_blocked(*rc, block, cores), "_layer_norm_fwd_fused", kw)
    assert set(kinds) == {"row_program"}
    _bits(got, want, ("Mean", "Rstd", "Y"))


@pytest.mark.parametrize("rows,cols,cores,step", [(24, 333, 4, 2), (12, 4000, 3, 1), (6, 16382, 3, 1)])
def test_log_softmax_rows_of_any_length(rows, cols, cores, step, build_lib):
    """Phases that are no normalisation: the interpreting kernel.  exp and log are the device's (f16 tolerance)."""
    x = (np.random.default_rng(cols).standard_normal((rows, cols)) * 3).astype(np.float16)
    got, want, kinds, symbols = _both(K.log_softmax_rows(rows, cols, cores, step), "log_softmax_kernel",
                                      dict(x_ptr=x, y_ptr=np.zeros_like(x)))
    assert kinds == ["row_program"] and symbols == ["ktb_launch_row_program_any"]
    np.testing.assert_allclose(got["y_ptr"].astype(np.float32), want["y_ptr"].astype(np.float32), rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("rows,block", [(13, 512), (512, 1024), (513, 1024), (7, 8)])
def test_two_column_blocks(rows, block, build_lib):
    """Two short blocks stay on the kernel that holds the row in registers; both sides of its line."""
    rng = np.random.default_rng(rows)
    rc = (rows, 2 * block)
    kw = dict(X=rng.standard_normal(rc).astype(np.float16), Y=np.zeros(rc, np.float16), W=rng.standard_normal(rc).astype(np.float16),
              B=rng.standard_normal(rc).astype(np.float16), Mean=np.zeros(rows, np.float16), Rstd=np.zeros(rows, np.float16), N=rc[1],
              eps=np.float16(1e-5), BLOCK_SIZE=block)
    got, want, kinds, _ = _both(K.layernorm_blocked(*rc, block, 4), "_layer_norm_fwd_fused", kw)
    assert kinds == ["row_program"]
    _bits(got, want, ("Mean", "Rstd", "Y"))


@pytest.mark.parametrize("rows", [1536, 1540])
def test_many_short_rows(rows, build_lib):
    rng = np.random.default_rng(rows)
    kw = dict(x_ptr=rng.standard_normal((rows, 512)).astype(np.float16), y_ptr=np.zeros((rows, 512), np.float16), rstd_ptr=np.zeros(rows, np.float32))
    got, want, kinds, _ = _both(K.rmsnorm_rows(rows, 512, 4, 1), "rmsnorm_kernel", kw)
    assert kinds == ["row_program"]
    _bits(got, want, ("y_ptr", "rstd_ptr"))


def _initial(src, max_init, sum_init):
    """The softmax kernel with other initial values of its two reductions."""
    for name, old, value in (("max_init", "ninf", max_init), ("sum_init", "zero", sum_init)):
        assert src.count(f"%{name} = tensor.splat %{old} : ") == 1
        src = src.replace(f"%{name} = tensor.splat %{old} : ", f"%{name}_v = arith.constant {value} : f32\n      %{name} = tensor.splat %{name}_v : ")
    return src


@pytest.mark.parametrize("cols", [250, 3000])
@pytest.mark.parametrize("max_init,sum_init,low,high", [("0.0", "0.0", -96, -89), ("0.0", "0.0", -3, 3), ("-65504.0", "0.0", -3, 3), ("-3.0e38", "0.0", -3, 3),
                                                        ("-3.0e38", "1.0", 59000, 60000), ("-3.0e38", "0.5", -3, 3)])
def test_softmax_with_initial_values(cols, max_init, sum_init, low, high, build_lib):
    """A maximum that starts above every element leaves weights, and a sum, below the normal numbers of f32 (spaced 2^-149:
    2^-10 of the smallest sum here, 250 e^-96); a sum that starts at one is not scaled with the rest.  As f16, 2^-11."""
    x = np.random.default_rng(cols).uniform(low, high, (8, cols)).astype(np.float16)
    src = _initial(K.softmax_rows(8, cols, 4, 2, True), max_init, sum_init)
    got, want, kinds, symbols = _both(src, "softmax_kernel", dict(output_ptr=np.zeros_like(x), input_ptr=x))
    assert kinds == ["row_softmax"] and symbols == ["ktb_launch_row_softmax_any"]
    np.testing.assert_allclose(got["output_ptr"].astype(np.float32), want["output_ptr"].astype(np.float32), rtol=2e-3, atol=2e-6)


def _f32(src):
    """The kernel over f32 tiles: no casts between the two types."""
    src = src.replace("f16", "f32")
    for name, of in re.findall(r"^ *(%\w+) = arith\.(?:extf|truncf) (%\w+) :.*\n", src, re.M):
        src = re.sub(rf"^ *{name} = arith\.(?:extf|truncf) {of} :.*\n", "", src, flags=re.M)
        src = re.sub(rf"{name}\b", of, src)
    return src


def _special_rows(rows, cols, dt):
    """NaN at one place and everywhere, infinities of either sign at one place and everywhere, the lowest value everywhere
    and in all places but one."""
    x = (np.random.default_rng(cols).standard_normal((rows, cols)) * 2).astype(dt)
    x[0, cols // 2], x[1] = np.nan, np.nan
    x[2, 0], x[3], x[4, 1:], x[5, cols - 1], x[6] = -np.inf, -np.inf, -np.inf, np.inf, np.inf
    x[7], x[8, 1:] = np.finfo(dt).min, np.finfo(dt).min
    x[9, 0], x[9, 1] = np.nan, np.inf
    return x


@pytest.mark.parametrize("maxop", ["maximumf", "maxnumf"])
@pytest.mark.parametrize("form", ["f16 rows, f32 statistics", "f16 arithmetic", "f32 rows"])
@pytest.mark.parametrize("cols", [5, 250, 3001])
def test_softmax_of_special_values(cols, form, maxop, build_lib):
    """f16 results: 2e-3 and 1e-2 as above.  f32 results: the sum in another order (cols 2^-24 at most) and two steps of the
    device's and of NumPy's exp (2^-21)."""
    x = _special_rows(12, cols, np.float32 if form == "f32 rows" else np.float16)
    src = K.softmax_rows(12, cols, 4, 1, form != "f16 arithmetic").replace("arith.maximumf", "arith." + maxop)
    if form == "f32 rows":
        src = _f32(src)
    with np.errstate(all="ignore"):
        got, want, kinds, symbols = _both(src, "softmax_kernel", dict(output_ptr=np.full_like(x, 9), input_ptr=x))
    assert kinds == ["row_softmax"] and symbols == ["ktb_launch_row_softmax_any"]
    rtol, atol = {"f32 rows": (2.0 ** -21 + cols * 2.0 ** -24, 0), "f16 arithmetic": (1e-2, 1e-5)}.get(form, (2e-3, 2e-6))
    np.testing.assert_allclose(got["output_ptr"].astype(np.float32), want["output_ptr"].astype(np.float32), rtol=rtol, atol=atol)


@pytest.mark.parametrize("form", ["f16 rows, f32 statistics", "f16 arithmetic", "f32 rows"])
@pytest.mark.parametrize("rows,cols", [(64, 250), (40, 2049), (8, 9001)])
def test_softmax_in_place(rows, cols, form, build_lib):
    x = np.random.default_rng(cols).standard_normal((rows, cols)).astype(np.float32 if form == "f32 rows" else np.float16)
    src = K.softmax_rows(rows, cols, 4, 2, form != "f16 arithmetic").replace("construct_memory_view %output_ptr", "construct_memory_view %input_ptr")
    if form == "f32 rows":
        src = _f32(src)
    got, want, kinds, symbols = _both(src, "softmax_kernel", dict(output_ptr=np.full_like(x, 9), input_ptr=x))
    assert kinds == ["row_softmax"] and symbols == ["ktb_launch_row_softmax_any"]
    rtol, atol = {"f32 rows": (2.0 ** -21 + cols * 2.0 ** -24, 0), "f16 arithmetic": (1e-2, 1e-5)}.get(form, (2e-3, 2e-6))
    np.testing.assert_allclose(got["input_ptr"].astype(np.float32), want["input_ptr"].astype(np.float32), rtol=rtol, atol=atol)
    np.testing.assert_array_equal(got["output_ptr"], 9)


# odd lengths, whole vectors, whole eighths (the wide first fold), one warp and several
F32_ROWS = [(24, 261), (12, 1000), (20, 1024), (6, 5001), (3, 9984)]


@pytest.mark.parametrize("rows,cols", F32_ROWS)
def test_normalisations_of_f32_tiles(rows, cols, build_lib):
    """The same kernel over f32 rows: plain row norm, layer norm and column blocks, the oracle's bits."""
    rng = np.random.default_rng(cols)
    f = lambda *s: rng.standard_normal(s, dtype=np.float32)     # noqa: E731
    x, w, b = f(rows, cols), f(cols), f(cols)
    cores = next(c for c in (4, 3, 2) if rows % c == 0)
    got, want, kinds, symbols = _both(_f32(K.rmsnorm_rows(rows, cols, cores, 1, weight=True)), "rmsnorm_kernel",
                                      dict(x_ptr=x, w_ptr=w, y_ptr=np.zeros_like(x), rstd_ptr=np.zeros(rows, np.float32)))
    assert kinds == ["row_program"]
    _bits(got, want, ("y_ptr", "rstd_ptr"))
    got, want, kinds, symbols = _both(_f32(K.layernorm_rows(rows, cols, cores)), "layernorm_kernel",
                                      dict(x_ptr=x, w_ptr=w, b_ptr=b, y_ptr=np.zeros_like(x), mean_ptr=np.zeros(rows, np.float32)))
    assert kinds == ["row_program"]
    _bits(got, want, ("y_ptr", "mean_ptr"))
    rc = (rows, 3 * (cols // 3))
    kw = dict(X=f(*rc), Y=np.zeros(rc, np.float32), W=f(*rc), B=f(*rc), Mean=np.zeros(rows, np.float32), Rstd=np.zeros(rows, np.float32), N=rc[1],
              eps=np.float32(1e-5), BLOCK_SIZE=cols // 3)
    got, want, kinds, symbols = _both(_f32(K.layernorm_blocked(*rc, cols // 3, cores)), "_layer_norm_fwd_fused", kw)
    assert kinds == ["row_program"]
    _bits(got, want, ("Mean", "Rstd", "Y"))
