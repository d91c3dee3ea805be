"""Row kernels for rows of any length and alignment (``ktb_launch_row_softmax_any``) against the oracle."""
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
