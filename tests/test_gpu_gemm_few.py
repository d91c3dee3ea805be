"""Products with few tiles: 128 x 64 / 128 x 128 tiles, K in ranges that a cluster adds up."""
import re

import numpy as np
import pytest

from ktir_cpu_b200 import KTIRInterpreter, kernels as K, runtime as R
from ktir_cpu_b200.interpreter import Session
from ktir_cpu_b200.lower_mm import few_tiles
from ktir_cpu_b200.parser import KTIRParser


def _run(M, N, Kd, bm, bn, bk, f32, plan=None):
    rng = np.random.default_rng(M + N + Kd)
    a, b = (rng.uniform(-1, 1, s).astype(np.float16) for s in ((M, Kd), (Kd, N)))
    cores = next(c for c in (8, 4, 3, 2, 1) if (M // bm) * (N // bn) % c == 0)
    it = KTIRInterpreter()
    it.load(K.tiled_matmul(M, N, Kd, bm, bn, bk, cores, f32))
    kw = dict(a_ptr=a, b_ptr=b, c_ptr=np.full((M, N), 9, np.float16))
    sess, _ = it.session("matmul_kernel", **kw)
    args = sess.plan.statements[0].args
    if plan is not None:
        args.tile_n, args.split_k = plan
    got = it.execute_function("matmul_kernel", **kw)["c_ptr"]
    it.close()
    return got, a.astype(np.float64) @ b.astype(np.float64), (args.tile_n, args.split_k)


# (M, N, K, bm, bn, bk): rows that do not fill a tile or its last one, N that ends inside a tile of 64 and of 128, K that
# ends inside a step of 64 and ranges of unequal length, one step for four ranges, a single tile
SHAPES = [(16, 64, 512, 16, 64, 64), (8, 32, 64, 8, 32, 64), (24, 96, 200, 24, 32, 40), (64, 160, 1032, 32, 32, 8), (144, 96, 320, 16, 32, 64),
          (128, 256, 256, 64, 64, 64), (272, 352, 712, 16, 32, 8), (300, 128, 4096, 20, 64, 64)]


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,Kd,bm,bn,bk", SHAPES)
def test_every_tile_and_split_gives_the_product(M, N, Kd, bm, bn, bk, build_lib):
    """f32 sums of K products of magnitude below 1 (error K 2^-24 at most) and one rounding to f16 (2^-11)."""
    base = None
    for plan in [(t, s) for t in (64, 128) for s in (1, 2, 4) if -(-Kd // 64) >= s] + [(0, 0)]:
        got, want, _ = _run(M, N, Kd, bm, bn, bk, True, plan)
        np.testing.assert_allclose(got.astype(np.float64), want, rtol=2.0 ** -11, atol=Kd * 2.0 ** -24 + 2.0 ** -12, err_msg=str(plan))
        if plan[1] in (0, 1):        # K in one range: the same sums whatever the tile
            base = got if base is None else base
            np.testing.assert_array_equal(got, base, err_msg=str(plan))


@pytest.mark.gpu
def test_f16_accumulator_form_takes_it_too(build_lib):
    got, want, plan = _run(64, 512, 2880, 64, 64, 64, False)
    assert plan == (64, 4)
    np.testing.assert_allclose(got.astype(np.float64), want, rtol=2e-2, atol=2e-1)


def test_rule():
    assert few_tiles(4096, 4096, 4096) == (0, 0) and few_tiles(2048, 2048, 512) == (0, 0)
    assert few_tiles(64, 5760, 2880) == (64, 1) and few_tiles(64, 4096, 4096) == (64, 2) and few_tiles(16, 512, 4096) == (64, 4)
    assert few_tiles(1536, 1536, 2048) == (128, 1) and few_tiles(256, 256, 256) == (64, 1)
    assert few_tiles(848, 1408, 352) == (0, 0) and few_tiles(848, 1408, 2048) == (128, 1)
    for M in (1, 100, 128, 1000, 2304):
        for N in (32, 512, 4096):
            for Kd in (8, 64, 1000, 8192):
                t, s = few_tiles(M, N, Kd)
                assert (t, s) == (0, 0) or (t in (64, 128) and s in (1, 2, 4) and (s == 1 or -(-Kd // 64) >= 4 * s))


def test_a_ranks_part_adds_up_like_the_whole():
    """Cores of one rank cover fewer rows, but K is cut as for the whole product."""
    src = K.tiled_matmul(256, 512, 4096, 64, 64, 64, 8, True)
    f16 = np.dtype(np.float16)
    t = [("a_ptr", (256, 4096), f16), ("b_ptr", (4096, 512), f16), ("c_ptr", (256, 512), f16)]
    func = KTIRParser().parse_module(src).get_function("matmul_kernel")
    whole = Session(R.PlanOnlyDevice(), func, t, {}, arena_ptr=0).plan.statements[0].args
    for rank in range(4):
        part = Session(R.PlanOnlyDevice(), func, t, {}, arena_ptr=0, shard=(rank, 4)).plan.statements[0].args
        assert part.M == 64 and (part.tile_n, part.split_k) == (whole.tile_n, whole.split_k)
    assert whole.split_k == 4


ADD_THEN_MUL = """
    %q_c = ktdp.get_compute_tile_id : index
    %q_blk = arith.constant 128 : index
    %q_c3 = arith.constant 3 : index
    %q_c4 = arith.constant 4 : index
    %q_half = arith.constant 512 : index
    %q_off = arith.muli %q_c, %q_blk : index
    %q_c7 = arith.addi %q_c, %q_c3 : index
    %q_far = arith.divui %q_c7, %q_c4 : index
    %q_skip = arith.muli %q_far, %q_half : index
    %q_from = arith.addi %q_off, %q_skip : index
""" + "".join(f"""    %q_{n}v = ktdp.construct_memory_view %{n}_ptr, sizes: [1024], strides: [1] {{
      coordinate_set = affine_set<(d0) : (d0 >= 0, -d0 + 1023 >= 0)>, memory_space = #ktdp.memory_space<global>
    }} : memref<1024xf16>
""" for n in "xoz") + "".join(f"""    %q_{n}t = ktdp.construct_access_tile %q_{v}v[%q_{off}] {{
      access_tile_set = affine_set<(d0) : (d0 >= 0, -d0 + 127 >= 0)>, access_tile_order = affine_map<(d0) -> (d0)>
    }} : memref<1024xf16> -> !ktdp.access_tile<128xindex>
""" for n, v, off in (("x", "x", "off"), ("o", "o", "off"), ("r", "o", "from"), ("z", "z", "off"))) + """
    %q_x = ktdp.load %q_xt : !ktdp.access_tile<128xindex> -> tensor<128xf16>
    %q_s = arith.addf %q_x, %q_x : tensor<128xf16>
    ktdp.store %q_s, %q_ot : tensor<128xf16>, !ktdp.access_tile<128xindex>
    %q_r = ktdp.load %q_rt : !ktdp.access_tile<128xindex> -> tensor<128xf16>
    %q_m = arith.mulf %q_r, %q_x : tensor<128xf16>
    ktdp.store %q_m, %q_zt : tensor<128xf16>, !ktdp.access_tile<128xindex>
"""


def test_statements_of_a_rank_follow_those_of_the_same_store():
    """Core 0 multiplies what it has just added up, the others old values: the two stores are two launches in the whole
    grid and one on the ranks without core 0.  The products behind them keep the ranges of K of their own counterparts."""
    def body(src, name):
        text = src[src.index("\n", src.index("func.func")) + 1:src.index("    return")]
        return re.sub(r"%(\w+)", lambda m: f"%{name}_{m.group(1)}", text)
    src = ('module {\n  func.func @k(%x_ptr: index, %o_ptr: index, %z_ptr: index, %m_a_ptr: index, %m_b_ptr: index, %m_c_ptr: index, '
           '%n_a_ptr: index, %n_b_ptr: index, %n_c_ptr: index) attributes {grid = [4, 1]} {' + ADD_THEN_MUL +
           body(K.tiled_matmul(256, 64, 4096, 64, 64, 64, 4, True), "m") + body(K.tiled_matmul(256, 64, 128, 64, 64, 64, 4, True), "n") +
           "    return\n  }\n}\n")
    f16 = np.dtype(np.float16)
    t = [(k, (1024,), f16) for k in ("x_ptr", "o_ptr", "z_ptr")]
    t += [(f"{n}_{k}_ptr", s, f16) for n, kd in (("m", 4096), ("n", 128)) for k, s in (("a", (256, kd)), ("b", (kd, 64)), ("c", (256, 64)))]
    func = KTIRParser().parse_module(src).get_function("k")
    kinds = lambda s: [x.kind for x in s.plan.statements]                                             # noqa: E731
    cuts = lambda s: [(x.args.K, x.args.split_k) for x in s.plan.statements if x.kind == "gemm_f16"]  # noqa: E731
    whole = Session(R.PlanOnlyDevice(), func, t, {}, arena_ptr=0)
    assert kinds(whole) == ["ew_stream", "ew_stream", "gemm_f16", "gemm_f16"] and cuts(whole) == [(4096, 4), (128, 0)]
    for rank in range(4):
        part = Session(R.PlanOnlyDevice(), func, t, {}, arena_ptr=0, shard=(rank, 4))
        assert kinds(part) == kinds(whole)[0 if rank == 0 else 1:] and cuts(part) == cuts(whole)


@pytest.mark.parametrize("shape,plan", [
    # the one-CTA kernel on 128 rows takes them up to 14 steps, and many tiles up to K = 2048 ...
    ((1024, 192, 384), (0, 0)), ((608, 128, 832), (0, 0)), ((640, 1024, 256), (0, 0)), ((65, 512, 896), (0, 0)), ((896, 2048, 1024), (0, 0)),
    # ... not beyond, nor up to 64 rows, nor where pairs would run
    ((608, 128, 897), (64, 2)), ((64, 512, 448), (64, 1)), ((256, 512, 192), (64, 1)), ((896, 2048, 2048), (128, 1)), ((1152, 1408, 1024), (128, 1)),
    # 33 clusters of four are resident at once; two ranges from nine steps on
    ((384, 704, 1280), (64, 4)), ((384, 768, 1280), (64, 2)), ((1152, 256, 4096), (64, 2)), ((64, 128, 512), (64, 1)), ((64, 128, 576), (64, 2))])
def test_products_that_the_other_kernels_are_faster_for(shape, plan):
    assert few_tiles(*shape) == plan
