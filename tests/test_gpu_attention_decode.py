"""Attention of a few query rows over a longer context: the kernel that cuts the context into pieces, against the oracle
(the bars of the attention tests: P is rounded to f16 before P V, 2^-11 of each weight)."""
import ctypes as C

import numpy as np
import pytest

from ktir_cpu_b200 import KTIRInterpreter, kernels as K, runtime as R
from ktir_cpu_b200.interpreter import Session
from ktir_cpu_b200.lower_attn import decode_pieces
from ktir_cpu_b200.parser import KTIRParser
from oracle.numpy_interp import OracleInterpreter


def _case(tokens, before, heads, kv_heads, page, seed=0):
    rng = np.random.default_rng(seed)
    nb = -(-(before + tokens) // page)
    f = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)     # noqa: E731
    kw = dict(output_ptr=np.zeros((tokens, heads, 128), np.float16), query_ptr=f(tokens, heads, 128),
              key_cache_ptr=f(nb, page, kv_heads, 128), value_cache_ptr=f(nb, page, kv_heads, 128),
              block_tables_ptr=rng.permutation(nb).astype(np.int32).reshape(1, -1), cur_batch_start_index=0,
              block_table_offset=0, num_tiles=nb, context_len=before, scale=np.float32(1 / np.sqrt(128)))
    return K.paged_attention(tokens, before + tokens, heads, kv_heads, 128, page, tokens), kw


# (tokens, positions before, query heads, K/V heads, page): one piece; pieces that end inside a page; an odd number of
# 32-row pages; 16 rows, 17 (the second tile of rows), 32; head counts that are no power of two; one piece per head
# and several waves; a long context in whole clusters with the last merge
CASES = [(1, 0, 4, 4, 64), (1, 63, 2, 2, 64), (1, 64, 8, 1, 128), (3, 92, 4, 2, 32), (16, 130, 2, 2, 64), (17, 300, 1, 1, 128),
         (4, 1000, 16, 2, 32), (2, 700, 9, 3, 64), (1, 65, 160, 160, 64), (1, 6000, 8, 1, 128), (32, 200, 3, 3, 32)]


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,before,heads,kv_heads,page", CASES)
def test_decode_matches_the_oracle(tokens, before, heads, kv_heads, page, build_lib):
    src, kw = _case(tokens, before, heads, kv_heads, page)
    gpu = KTIRInterpreter()
    gpu.load(src)
    first = gpu.execute_function("paged_attention_kernel", **kw)["output_ptr"]
    again = gpu.execute_function("paged_attention_kernel", **kw)["output_ptr"]      # (the counters are back at zero)
    st, = [s for sess in gpu._sessions.values() for s in sess.plan.statements]
    assert st.kind == "attention_fwd" and st.args.splits >= 1 and st.args.dev_scratch
    gpu.close()
    ora = OracleInterpreter()
    ora.load(src)
    want = ora.execute_function("paged_attention_kernel", **kw)["output_ptr"]
    np.testing.assert_allclose(first.astype(np.float32), want.astype(np.float32), rtol=1e-2, atol=2e-3)
    np.testing.assert_array_equal(first, again)


@pytest.mark.gpu
def test_negative_page_is_reported(build_lib):
    src, kw = _case(1, 500, 4, 2, 64)
    kw["block_tables_ptr"][0, 3] = -7
    gpu = KTIRInterpreter()
    gpu.load(src)
    with pytest.raises(IndexError, match="-7 is negative"):
        gpu.execute_function("paged_attention_kernel", **kw)
    kw["block_tables_ptr"][0, 3] = 3
    gpu.execute_function("paged_attention_kernel", **kw)
    gpu.close()


@pytest.mark.parametrize("tokens,before,heads,kv_heads,splits", [(1, 8191, 64, 8, 16), (1, 60, 8, 8, 1), (4, 300, 32, 4, 4), (1, 5000, 2, 1, 76),
                                                                 (1, 4000, 160, 160, 1), (1, 9999, 74, 74, 2), (33, 4000, 1, 1, 0)])
def test_pieces_fill_clusters_and_no_more_than_the_context(tokens, before, heads, kv_heads, splits):
    nb = -(-(before + tokens) // 64)
    src = K.paged_attention(tokens, before + tokens, heads, kv_heads, 128, 64, tokens)
    f16 = np.dtype(np.float16)
    t = [("output_ptr", (tokens, heads, 128), f16), ("query_ptr", (tokens, heads, 128), f16), ("key_cache_ptr", (nb, 64, kv_heads, 128), f16),
         ("value_cache_ptr", (nb, 64, kv_heads, 128), f16), ("block_tables_ptr", (1, nb), np.dtype(np.int32))]
    s = Session(R.PlanOnlyDevice(), KTIRParser().parse_module(src).get_function("paged_attention_kernel"), t,
                dict(cur_batch_start_index=0, block_table_offset=0, num_tiles=nb, context_len=before, scale=np.float32(0.1)), arena_ptr=0)
    a = s.plan.statements[0].args
    assert a.splits == splits and kv_heads * max(a.splits, 1) <= max(148, kv_heads)
    assert a.splits < 4 or a.splits % 4 == 0


@pytest.mark.gpu
@pytest.mark.parametrize("kv_heads,group", [(17, 1), (18, 2), (32, 1), (8, 4)])
def test_whole_and_parts_share_the_scratch(kv_heads, group, build_lib):
    """Eight or more pieces (two clusters per head and slice, so the counters in scratch are used): launches over all
    heads, over parts of them and over all again, on one scratch, give the same bits, those of the oracle's bar."""
    src, kw = _case(1, 1200, kv_heads * group, kv_heads, 64)
    gpu = KTIRInterpreter()
    gpu.load(src)
    sess, _ = gpu.session("paged_attention_kernel", **kw)
    st, = sess.plan.statements
    if kv_heads in (17, 18):             # (the planner would take four)
        st._cut(gpu.device, 8, st.args.steps)
    parts = [c.launch for c in st.split(st.bytes_moved() // 4)]
    assert len(parts) == 4 and st.args.splits == (4 if kv_heads == 32 else 8 if kv_heads in (17, 18) else 16)
    for k, v in kw.items():
        if isinstance(v, np.ndarray):
            sess.upload(k, v)

    def output(whole):
        sess.upload("output_ptr", kw["output_ptr"])
        if whole:
            sess.run()
        for name, args in [] if whole else parts:
            args.arena = sess.arena
            gpu.device.check(getattr(gpu.device.lib, name)(gpu.device.h, C.byref(args)))
        out = sess.download("output_ptr")
        gpu.device.sync()
        return out.view(np.uint16)
    got = [output(whole) for whole in (True, False, True, True, False, True)]
    gpu.close()
    for other in got[1:]:
        np.testing.assert_array_equal(got[0], other)
    ora = OracleInterpreter()
    ora.load(src)
    want = ora.execute_function("paged_attention_kernel", **kw)["output_ptr"]
    np.testing.assert_allclose(got[0].view(np.float16).astype(np.float32), want.astype(np.float32), rtol=1e-2, atol=2e-3)


def test_counters_are_zero_before_planning_returns():
    """Tables are uploaded with a wait; the zeros of the merge counters too: the context may go to another stream between
    planning and the first run, and the memset is queued on the one of the planning."""
    calls = []

    class Device(R.PlanOnlyDevice):
        def memset(self, ptr, value, nbytes):
            calls.append(("memset", value, nbytes))

        def sync(self):
            calls.append(("sync",))
            return R.Status()
    src, kw = _case(1, 2000, 8, 4, 64)
    Session(Device(), KTIRParser().parse_module(src).get_function("paged_attention_kernel"),
            [(k, v.shape, v.dtype) for k, v in kw.items() if isinstance(v, np.ndarray)],
            {k: v for k, v in kw.items() if not isinstance(v, np.ndarray)}, arena_ptr=0)
    assert calls == [("memset", 0, 256), ("sync",)]


# (tokens, positions before, query heads, K/V heads, rows per tile, ranks): heads dealt out; tokens dealt out, the context of
# the first ones a step shorter; more rows in the whole than the pieces take, fewer on a rank
SHARDS = [(1, 2100, 64, 8, 1, 2), (1, 2100, 64, 8, 1, 8), (4, 62, 4, 1, 1, 4), (4, 1021, 4, 1, 1, 2), (40, 500, 1, 1, 8, 5), (2, 900, 6, 3, 1, 3)]


def _shard_case(tokens, before, heads, kv_heads, q):
    src, kw = _case(tokens, before, heads, kv_heads, 64)
    return K.paged_attention(tokens, before + tokens, heads, kv_heads, 128, 64, q), kw


@pytest.mark.parametrize("tokens,before,heads,kv_heads,q,world", SHARDS)
def test_a_rank_cuts_the_context_as_the_whole_grid(tokens, before, heads, kv_heads, q, world):
    src, kw = _shard_case(tokens, before, heads, kv_heads, q)
    func = KTIRParser().parse_module(src).get_function("paged_attention_kernel")

    class Device(R.PlanOnlyDevice):
        held = []

        def alloc(self, nbytes):
            self.held.append(nbytes)
            return nbytes

        def free(self, ptr):
            self.held.remove(ptr)

    def plan(shard, dev):
        s = Session(dev, func, [(k, v.shape, v.dtype) for k, v in kw.items() if isinstance(v, np.ndarray)],
                    {k: v for k, v in kw.items() if not isinstance(v, np.ndarray)}, arena_ptr=0, shard=shard)
        st, = s.plan.statements
        assert st.kind == "attention_fwd"
        return st.args
    whole = plan(None, R.PlanOnlyDevice())
    for rank in range(world):
        dev = Device()
        dev.held = []
        a = plan((rank, world), dev)
        assert a.heads * a.seq_q * world == heads * tokens and (a.splits, a.steps) == (whole.splits, whole.steps)
        n = a.heads // a.kv_group
        assert dev.held == ([(n * 32 + 255) // 256 * 256 + n * a.splits * a.seq_q * a.kv_group * 768] if a.splits else [])


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,before,heads,kv_heads,q,world", SHARDS)
def test_shards_give_the_bits_of_the_whole(tokens, before, heads, kv_heads, q, world, build_lib):
    from test_gpu_parity import _sharded_on_one_gpu
    src, kw = _shard_case(tokens, before, heads, kv_heads, q)
    gpu = KTIRInterpreter()
    gpu.load(src)
    full = gpu.execute_function("paged_attention_kernel", **kw)["output_ptr"]
    gpu.close()
    got, covered = _sharded_on_one_gpu(src, "paged_attention_kernel", kw, world, "output_ptr")
    np.testing.assert_array_equal(got.view(np.uint16), full.view(np.uint16))
    assert covered == full.nbytes


@pytest.mark.parametrize("steps,page,rows,heads,kv_heads,pieces", [
    # a second tile of rows, query heads in one wave (two with pages above 32): few steps stay with one CTA per query head
    (1, 64, 32, 32, 4, 0), (2, 32, 32, 32, 4, 0), (3, 32, 17, 4, 4, 0), (4, 32, 32, 32, 4, 4), (4, 64, 24, 32, 4, 0), (4, 64, 18, 8, 4, 4),
    (5, 64, 32, 32, 4, 4), (7, 64, 32, 128, 32, 0), (8, 64, 32, 128, 32, 4), (6, 128, 32, 128, 32, 0), (7, 128, 32, 128, 32, 4), (6, 32, 32, 128, 32, 4), (2, 64, 32, 256, 32, 0), (2, 32, 32, 256, 32, 1),
    (1, 64, 32, 256, 32, 1), (2, 64, 32, 1024, 128, 1), (4, 64, 32, 256, 32, 4),
    # less than four pieces per head
    (12, 64, 32, 36, 36, 0), (13, 64, 32, 36, 36, 2), (99, 64, 17, 75, 75, 0), (99, 64, 16, 75, 75, 1), (7, 32, 17, 75, 75, 0), (8, 32, 17, 75, 75, 1), (5, 32, 32, 36, 36, 0), (6, 32, 32, 36, 36, 2), (4, 64, 10, 36, 36, 0), (4, 32, 10, 36, 36, 2),
    (4, 64, 9, 36, 36, 2), (12, 64, 32, 288, 36, 2),
    # 10 to 16 rows: two or three steps in one piece
    (2, 32, 16, 4, 4, 1), (3, 128, 10, 4, 4, 1), (3, 64, 9, 4, 4, 2), (4, 64, 16, 4, 4, 4),
    # a second cluster per head from 12 steps on, for up to 16 rows at once; no more clusters than are resident
    (8, 64, 32, 32, 4, 4), (12, 64, 32, 32, 4, 12), (8, 64, 16, 16, 4, 8), (16, 64, 8, 144, 18, 4), (200, 64, 8, 136, 17, 4), (200, 64, 8, 128, 16, 8),
    (200, 64, 8, 32, 4, 32), (200, 64, 8, 264, 33, 4), (200, 64, 8, 272, 34, 2), (200, 64, 8, 592, 74, 2), (200, 64, 8, 600, 75, 1), (200, 64, 33, 33, 1, 0)])
def test_pieces_of_a_context(steps, page, rows, heads, kv_heads, pieces):
    assert decode_pieces(steps, page, rows, heads, kv_heads) == pieces


def _against_oracle(src, kw, one_plan=True):
    gpu = KTIRInterpreter()
    gpu.load(src)
    got = gpu.execute_function("paged_attention_kernel", **kw)["output_ptr"]
    st, = [s for sess in gpu._sessions.values() for s in sess.plan.statements]
    assert st.kind == "attention_fwd" and st.args.splits >= 1
    gpu.close()
    ora = OracleInterpreter()
    ora.load(src)
    with np.errstate(all="ignore"):
        want = ora.execute_function("paged_attention_kernel", **kw)["output_ptr"]
    np.testing.assert_allclose(got.astype(np.float32), want.astype(np.float32), rtol=1e-2, atol=2e-3)
    return st


# one piece, a cluster, several clusters with the merge through scratch
FORMS = [(1, 63, 4, 2, 64), (3, 509, 6, 3, 128), (8, 1016, 4, 1, 32), (32, 992, 1, 1, 64)]


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,before,heads,kv_heads,page", FORMS)
def test_decode_without_a_mask(tokens, before, heads, kv_heads, page, build_lib):
    """Every row sees every position."""
    src, kw = _case(tokens, before, heads, kv_heads, page)
    assert (tokens + before) % page == 0
    for use in ("ins(%masked :", "ins(%masked,"):
        assert src.count(use) == 1
        src = src.replace(use, use.replace("%masked", "%sc"))
    assert not _against_oracle(src, kw).args.causal


@pytest.mark.gpu
@pytest.mark.parametrize("m_init,l_init", [(0.5, 3.0), (-2.0, 0.0), (6.0, 1.0)])
@pytest.mark.parametrize("tokens,before,heads,kv_heads,page", FORMS)
def test_decode_with_initial_maximum_and_sum(tokens, before, heads, kv_heads, page, m_init, l_init, build_lib):
    """A running maximum and sum that start at finite values (a position without a value): once per row, however many pieces."""
    src, kw = _case(tokens, before, heads, kv_heads, page)
    for name, old, value in (("m_init", "ninf", m_init), ("l_init", "one", l_init)):
        assert src.count(f"%{name} = tensor.splat %{old} ") == 1
        src = src.replace(f"%{name} = tensor.splat %{old} ", f"%{name}_v = arith.constant {value} : f32\n    %{name} = tensor.splat %{name}_v ")
    a = _against_oracle(src, kw).args
    assert (a.m_init, a.l_init) == (m_init, l_init)


@pytest.mark.gpu
@pytest.mark.parametrize("which,value", [("key_cache_ptr", np.nan), ("key_cache_ptr", np.inf), ("value_cache_ptr", np.nan), ("value_cache_ptr", -np.inf)])
@pytest.mark.parametrize("tokens,before,heads,kv_heads,page", FORMS)
def test_decode_of_special_values(tokens, before, heads, kv_heads, page, which, value, build_lib):
    """One element of one visible position of K/V head 0: NaN reaches every row that sees it, an infinite score makes NaN
    (or vanishes, where it is negative), an infinite value stays."""
    src, kw = _case(tokens, before, heads, kv_heads, page)
    pos = before // 2
    kw[which] = kw[which].copy()
    kw[which][kw["block_tables_ptr"][0, pos // page], pos % page, 0, 5] = value
    _against_oracle(src, kw)
