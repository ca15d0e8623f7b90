"""GPU: the chunk backward over ragged chunks, with one item per CTA and with many (buffers, barriers and tensor memory reused): sequences of 1, 15, 16, 17,
33, 63, 64, 65 and 100 tokens have the same gradients, bit for bit, alone and in every copy of a batch of thirty of each.  Forward-only calls, which do
not keep A, have the outputs of the others."""
import pytest
import torch

import mogankda_b200 as mk
from mogankda_b200.index import get_layout
from oracle import kda_oracle as orc
from tests.common import compare, make_inputs, run

pytestmark = pytest.mark.gpu
LENS, TIMES = (1, 15, 16, 17, 33, 63, 64, 65, 100), 30


@pytest.mark.parametrize("scalar", [False, True])
@pytest.mark.parametrize("dtype,l2", [(torch.bfloat16, True), (torch.float16, False), (torch.float32, True)])
def test_ragged_chunks_have_the_same_gradients_everywhere(dtype, l2, scalar):
    T = sum(LENS)
    cu = [0, *torch.tensor(LENS).cumsum(0).tolist()]
    lv, do, dht, opts, epi = make_inputs(T=T, HK=2, HV=4, cu=tuple(cu), dtype=dtype, gate="precomputed" if scalar else "kimi", scalar=scalar, l2=l2, epi=None, seed=53)
    one = run(mk.chunk_delta_rule, lv, do, dht, opts, epi)
    compare(one, run(orc.chunked_delta_rule, lv, do, dht, opts, epi, f64=True))
    tokens = lambda t: t.dim() >= 3 and t.shape[1] == T                                  # noqa: E731
    rep = lambda t: torch.cat([t] * TIMES, 1 if tokens(t) else 0)                         # noqa: E731
    many_lv = {k: rep(t) if tokens(t) or k == "h0" else t for k, t in lv.items()}
    many_cu = torch.tensor([0] + [cu[i + 1] + T * r for r in range(TIMES) for i in range(len(LENS))], dtype=torch.int32, device="cuda")
    many_opts = dict(opts, cu_seqlens=many_cu)
    many = run(mk.chunk_delta_rule, many_lv, rep(do), rep(dht), many_opts, epi)
    for k in ("o", "dq", "dk", "dv", "dg", "dbeta"):
        assert torch.equal(many[k], torch.cat([one[k]] * TIMES, 1)), k
    for k in ("ht", "dh0"):
        assert torch.equal(many[k], torch.cat([one[k]] * TIMES, 0)), k
    lone = run(mk.chunk_delta_rule, {k: t for k, t in many_lv.items() if k != "h0"}, rep(do), rep(dht), many_opts, epi)
    with torch.no_grad():
        forward = run(mk.chunk_delta_rule, {k: t for k, t in many_lv.items() if k != "h0"}, rep(do), rep(dht), many_opts, epi, grads=False)
    assert torch.equal(forward["o"], lone["o"]) and torch.equal(forward["ht"], lone["ht"])


@pytest.mark.parametrize("scalar", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_rows_past_the_end_are_zero_whatever_the_others_hold(dtype, scalar):
    """dq_v, dk_v and dgp leave as tiles of 64 rows, and a caller may add up whole tiles: rows past the end of a chunk are zero also where q, k or the states
    are not finite.  One, some and no rows missing, in the first, a middle and the last block of 16, two v-heads per q/k head."""
    from mogankda_b200 import ops
    lens, HK, HV = (1, 15, 16, 31, 40, 63, 64), 2, 4
    T, cu = sum(lens), [0, *torch.tensor(lens).cumsum(0).tolist()]
    lv, do, _, opts, _ = make_inputs(T=T, HK=HK, HV=HV, cu=tuple(cu), dtype=dtype, gate="precomputed", scalar=scalar, epi=None, h0=False, seed=61)
    lay = get_layout(1, T, opts["cu_seqlens"], lv["q"].device, 32)
    g_c, be = ops.gate_cumsum_fwd(lay, lv["g"], "precomputed", None, None, -5.0, HV, beta_raw=lv["beta"], beta_sigmoid=True, beta_scale=2.0)
    rq, rk = ops.l2norm_rstd(lv["q"]), ops.l2norm_rstd(lv["k"])
    A, Aqk, nw, u, kbar, qs, gl = ops.intra_fwd(lay, lv["q"], lv["k"], lv["v"], rq, rk, g_c, be, 128 ** -0.5, HK, HV, scalar_gate=scalar)
    h, Vd, _, _ = ops.recur_fwd(lay, nw, u, kbar, gl, HK, HV)
    dh, dVd, dO, _ = ops.bwd_dh(lay, do, kbar, qs, gl, Aqk, nw, HK, HV)
    last = torch.tensor(cu[1:], device="cuda") - 1

    def at_last(t, x):
        t = t.clone()
        t[0, last, :, 5] = x
        return t

    def tile(t, x):          # one value of the high half of every state
        t = t.clone()
        t.view(torch.bfloat16).reshape(lay.NC, HV, -1)[..., 7] = x
        return t

    for x in (float("inf"), float("nan")):
        for q, k, S, dS in ((lv["q"], at_last(lv["k"], x), h, dh), (at_last(lv["q"], x), lv["k"], h, dh), (lv["q"], lv["k"], tile(h, x), dh),
                            (lv["q"], lv["k"], h, tile(dh, x))):
            for t in ops.bwd_chunk(lay, q, k, lv["v"], rq, rk, g_c, be, A, S, dS, Vd, dO, dVd, 128 ** -0.5, HK, HV, lv["beta"], True, 2.0, scalar_gate=scalar)[:3]:
                for c, n in enumerate(lay.chunk_len.tolist()):
                    assert (t[c, :, n:] == 0).all(), (x, c, n)


@pytest.mark.parametrize("scalar", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_finished_dq_and_dk(dtype, scalar, monkeypatch):
    """mkda_bwd_chunk_rows leaves the bits of mkda_bwd_chunk and mkda_qk_grad_finish (no L2 norm, one v-head per q/k head), and nothing outside the chunks."""
    import ctypes
    from mogankda_b200 import _lib, ops
    lens, H = (1, 15, 16, 17, 33, 63, 64, 65), 3
    T, cu = sum(lens), [0, *torch.tensor(lens).cumsum(0).tolist()]
    lv, do, _, opts, _ = make_inputs(T=T, HK=H, HV=H, cu=tuple(cu), dtype=dtype, gate="precomputed", scalar=scalar, l2=False, epi=None, h0=False, seed=67)
    lay = get_layout(1, T, opts["cu_seqlens"], lv["q"].device, 32)
    g_c, be = ops.gate_cumsum_fwd(lay, lv["g"], "precomputed", None, None, -5.0, H, beta_raw=lv["beta"], beta_sigmoid=True, beta_scale=2.0)
    A, Aqk, nw, u, kbar, qs, gl = ops.intra_fwd(lay, lv["q"], lv["k"], lv["v"], None, None, g_c, be, 128 ** -0.5, H, H, scalar_gate=scalar)
    h, Vd, _, _ = ops.recur_fwd(lay, nw, u, kbar, gl, H, H)
    dh, dVd, dO, _ = ops.bwd_dh(lay, do, kbar, qs, gl, Aqk, nw, H, H)
    args = (lay, lv["q"], lv["k"], lv["v"], None, None, g_c, be, A, h, dh, Vd, dO, dVd, 128 ** -0.5, H, H, lv["beta"], True, 2.0)
    want = ops.bwd_chunk(*args, scalar_gate=scalar)
    rows = ops.qk_grad_finish(lay, want[0], want[1], lv["q"], lv["k"], None, None, H, H)
    # a row more in front and behind: outside every chunk
    got = [torch.full((T + 2, H, 128), 7.0, dtype=dtype, device="cuda") for _ in range(2)]
    monkeypatch.setattr(_lib, "call", lambda name, p, *a: _lib.load().mkda_bwd_chunk_rows(ctypes.byref(p), None, *(ctypes.c_void_p(t[1:].data_ptr()) for t in got), ctypes.c_void_p(a[0])))
    out = ops.bwd_chunk(*args, scalar_gate=scalar)
    monkeypatch.undo()
    for t, w in zip(got, rows):
        assert torch.equal(t[1:-1], w.view(T, H, 128)) and (t[[0, -1]] == 7).all()
    for a, b in zip(out[2:], want[2:]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("finish", [False, True])
@pytest.mark.parametrize("times", [1, 12])
@pytest.mark.parametrize("lens", [(1, 15, 64, 65, 63, 128), (64, 128, 192)])
@pytest.mark.parametrize("scalar", [False, True])
def test_rows_of_dO(scalar, lens, times, finish, monkeypatch):
    """mkda_bwd_dh_rows and mkda_bwd_chunk_rows on bf16 rows give the bits of the tiles, chains shared between two CTAs or not, one and many items per CTA; full
    chunks have no tile, and of the others' the low halves are not looked at."""
    import ctypes
    from mogankda_b200 import _lib, ops
    lens, HK, HV = lens * times, 2, 2 if finish else 4
    T, cu = sum(lens), [0, *torch.tensor(lens).cumsum(0).tolist()]
    lv, do, dht, opts, _ = make_inputs(T=T, HK=HK, HV=HV, cu=tuple(cu), dtype=torch.bfloat16, gate="precomputed", scalar=scalar, l2=False, epi=None, h0=False, seed=71)
    lay = get_layout(1, T, opts["cu_seqlens"], lv["q"].device, 32)
    g_c, be = ops.gate_cumsum_fwd(lay, lv["g"], "precomputed", None, None, -5.0, HV, beta_raw=lv["beta"], beta_sigmoid=True, beta_scale=2.0)
    A, Aqk, nw, u, kbar, qs, gl = ops.intra_fwd(lay, lv["q"], lv["k"], lv["v"], None, None, g_c, be, 128 ** -0.5, HK, HV, scalar_gate=scalar)
    h, Vd, _, _ = ops.recur_fwd(lay, nw, u, kbar, gl, HK, HV)
    do = do.to(torch.bfloat16).contiguous()

    def both():
        dh, dVd, dO, dh0 = ops.bwd_dh(lay, do, kbar, qs, gl, Aqk, nw, HK, HV, want_dh0=True)
        if rows:
            t = dO.view(torch.bfloat16).reshape(lay.NC, HV, 2, -1)
            t[:, :, 1] = float("nan")
            t[lay.chunk_len == 64] = float("nan")
        out = ops.bwd_chunk(lay, lv["q"], lv["k"], lv["v"], None, None, g_c, be, A, h, dh, Vd, dO, dVd, 128 ** -0.5, HK, HV, lv["beta"], True, 2.0, scalar_gate=scalar)
        return dh, dVd, dh0, *out

    rows = False
    want = both()
    fin = ops.qk_grad_finish(lay, want[3], want[4], lv["q"], lv["k"], None, None, HK, HV)
    rows, got_q, got_k = True, torch.empty_like(lv["q"]), torch.empty_like(lv["k"])

    def call(name, p, *args):
        lib, stream = _lib.load(), args[-1]
        if name == "mkda_bwd_dh_ordered":
            assert lib.mkda_bwd_dh_rows(ctypes.byref(p), *args) == 0
        else:
            dq, dk = (got_q.data_ptr(), got_k.data_ptr()) if finish else (None, None)
            assert lib.mkda_bwd_chunk_rows(ctypes.byref(p), do.data_ptr(), dq, dk, stream) == 0
    monkeypatch.setattr(_lib, "call", call)
    got = both()
    monkeypatch.undo()
    for i, (a, b) in enumerate(zip(got, want)):
        if not (finish and i in (3, 4)):
            assert torch.equal(a.view(torch.int32) if a.dtype == torch.float32 else a, b.view(torch.int32) if b.dtype == torch.float32 else b), i
    if finish:
        assert torch.equal(got_q.view(-1), fin[0].view(-1)) and torch.equal(got_k.view(-1), fin[1].view(-1))


@pytest.mark.parametrize("times", [1, 12])
@pytest.mark.parametrize("lens", [(1, 15, 64, 65, 63, 128), (64, 128, 192)])
@pytest.mark.parametrize("scalar", [False, True])
def test_rows_of_dO_with_v_heads_spread_and_without_tiles(scalar, lens, times, monkeypatch):
    """The bits of the tiles also with a dq and dk tile per v-head, and where no chunk is ragged without any tiles of dO."""
    import ctypes
    from mogankda_b200 import _lib, ops
    full, lens, HK, HV = all(n % 64 == 0 for n in lens), lens * times, 2, 4
    T, cu = sum(lens), [0, *torch.tensor(lens).cumsum(0).tolist()]
    lv, do, _, opts, _ = make_inputs(T=T, HK=HK, HV=HV, cu=tuple(cu), dtype=torch.bfloat16, gate="precomputed", scalar=scalar, l2=False, epi=None, h0=False, seed=73)
    lay = get_layout(1, T, opts["cu_seqlens"], lv["q"].device, 32)
    g_c, be = ops.gate_cumsum_fwd(lay, lv["g"], "precomputed", None, None, -5.0, HV, beta_raw=lv["beta"], beta_sigmoid=True, beta_scale=2.0)
    A, Aqk, nw, u, kbar, qs, gl = ops.intra_fwd(lay, lv["q"], lv["k"], lv["v"], None, None, g_c, be, 128 ** -0.5, HK, HV, scalar_gate=scalar)
    h, Vd, _, _ = ops.recur_fwd(lay, nw, u, kbar, gl, HK, HV)
    do = do.to(torch.bfloat16).contiguous()
    lib, both = _lib.load(), []

    def call(name, p, *args):
        if name == "mkda_bwd_chunk":
            p.per_v_head, p.dq_v, p.dk_v = 1, dq.data_ptr(), dk.data_ptr()
        if rows and full:
            p.dO_t = None
        if name == "mkda_bwd_dh_ordered":
            assert (lib.mkda_bwd_dh_rows if rows else lib.mkda_bwd_dh_ordered)(ctypes.byref(p), *args) == 0
        elif rows:
            assert lib.mkda_bwd_chunk_rows(ctypes.byref(p), do.data_ptr(), None, None, *args) == 0
        else:
            assert lib.mkda_bwd_chunk(ctypes.byref(p), *args) == 0
    monkeypatch.setattr(_lib, "call", call)
    for rows in (False, True):
        dq, dk = (torch.full((lay.NC, HV, 64, 128), float("nan"), device="cuda") for _ in range(2))
        dh, dVd, dO, dh0 = ops.bwd_dh(lay, do, kbar, qs, gl, Aqk, nw, HK, HV, want_dh0=True)
        out = ops.bwd_chunk(lay, lv["q"], lv["k"], lv["v"], None, None, g_c, be, A, h, dh, Vd, dO, dVd, 128 ** -0.5, HK, HV, lv["beta"], True, 2.0, scalar_gate=scalar)
        both.append((dh, dVd, dh0, dq, dk, *out[2:]))
    for i, (a, b) in enumerate(zip(*both)):
        assert torch.equal(a.view(torch.int32) if a.dtype == torch.float32 else a, b.view(torch.int32) if b.dtype == torch.float32 else b), i
    assert not torch.isnan(both[1][3]).any() and not torch.isnan(both[1][4]).any()
