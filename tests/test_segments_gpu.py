"""GPU: sequences longer than two segments are cut (pre-pass, prefix combine, main pass), shorter ones are not: a sequence at each side of the
line, with and without warm-up truncation, against the uncut call."""
import pytest
import torch

import mogankda_b200 as mk
from mogankda_b200.index import get_layout
from tests.common import check, make_inputs, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warm", [None, -10.0])
@pytest.mark.parametrize("chunks,decay", [(64, -1e-4), (65, -1e-4), (65, -0.5)])
def test_sequences_around_two_segments(chunks, decay, warm):
    """Weak decay: truncation skips nothing and the results are bit for bit those of the cut call without it.  Strong decay: the pre-passes are
    truncated.  All against the uncut call."""
    lv, do, dht, opts, epi = make_inputs(B=1, T=64 * chunks - 23, dtype=torch.float32, gate="precomputed", seed=15, HV=2)
    lv["g"] = torch.full_like(lv["g"], decay)
    ratio = 2.5 if warm is None else 1.25
    assert get_layout(1, 64 * chunks - 23, None, lv["q"].device, 32, 2, ratio).segmented == (chunks > 64 or warm is not None)
    flat = run(mk.chunk_delta_rule, lv, do, dht, opts, epi, vfirst=True, auto_cp=False)
    got = run(mk.chunk_delta_rule, lv, do, dht, opts, epi, vfirst=True, warmup_threshold=warm)
    for n, t in flat.items():
        check(n, got[n], t)
    if warm is not None and decay > -1e-3 and chunks > 64:
        exact = run(mk.chunk_delta_rule, lv, do, dht, opts, epi, vfirst=True)
        assert all(torch.equal(t, got[n]) for n, t in exact.items())


def test_longest_first_changes_nothing():
    """More (document, head) chains than SMs are started longest first: every document, its states included, has the bits of its own call."""
    lens, HV = (70, 1, 200, 64, 129, 0, 70, 333), 32
    cu = [0, *torch.tensor(lens).cumsum(0).tolist()]
    lv, do, dht, opts, epi = make_inputs(T=cu[-1], HK=16, HV=HV, cu=tuple(cu), dtype=torch.bfloat16, gate="kimi", epi=None, seed=29)
    lay = get_layout(1, cu[-1], opts["cu_seqlens"], lv["q"].device, 32, HV)
    assert not lay.segmented and len(lens) * HV > torch.cuda.get_device_properties(0).multi_processor_count
    assert lay.host["seg_order"] == [7, 2, 4, 0, 6, 1, 3, 5]              # by chunks: 6, 4, 3, 2, 2, 1, 1, 0
    got = run(mk.chunk_delta_rule, lv, do, dht, opts, epi)
    for d, n in enumerate(lens):
        if n == 0:
            continue
        s, e = cu[d], cu[d + 1]
        sub = {k: (t[:, s:e].contiguous() if t.dim() >= 3 and t.shape[1] == cu[-1] else t) for k, t in lv.items()}
        sub["h0"] = lv["h0"][d:d + 1].contiguous()
        one = run(mk.chunk_delta_rule, sub, do[:, s:e].contiguous(), dht[d:d + 1].contiguous(), dict(opts, cu_seqlens=None), epi)
        assert torch.equal(got["ht"][d:d + 1], one["ht"]) and torch.equal(got["dh0"][d:d + 1], one["dh0"])
        for k in ("o", "dq", "dk", "dv", "dg", "dbeta"):
            assert torch.equal(got[k][:, s:e], one[k]), (k, d)


@pytest.mark.parametrize("lens", [(1,), (64,), (65, 1), (64 * 9 + 1, 0, 130)])
def test_state_and_transition_in_one_cta(lens):
    """More than one (segment, head) pair per two SMs: mkda_recur_fwd carries state and transition of a pair in one CTA; with a state to start
    from (here zero) in two.  Segments of 0 to 3 chunks, ragged ends: the same bits."""
    from mogankda_b200 import ops
    cu, HV = [0, *torch.tensor(lens).cumsum(0).tolist()], 80
    lv, _, _, opts, _ = make_inputs(T=cu[-1], HK=HV, HV=HV, cu=tuple(cu), dtype=torch.bfloat16, gate="kimi", epi=None, h0=False, seed=31)
    lay = get_layout(1, cu[-1], opts["cu_seqlens"], lv["q"].device, 3)
    assert 2 * HV * lay.NS > torch.cuda.get_device_properties(0).multi_processor_count
    g_c, be = ops.gate_cumsum_fwd(lay, lv["g"], "kimi", lv["A_log"], lv["dt_bias"], -5.0, HV, beta_raw=lv["beta"], beta_sigmoid=True, beta_scale=2.0)
    rq, rk = ops.l2norm_rstd(lv["q"]), ops.l2norm_rstd(lv["k"])
    _, _, nw, u, kbar, _, gl = ops.intra_fwd(lay, lv["q"], lv["k"], lv["v"], rq, rk, g_c, be, 128 ** -0.5, HV, HV)
    kw = dict(store_h=False, store_vd=False, want_transition=True)
    _, _, ht, mt = ops.recur_fwd(lay, nw, u, kbar, gl, HV, HV, **kw)
    _, _, ht2, mt2 = ops.recur_fwd(lay, nw, u, kbar, gl, HV, HV, h0=torch.zeros(lay.NS, HV, 128, 128, device="cuda"), **kw)
    assert torch.equal(ht, ht2) and torch.equal(mt, mt2) and torch.isfinite(ht).all() and torch.isfinite(mt).all()
