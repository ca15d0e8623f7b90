"""GPU: sequences longer than 1.85 segments are cut (pre-pass, prefix combine, main pass), shorter ones are not: a sequence at each side of the
line, with and without warm-up truncation, against the uncut call."""
import pytest
import torch

import mogankda_b200 as mk
from mogankda_b200.index import get_layout
from oracle import kda_oracle as orc
from tests.common import check, compare, make_inputs, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks,decay,warm", [(59, -1e-4, -10.0), (60, -1e-4, None), (60, -1e-4, -10.0), (65, -0.5, None), (65, -0.5, -10.0)])
def test_sequences_around_the_line(chunks, decay, warm):
    """Weak decay: truncation skips nothing and the results are bit for bit those of the cut call without it.  Strong decay: the pre-passes are
    truncated.  All against the uncut call."""
    lv, do, dht, opts, epi = make_inputs(B=1, T=64 * chunks - 23, dtype=torch.float32, gate="precomputed", seed=15, HV=2)
    lv["g"] = torch.full_like(lv["g"], decay)
    cut = lambda ratio: get_layout(1, 64 * chunks - 23, None, lv["q"].device, 32, 2, ratio).segmented      # noqa: E731
    assert cut(2.5) == (chunks > 59) and cut(1.25)                    # without and with truncation
    flat = run(mk.chunk_delta_rule, lv, do, dht, opts, epi, vfirst=True, auto_cp=False)
    got = run(mk.chunk_delta_rule, lv, do, dht, opts, epi, vfirst=True, warmup_threshold=warm)
    for n, t in flat.items():
        check(n, got[n], t)
    if warm is not None and decay > -1e-3 and chunks > 59:
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


def test_cut_batch_with_segments_of_unequal_length():
    """More (segment, head) chains than SMs and a natural order that is not longest first: every pass of a cut batch, forward and backward, is
    started on in another order.  Against the oracle, states in and out."""
    lens, HV = (64 * 69 + 7, 64 * 3, 64 * 40 + 1, *(64 * (1 + i % 8) - 5 * i for i in range(14))), 8
    cu = [0, *torch.tensor(lens).cumsum(0).tolist()]
    lv, do, dht, opts, epi = make_inputs(T=cu[-1], HK=4, HV=HV, cu=tuple(cu), dtype=torch.float32, gate="kimi", seed=37)
    lay = get_layout(1, cu[-1], opts["cu_seqlens"], lv["q"].device, 32, HV)
    assert lay.segmented and lay.NS * HV > torch.cuda.get_device_properties(0).multi_processor_count
    assert lay.host["seg_order"][:4] == [0, 1, 4, 5]                      # 32, 32, 32 and 9 chunks; 6 and 3 lie between
    compare(run(mk.chunk_delta_rule, lv, do, dht, opts, epi, vfirst=True), run(orc.chunked_delta_rule, lv, do, dht, opts, epi, f64=True, vfirst=True))


@pytest.mark.parametrize("vfirst", [False, True])
@pytest.mark.parametrize("lens,seg", [((1,), 3), ((64,), 3), ((65, 1), 3), ((64 * 9 + 1, 0, 130), 3), ((64 * 45 - 3, 300), 32)])
def test_state_and_transition_in_one_cta(lens, seg, vfirst, monkeypatch):
    """More than one (segment, head) pair per two SMs: mkda_recur_fwd carries state and transition of a pair in one CTA; with a state to start
    from (here zero) in two.  Segments of 0 to 3 and of 5 to 32 chunks, ragged ends, started on in any order, final states of the last and of the
    first segment only and swapped: the same bits."""
    from mogankda_b200 import _lib, ops
    cu, HV = [0, *torch.tensor(lens).cumsum(0).tolist()], 80
    lv, _, _, opts, _ = make_inputs(T=cu[-1], HK=HV, HV=HV, cu=tuple(cu), dtype=torch.bfloat16, gate="kimi", epi=None, h0=False, seed=31)
    lay = get_layout(1, cu[-1], opts["cu_seqlens"], lv["q"].device, seg)
    assert 2 * HV * lay.NS > torch.cuda.get_device_properties(0).multi_processor_count
    g_c, be = ops.gate_cumsum_fwd(lay, lv["g"], "kimi", lv["A_log"], lv["dt_bias"], -5.0, HV, beta_raw=lv["beta"], beta_sigmoid=True, beta_scale=2.0)
    rq, rk = ops.l2norm_rstd(lv["q"]), ops.l2norm_rstd(lv["k"])
    _, _, nw, u, kbar, _, gl = ops.intra_fwd(lay, lv["q"], lv["k"], lv["v"], rq, rk, g_c, be, 128 ** -0.5, HV, HV)
    kw = dict(store_h=False, store_vd=False, want_transition=True, state_v_first=vfirst)
    order = torch.randperm(lay.NS, generator=torch.Generator().manual_seed(7)).int().cuda()
    zero = torch.zeros(lay.NS, HV, 128, 128, device="cuda")
    _, _, ht, mt = ops.recur_fwd(lay, nw, u, kbar, gl, HV, HV, seg_order=order, **kw)
    _, _, ht2, mt2 = ops.recur_fwd(lay, nw, u, kbar, gl, HV, HV, h0=zero, **kw)
    assert torch.equal(ht, ht2) and torch.equal(mt, mt2) and torch.isfinite(ht).all() and torch.isfinite(mt).all()
    rows = torch.full((lay.NS,), -1, dtype=torch.int32, device="cuda")
    rows[0], rows[-1] = lay.NS - 1, 0
    call, empty = _lib.call, torch.empty

    def chosen(name, p, *args):
        p.seg_ht = rows.data_ptr()
        return call(name, p, *args)
    monkeypatch.setattr(_lib, "call", chosen)
    monkeypatch.setattr(torch, "empty", lambda *a, **k: empty(*a, **k).fill_(7.0))
    _, _, ht3, mt3 = ops.recur_fwd(lay, nw, u, kbar, gl, HV, HV, **kw)
    assert torch.equal(ht3[-1], ht[0]) and torch.equal(ht3[0], ht[-1]) and (ht3[1:-1] == 7).all() and torch.equal(mt3, mt)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("epi,scalar,dtype", [("silu", False, torch.float32), (None, False, torch.bfloat16), (None, True, torch.float16)])
@pytest.mark.parametrize("T", [1, 64, 193])
def test_a_sequence_alone_and_among_many(T, epi, scalar, dtype):
    """A sequence has the same bits alone (serial kernels by two CTAs per chain where they are separate ones, few items) and among so many others that no
    chain is shared, states in and out in both layouts, forward only and with a backward pass; forward only without a state to start from, which
    a continuation of at most 16 tokens would take to another kernel."""
    HV, N = 4, torch.cuda.get_device_properties(0).multi_processor_count // 8 + 1
    gate = "precomputed" if scalar else "eda"
    lv, do, dht, opts, epi = make_inputs(B=N, T=T, HK=2, HV=HV, dtype=dtype, gate=gate, scalar=scalar, epi=epi, seed=41)
    first = lambda t: t[:1].contiguous() if t.dim() >= 3 and t.shape[0] == N else t          # noqa: E731
    for vfirst in (False, True):
        many = run(mk.chunk_delta_rule, lv, do, dht, opts, epi, vfirst=vfirst)
        one = run(mk.chunk_delta_rule, {k: first(t) for k, t in lv.items()}, first(do), first(dht), opts, epi, vfirst=vfirst)
        for k in ("o", "ht", "dq", "dk", "dv", "dg", "dbeta", "dh0"):
            assert torch.equal(many[k][:1], one[k]), k
        lone = {k: t for k, t in lv.items() if k != "h0"}
        with torch.no_grad():
            many = run(mk.chunk_delta_rule, lone, do, dht, opts, epi, vfirst=vfirst, grads=False)
            one = run(mk.chunk_delta_rule, {k: first(t) for k, t in lone.items()}, first(do), first(dht), opts, epi, vfirst=vfirst, grads=False)
        for k in ("o", "ht"):
            assert torch.equal(many[k][:1], one[k]), k


@pytest.mark.parametrize("vfirst", [False, True])
@pytest.mark.parametrize("lens", [(1,), (64, 0), (193, 65, 0, 128)])
def test_a_chain_shared_by_two_ctas(lens, vfirst):
    """recur_fwd and bwd_dh: up to half as many (sequence, head) chains as SMs, those of the transitions counted, are shared by two CTAs of 64 rows of the
    transposed state each.  Every sequence, an empty one too, has the bits that it has among so many copies that no chain is shared: states, Vd, final
    states and transitions (a state to start from keeps state and transition in CTAs of their own), and their reverses."""
    from mogankda_b200 import ops
    HV, N, sms = 4, len(lens), torch.cuda.get_device_properties(0).multi_processor_count
    times = sms // (2 * HV * N) + 1
    T, cu = sum(lens), [0, *torch.tensor(lens).cumsum(0).tolist()]
    lv, do, dht, opts, _ = make_inputs(T=T, HK=HV, HV=HV, cu=tuple(cu), dtype=torch.bfloat16, gate="kimi", epi=None, seed=43)
    assert 2 * 2 * HV * N <= sms < 2 * HV * N * times

    def serial(copies, transition):
        rep = lambda t, dim: torch.cat([t] * copies, dim)                                  # noqa: E731
        many = torch.tensor([0] + [c + T * r for r in range(copies) for c in cu[1:]], dtype=torch.int32, device="cuda")
        lay = get_layout(1, T * copies, many, lv["q"].device, 32)
        q, k, v, g, b = (rep(lv[n], 1) for n in ("q", "k", "v", "g", "beta"))
        g_c, be = ops.gate_cumsum_fwd(lay, g, "kimi", lv["A_log"], lv["dt_bias"], -5.0, HV, beta_raw=b, beta_sigmoid=True, beta_scale=2.0)
        _, Aqk, nw, u, kbar, qs, gl = ops.intra_fwd(lay, q, k, v, ops.l2norm_rstd(q), ops.l2norm_rstd(k), g_c, be, 128 ** -0.5, HV, HV)
        h, Vd, ht, mt = ops.recur_fwd(lay, nw, u, kbar, gl, HV, HV, h0=rep(lv["h0"], 0), state_v_first=vfirst, want_transition=transition)
        dh, dVd, _, dh0 = ops.bwd_dh(lay, rep(do, 1), kbar, qs, gl, Aqk, nw, HV, HV, dht=rep(dht, 0), state_v_first=vfirst)
        _, _, _, short = ops.bwd_dh(lay, rep(do, 1), kbar, qs, gl, Aqk, nw, HV, HV, dht=rep(dht, 0), state_v_first=vfirst, store=False)
        return dict(h=h, Vd=Vd, ht=ht, dh=dh, dVd=dVd, dh0=dh0, dh0_only=short, **(dict(mt=mt) if transition else {}))

    for transition in (False, True):
        shared, whole = serial(1, transition), serial(times, transition)
        for k, t in shared.items():
            assert torch.isfinite(t.view(torch.bfloat16) if k in ("h", "Vd", "dh", "dVd") else t).all(), k
            for r in range(times):
                assert torch.equal(whole[k][r * t.shape[0]:(r + 1) * t.shape[0]].view(torch.int32), t.view(torch.int32)), (k, r, transition)


# chunks of the documents, v-heads, norm, backward pass -> output in a kernel of its own.  148 SMs; faster by (us, fused and separate) ...
@pytest.mark.parametrize("chunks,HV,norm,train,apart", [
    ((47, 32, 24, 16, 11), 16, True, True, True),          # 420, 377: more chains than half the SMs, but the longest sets the time
    ((32, *[8] * 12), 16, True, True, True),               # 307, 285
    ((48, *[1] * 12), 8, True, False, True),               # 246, 209
    ((48, *[1] * 12), 8, False, True, True),               # 231, 207
    ((48, *[1] * 12), 8, False, False, False),             # without a norm and forward only the fused step is no longer than that of the state alone
    ((24,) * 5, 16, True, True, False),                    # 279, 291: equal chains
    ((24,) * 8, 16, True, False, False),                   # 317, 416
    ((24,) * 4, 16, True, True, True),                     # 258, 242: chains that two CTAs share
    ((24,) * 4, 16, True, False, False),                   # 219, 236
])
def test_output_in_the_chain_or_apart(chunks, HV, norm, train, apart):
    """The faster one also where chains are of unequal length: gate, WY preparation and chain are three launches, a separate output is one more.  Either way each
    document has the bits of its own call."""
    from mogankda_b200 import _lib
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("measured on 148 SMs")
    lens = [64 * n - 3 for n in chunks]
    cu = [0, *torch.tensor(lens).cumsum(0).tolist()]
    lv, _, _, opts, epi = make_inputs(T=cu[-1], HK=HV // 2, HV=HV, cu=tuple(cu), dtype=torch.bfloat16, gate="kimi", epi="silu" if norm else None, h0=False, seed=53)
    assert not get_layout(1, cu[-1], opts["cu_seqlens"], lv["q"].device, 32, HV).segmented

    def call(lv, cu):
        with torch.set_grad_enabled(train):
            norm_ = dict(weight=lv["ep_w"], gate=lv["ep_gate"], act=epi, eps=1e-6) if norm else None
            before = _lib.launch_count()
            o, ht = mk.chunk_kda(lv["q"].detach().requires_grad_(train), lv["k"], lv["v"], lv["g"], lv["beta"], A_log=lv["A_log"], dt_bias=lv["dt_bias"],
                                 output_norm=norm_, **dict(opts, cu_seqlens=cu))
            return o.detach(), ht.detach(), _lib.launch_count() - before
    o, ht, launches = call(lv, opts["cu_seqlens"])
    assert launches == 3 + apart
    for d in (0, len(lens) - 1):
        s, e = cu[d], cu[d + 1]
        one = call({k: (t[:, s:e].contiguous() if t.dim() >= 3 and t.shape[1] == cu[-1] else t) for k, t in lv.items()}, None)
        assert torch.equal(o[:, s:e], one[0]) and torch.equal(ht[d:d + 1], one[1]), d


@pytest.mark.parametrize("chunks,HV", [((4,) * 4, 8), ((4, 4), 16)])       # 38.1 us fused and 36.6 separate; 38.2, 36.8
def test_output_apart_in_small_calls(chunks, HV):
    """States and Vd that only the separate kernels allocate are no reason to stay with the slower one where they are a few MB."""
    from mogankda_b200 import _lib
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("measured on 148 SMs")
    cu = [0, *torch.tensor([64 * n for n in chunks]).cumsum(0).tolist()]
    lv, _, _, opts, epi = make_inputs(T=cu[-1], HK=HV // 2, HV=HV, cu=tuple(cu), dtype=torch.bfloat16, gate="kimi", epi="silu", h0=False, seed=61)
    before = _lib.launch_count()
    with torch.no_grad():
        mk.chunk_kda(lv["q"], lv["k"], lv["v"], lv["g"], lv["beta"], A_log=lv["A_log"], dt_bias=lv["dt_bias"],
                     output_norm=dict(weight=lv["ep_w"], gate=lv["ep_gate"], act=epi, eps=1e-6), **opts)
    assert _lib.launch_count() - before == 3               # gate and WY preparation, chain, output


# ... and with a 32-bit gate (us, fused and separate)
@pytest.mark.parametrize("chunks,HV,train,apart", [
    ((48, *[1] * 30), 16, False, True),                    # 674, 285
    ((48,) * 6, 16, True, True),                           # 1021, 621
    ((16,) * 8, 8, False, True),                           # chains that two CTAs share
    ((1,) * 2, 4, False, False),                           # one step: 27.5, 28.9
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_output_apart_from_the_chain_with_a_32_bit_gate(dtype, chunks, HV, train, apart):
    """The fused kernel has no place for the rows of such a gate and fetches them while everything waits.  The gate's type decides, not that of q, k and v; the bits are
    those of each document's own call."""
    from mogankda_b200 import _lib
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("measured on 148 SMs")
    lens = [64 * n - 3 for n in chunks]
    cu = [0, *torch.tensor(lens).cumsum(0).tolist()]
    lv, _, _, opts, epi = make_inputs(T=cu[-1], HK=HV // 2, HV=HV, cu=tuple(cu), dtype=dtype, gate="kimi", epi="silu", h0=False, seed=59)

    def call(lv, cu):
        with torch.set_grad_enabled(train):
            before = _lib.launch_count()
            o, ht = mk.chunk_kda(lv["q"].detach().requires_grad_(train), lv["k"], lv["v"], lv["g"], lv["beta"], A_log=lv["A_log"], dt_bias=lv["dt_bias"],
                                 output_norm=dict(weight=lv["ep_w"], gate=lv["ep_gate"].float(), act=epi, eps=1e-6), **dict(opts, cu_seqlens=cu))
            return o.detach(), ht.detach(), _lib.launch_count() - before
    o, ht, launches = call(lv, opts["cu_seqlens"])
    one_kernel = sum(chunks) * HV <= 148                   # gate and WY preparation
    assert launches == 3 - one_kernel + apart
    for d in (0, len(lens) - 1):
        s, e = cu[d], cu[d + 1]
        one = call({k: (t[:, s:e].contiguous() if t.dim() >= 3 and t.shape[1] == cu[-1] else t) for k, t in lv.items()}, None)
        assert torch.equal(o[:, s:e], one[0]) and torch.equal(ht[d:d + 1], one[1]), d
