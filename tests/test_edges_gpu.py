"""GPU: branches of the kernels and of their dispatch at the sizes and values where they can go wrong, against the fp64 oracle with the
bars of tests/common.py."""
import pytest
import torch

import mogankda_b200 as mk
from oracle import kda_oracle as orc
from tests.common import compare, make_inputs, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scalar", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_precomputed_beta_of_zero_and_near_zero(scalar, dtype):
    """dbeta does not go through a division by beta.  Chunks without a row of beta near zero, with one, with all rows zero, and a ragged last
    chunk."""
    lv, do, dht, opts, _ = make_inputs(B=2, T=64 * 3 + 21, HK=2, HV=4, dtype=dtype, gate="precomputed", scalar=scalar, beta="precomputed",
                                       epi=None, seed=41)
    lv["beta"][0, 70] = 0.0
    lv["beta"][0, 71] = 1e-13
    lv["beta"][1, 64:128] = 0.0
    lv["beta"][1, 64 * 3 + 20, 1] = 0.0
    compare(run(mk.chunk_delta_rule, lv, do, dht, opts, None),
            run(orc.chunked_delta_rule, lv, do, dht, opts, None, f64=True))


@pytest.mark.parametrize("b_mn", [0, 1])
@pytest.mark.parametrize("N,K", [(64, 64), (64, 128), (128, 64), (128, 128)])
def test_tensor_core_product_with_the_left_operand_in_tensor_memory(b_mn, N, K):
    """mkda_selftest_umma, mode bit 2: the error must be at the 2^-16 level of the split, as with both operands in shared memory."""
    from mogankda_b200 import _lib
    torch.manual_seed(11)
    A, B, D = torch.randn(128, K, device="cuda"), torch.randn(N, K, device="cuda"), torch.zeros(128, N, device="cuda")
    p = _lib.STRUCTS["MkdaSelfTest"]()
    p.A, p.B, p.D, p.N, p.K, p.mode = A.data_ptr(), B.data_ptr(), D.data_ptr(), N, K, 4 | b_mn
    _lib.call("mkda_selftest_umma", p, torch.cuda.current_stream().cuda_stream)
    ref = A.double() @ B.double().T
    assert ((D.double() - ref).abs().max() / ref.abs().max()).item() < 5e-5


@pytest.mark.parametrize("offset", [4, 8])
def test_states_at_odd_storage_offsets(offset):
    """[V,K] states travel in 32-byte pieces: views 16 and 32 bytes into their storage, and gradients that arrive as such views."""
    lv, do, dht, opts, epi = make_inputs(B=2, T=150, dtype=torch.bfloat16, gate="eda", seed=43)
    flat = torch.zeros(lv["h0"].numel() + offset, device="cuda")
    flat[offset:] = lv["h0"].transpose(-1, -2).reshape(-1)
    h0 = flat[offset:].view(lv["h0"].shape)
    up = torch.zeros(dht.numel() + offset, device="cuda")
    up[offset:] = dht.reshape(-1)

    def call(h0, dht):
        h0 = h0.detach().requires_grad_(True)
        o, ht = mk.chunk_delta_rule(lv["q"], lv["k"], lv["v"], lv["g"], lv["beta"], A_log=lv["A_log"], dt_bias=lv["dt_bias"], initial_state=h0,
                                    state_v_first=True, **opts)
        return o, ht, torch.autograd.grad(ht, h0, dht)[0]

    for a, b in zip(call(h0.clone(), dht), call(h0, up[offset:].view(dht.shape))):
        assert torch.equal(a, b)


@pytest.mark.parametrize("case", [
    dict(B=3, T=1, gate="kimi", dtype=torch.bfloat16, epi="silu"),
    dict(B=2, T=16, gate="eda", dtype=torch.float32, epi="sigmoid", vfirst=True),
    dict(B=2, T=17, gate="eda", dtype=torch.float32, epi=None),
    dict(cu=(0, 1, 1, 6, 22, 22), T=25, gate="gdn", dtype=torch.float16, epi="silu", vfirst=True),
    dict(B=5, T=2, gate="gdn", scalar=True, dtype=torch.bfloat16, epi=None, vfirst=True),
    dict(B=1, T=9, gate="precomputed", beta="precomputed", l2=False, dtype=torch.float32, epi=None, h0=False),
    dict(B=2, T=4, gate="eda", dtype=torch.bfloat16, epi="silu", x_dtype=torch.bfloat16)], ids=str)
def test_forward_of_very_short_sequences(case):
    """Without gradients and with an initial state, sequences of up to 16 tokens run token by token; 17 tokens, and a sequence that starts from
    zero, take the chunk kernels.  Empty sequences, padding and 4 v-heads on 2 q/k heads included."""
    case = dict(case)
    vfirst = case.pop("vfirst", False)
    lv, do, dht, opts, epi = make_inputs(HK=2, HV=4, seed=47, **case)
    got = run(mk.chunk_delta_rule, lv, do, dht, opts, epi, vfirst=vfirst, grads=False)
    end = case["cu"][-1] if "cu" in case else case["T"]
    cut = {n: (t[:, :end].contiguous() if t.dim() >= 3 and n != "h0" else t) for n, t in lv.items()}
    ref = run(orc.recurrent_delta_rule, cut, do[:, :end], dht, opts, epi, f64=True, vfirst=vfirst, grads=False)
    assert (got["o"][:, end:] == 0).all()
    got["o"] = got["o"][:, :end]
    compare(got, ref)


@pytest.mark.parametrize("NC,G", [(1, 2), (3, 4), (149, 2), (300, 2)])
def test_few_groups_are_spread_over_v_heads(NC, G):
    """With few (chunk, q/k head) groups the backward pass gives every v-head tiles of its own, which the finishing kernel adds: the same
    sums in the same order, so expanding one head's work over more chunks must not change a bit of an earlier chunk."""
    lv, do, dht, opts, epi = make_inputs(B=NC, T=64, HK=1, HV=G, dtype=torch.float32, gate="eda", seed=53, h0=False, epi=None)
    full = run(mk.chunk_delta_rule, lv, do, dht, opts, epi)
    sub = {n: (t[:1].contiguous() if t.dim() >= 3 else t) for n, t in lv.items()}
    one = run(mk.chunk_delta_rule, sub, do[:1], dht[:1], opts, epi)
    for n in ("dq", "dk", "dv", "dg", "dbeta"):
        assert torch.equal(full[n][:1], one[n]), n
    compare(one, run(orc.chunked_delta_rule, sub, do[:1], dht[:1], opts, epi, f64=True))


@pytest.mark.parametrize("scalar", [False, True])
def test_next_items_brought_into_l2(scalar):
    """From 964 (chunk, v-head) items on the backward kernel hints the next item's tiles into L2, and a CTA walks several items: no bit of the
    gradients may differ from those of the same heads in calls of 510 items."""
    lv, do, dht, opts, epi = make_inputs(T=64 * 16 + 21, HK=60, HV=60, dtype=torch.bfloat16, gate="precomputed", scalar=scalar, beta="precomputed", h0=False, epi=None, seed=71)
    full = run(mk.chunk_delta_rule, lv, do, dht, opts, epi)
    for h in (slice(0, 30), slice(30, 60)):
        sub = {n: t[:, :, h].contiguous() for n, t in lv.items()}
        part = run(mk.chunk_delta_rule, sub, do[:, :, h].contiguous(), dht[:, h].contiguous(), opts, epi)
        for n in ("dq", "dk", "dv", "dg", "dbeta"):
            assert torch.equal(full[n][:, :, h], part[n]), n


@pytest.mark.parametrize("rows,cols,group", [(1, 1, 1), (33, 7, 1), (255, 64, 1), (257, 33, 1), (1184, 128, 1), (5, 256, 128), (64, 384, 3)])
def test_partial_reductions(rows, cols, group):
    from mogankda_b200 import ops
    x = torch.randn(rows, cols, device="cuda")
    got = ops.reduce_partials(x, rows, cols, group)
    ref = x.double().view(rows, cols // group, group).sum((0, 2))
    assert got.shape == ref.shape and ((got - ref).abs() <= 1e-6 * x.double().abs().view(rows, cols // group, group).sum((0, 2))).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_value_gradient_on_a_16_byte_boundary(dtype, monkeypatch):
    """mkda_bwd_chunk stores dv in 32-byte pieces where its address allows that, in 16-byte pieces otherwise: the same bits, and none beside
    them.  Chunks of 1, 64 and 35 rows."""
    from mogankda_b200 import _lib, ops
    from mogankda_b200.index import get_layout
    lv, do, _, opts, _ = make_inputs(cu=(0, 1, 100), T=100, HK=1, HV=2, dtype=dtype, gate="eda", h0=False, epi=None, seed=83)
    lay = get_layout(1, 100, opts["cu_seqlens"], lv["q"].device)
    rq, rk = ops.l2norm_rstd(lv["q"]), ops.l2norm_rstd(lv["k"])
    g_c, be = ops.gate_cumsum_fwd(lay, lv["g"], "eda", lv["A_log"], lv["dt_bias"], -5.0, 2, beta_raw=lv["beta"], beta_sigmoid=True, beta_scale=2.0)
    A, Aqk, nw, u, kbar, qs, gl = ops.intra_fwd(lay, lv["q"], lv["k"], lv["v"], rq, rk, g_c, be, 128 ** -0.5, 1, 2)
    h, Vd, _, _ = ops.recur_fwd(lay, nw, u, kbar, gl, 1, 2)
    dh, dVd_t, dO_t, _ = ops.bwd_dh(lay, do.to(dtype), kbar, qs, gl, Aqk, nw, 1, 2)
    args = (lay, lv["q"], lv["k"], lv["v"], rq, rk, g_c, be, A, h, dh, Vd, dO_t, dVd_t, 128 ** -0.5, 1, 2, lv["beta"], True, 2.0)
    dv = ops.bwd_chunk(*args)[4]
    buf = torch.full((100 * 2 * 128 + 16,), 7.0, dtype=dtype, device="cuda")
    call = _lib.call

    def shifted(name, p, stream):
        p.dv = buf.data_ptr() + 16
        return call(name, p, stream)
    monkeypatch.setattr(_lib, "call", shifted)
    ops.bwd_chunk(*args)
    assert torch.equal(buf[8:-8].view_as(dv), dv) and (buf[:8] == 7).all() and (buf[-8:] == 7).all()


@pytest.mark.parametrize("epi", [None, "silu"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_output_in_the_chain_kernel(dtype, epi):
    """mkda_chain_fwd against mkda_recur_fwd + mkda_out_fwd: chunks of 1, 15, 16, 17, 48 and 64 rows (its rows leave in groups of 16), states and
    Vd saved or not.  Which of the two runs depends on the sizes of the call, results must not: bit for bit the same."""
    from mogankda_b200 import _lib, ops
    from mogankda_b200.index import get_layout
    cu = (0, 1, 16, 32, 49, 97, 225, 225, 400)
    lv, do, dht, opts, _ = make_inputs(cu=cu, T=404, HK=2, HV=4, dtype=dtype, gate="eda", seed=61)
    lay = get_layout(1, 404, opts["cu_seqlens"], lv["q"].device)
    rq, rk = ops.l2norm_rstd(lv["q"]), ops.l2norm_rstd(lv["k"])
    g_c, be = ops.gate_cumsum_fwd(lay, lv["g"], "eda", lv["A_log"], lv["dt_bias"], -5.0, 4, beta_raw=lv["beta"], beta_sigmoid=True, beta_scale=2.0)
    A, Aqk, nw, u, kbar, qs, gl = ops.intra_fwd(lay, lv["q"], lv["k"], lv["v"], rq, rk, g_c, be, 128 ** -0.5, 2, 4)
    h, Vd, ht, _ = ops.recur_fwd(lay, nw, u, kbar, gl, 2, 4, h0=lv["h0"])
    norm = None if epi is None else dict(weight=lv["ep_w"], gate=lv["ep_gate"], act=epi, eps=1e-6)
    odt = dtype if epi is None else torch.float32
    out, raw = ops.out_fwd(lay, qs, Aqk, Vd, h, 2, 4, odt, norm=norm, keep_raw=epi is not None)
    for save in (True, False):
        p = _lib.STRUCTS["MkdaChainFwd"]()
        h2, Vd2, ht2 = torch.empty_like(h), torch.empty_like(Vd), torch.empty_like(ht)
        out2, raw2 = torch.zeros_like(out), torch.zeros(404, 4, 128, device="cuda")
        p.r.L = p.o.L = ops._layout_struct(lay, 2, 4)
        p.r.nw, p.r.u, p.r.kbar, p.r.gl, p.r.h0, p.r.ht = nw.data_ptr(), u.data_ptr(), kbar.data_ptr(), gl.data_ptr(), lv["h0"].data_ptr(), ht2.data_ptr()
        if save:
            p.r.h, p.r.Vd = h2.data_ptr(), Vd2.data_ptr()
        p.o.qs, p.o.Aqk, p.o.out, p.o.out_dtype = qs.data_ptr(), Aqk.data_ptr(), out2.data_ptr(), ops._dt(out2)
        if epi:
            p.o.has_norm, p.o.norm_w, p.o.norm_w_dtype, p.o.gate, p.o.gate_dtype = 1, lv["ep_w"].data_ptr(), 0, lv["ep_gate"].data_ptr(), ops._dt(lv["ep_gate"])
            p.o.act, p.o.eps, p.o.o_raw = ops.ACTS[epi], 1e-6, raw2.data_ptr()
        _lib.call("mkda_chain_fwd", p, torch.cuda.current_stream().cuda_stream)
        assert torch.equal(ht, ht2) and (not save or (torch.equal(h, h2) and torch.equal(Vd, Vd2)))
        if epi:
            assert torch.equal(raw, raw2)
        assert torch.equal(out, out2)


@pytest.mark.parametrize("scalar,bound", [(False, 6.9e-6), (True, 5.7e-6)])
def test_beta_gradient_keeps_the_accuracy_of_v(scalar, bound):
    """dbeta = rowsum(dW * V) - rowsum(k~ * (dW S^T)) + rowsum(k * T) contracts all of dW with V itself.  On these inputs its error is 5.8e-6 (per
    channel) and 4.5e-6 (scalar gate); formed as (dW Vd^T)_ii / beta_i it inherits the errors of Vd, which went through the state chain: 8.1e-6
    and 7.4e-6.  The bounds are the geometric means of the two."""
    lv, do, dht, opts, _ = make_inputs(T=64 * 20 + 13, HK=8, HV=8, dtype=torch.bfloat16, gate="precomputed", scalar=scalar, beta="precomputed", epi=None,
                                       h0=False, seed=89)
    lv["g"] = lv["g"] * (0.02 if scalar else 0.1)          # weak decay: the state carries much of Vd
    got = run(mk.chunk_delta_rule, lv, do, dht, opts, None)["dbeta"].double()
    ref = run(orc.chunked_delta_rule, lv, do, dht, opts, None, f64=True)["dbeta"]
    assert ((got - ref).norm() / ref.norm()).item() < bound


@pytest.mark.parametrize("size", [1e-4, 1e-3, 1.0, 1e3, 1e7, 1e12])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("decay", [-5.0, -0.5])
def test_l2_norm_takes_rows_of_any_size(dtype, size, decay):
    """With the L2 norm in the kernels the scale of the raw q and k rows is the caller's: the anchored operands (decay factors up to 2^108 at the
    bound of -5 per token) must neither overflow nor lose their low halves.  Three full chunks and a ragged one."""
    lv, do, dht, opts, _ = make_inputs(T=64 * 3 + 21, HK=1, HV=2, dtype=dtype, gate="precomputed", epi=None, seed=97)
    lv["g"] = torch.full_like(lv["g"], decay)
    lv["q"], lv["k"] = (lv["q"].float() * size).to(dtype), (lv["k"].float() * size).to(dtype)
    compare(run(mk.chunk_delta_rule, lv, do, dht, opts, None), run(orc.chunked_delta_rule, lv, do, dht, opts, None, f64=True))


def test_calls_with_parameters_of_other_sizes_are_refused():
    lv, _, _, opts, _ = make_inputs(T=70, dtype=torch.bfloat16, gate="eda", epi="silu", h0=False, seed=101)
    call = lambda A, b, w, z: mk.chunk_kda(lv["q"], lv["k"], lv["v"], lv["g"], lv["beta"], A_log=A, dt_bias=b,          # noqa: E731
                                           output_norm=dict(weight=w, gate=z, act="silu"), **opts)
    good = (lv["A_log"], lv["dt_bias"], lv["ep_w"], lv["ep_gate"])
    call(*good)
    for i, bad in enumerate((lv["A_log"][:3], lv["dt_bias"][:, 0], lv["ep_w"][:64], lv["ep_gate"][:, :69])):
        with pytest.raises(AssertionError):
            call(*good[:i], bad.contiguous(), *good[i + 1:])


@pytest.mark.parametrize("scalar", [False, True])
def test_gradients_of_a_batch_without_tokens_are_zero(scalar):
    """Only empty sequences (padding tokens on a data-parallel rank): no kernel writes a partial sum, and every gradient is exactly zero, that of
    the initial state the upstream one.  Freed memory full of NaN stands ready for whatever is allocated."""
    from mogankda_b200 import ops
    from mogankda_b200.index import get_layout
    lv, do, dht, opts, epi = make_inputs(cu=(0, 0, 0), T=7, dtype=torch.bfloat16, gate="eda", scalar=scalar, epi="silu", seed=103)
    for n in (1 << 9, 1 << 12, 1 << 16, 1 << 20, 1 << 24):
        junk = [torch.full((n,), float("nan"), device="cuda") for _ in range(4)]
        del junk
    got = run(mk.chunk_delta_rule, lv, do, dht, opts, epi)
    assert torch.equal(got.pop("dh0"), dht) and torch.equal(got.pop("ht"), lv["h0"])
    for n, t in got.items():
        assert (t == 0).all(), n
    lay = get_layout(1, 7, opts["cu_seqlens"], do.device)
    _, db, da = ops.gate_bwd(lay, lv["g"], torch.empty(1, device="cuda"), "eda", lv["A_log"], lv["dt_bias"], -5.0, 4, True, True)
    assert (db == 0).all() and (da == 0).all()


def _training_call(T, epi, seed):
    lv, do, dht, opts, epi = make_inputs(T=T, HK=2, HV=4, dtype=torch.bfloat16, gate="eda", epi=epi, seed=seed)
    x = {n: t.clone().requires_grad_(True) for n, t in lv.items()}
    norm = None if epi is None else dict(weight=x["ep_w"], gate=x["ep_gate"], act=epi)
    f = lambda q: mk.chunk_delta_rule(q, x["k"], x["v"], x["g"], x["beta"], A_log=x["A_log"], dt_bias=x["dt_bias"], initial_state=x["h0"],          # noqa: E731
                                      output_norm=norm, **opts)
    grads = lambda o, ht: torch.autograd.grad((o, ht), list(x.values()), (do.to(o.dtype), dht))          # noqa: E731
    return f, x["q"], grads


# intermediates in one block | in a block each | sequences cut into segments
@pytest.mark.parametrize("T,epi", [(130, "silu"), (130, None), (64 * 80, "silu"), (64 * 300 + 9, None)])
def test_saved_tensor_hooks_get_the_intermediates(T, epi):
    """Offloading moves everything the backward pass needs, and what a hook brings back from another place is used: the same bits."""
    f, q, grads = _training_call(T, epi, 107)
    ref = grads(*f(q))
    sizes = []

    def pack(t):
        sizes.append(t.numel() * t.element_size())
        return t.cpu()
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        o, ht = f(q)
    chunk_heads = (T + 63) // 64 * 4
    assert sum(sizes) > chunk_heads * (65536 + 4 * 32768)          # states, nw, kbar, qs, Vd are among them
    for a, b in zip(ref, grads(o, ht)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("T,epi", [(130, "silu"), (64 * 80, "silu"), (64 * 300 + 9, None)])
def test_activation_checkpointing_frees_the_intermediates(T, epi):
    import gc
    from torch.utils.checkpoint import checkpoint
    f, q, grads = _training_call(T, epi, 109)
    ref = grads(*f(q))
    gc.collect()
    before = torch.cuda.memory_allocated()
    o, ht = checkpoint(f, q, use_reentrant=False)
    held = torch.cuda.memory_allocated() - before - o.numel() * o.element_size() - ht.numel() * 4
    assert held < 1 << 16, held
    for a, b in zip(ref, grads(o, ht)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("grads", [False, True])
def test_forward_mode_ad_is_refused(grads):
    """... not answered without a tangent, whichever tensor carries it."""
    import torch.autograd.forward_ad as fwad
    f, q, _ = _training_call(70, None, 113)
    with torch.set_grad_enabled(grads), fwad.dual_level():
        with pytest.raises(NotImplementedError):
            f(fwad.make_dual(q, torch.ones_like(q)))
    f(q)


def test_errors_of_the_library_are_mkda_errors():
    """A lower bound that is not negative is refused by the kernels' entry points, on the chunk path and on the path of a few tokens."""
    from mogankda_b200 import _lib
    lv, _, _, opts, _ = make_inputs(T=70, dtype=torch.bfloat16, gate="kimi", epi=None, h0=False, seed=127)
    for T in (70, 3):
        cut = {n: t[:, :T].contiguous() for n, t in lv.items() if t.dim() > 2}
        h0 = torch.zeros(1, 4, 128, 128, device="cuda") if T == 3 else None
        with torch.no_grad(), pytest.raises(_lib.MkdaError, match="lower_bound"):
            mk.chunk_kda(cut["q"], cut["k"], cut["v"], cut["g"], cut["beta"], A_log=lv["A_log"], dt_bias=lv["dt_bias"], initial_state=h0,
                         **dict(opts, lower_bound=1.0))


@pytest.mark.parametrize("epi", [None, "silu"])
@pytest.mark.parametrize("vfirst", [False, True])
def test_a_short_continuation_does_not_depend_on_the_rest_of_the_batch(epi, vfirst):
    """Forward-only calls with states: sequences of 0, 1, 5, 16 (token by token), 17, 40 and 100 tokens (chunks) packed together and padding behind
    them give the bits that each gives alone."""
    cu = (0, 5, 45, 45, 46, 62, 79, 179)
    lv, do, dht, opts, _ = make_inputs(cu=cu, T=183, HK=2, HV=4, dtype=torch.bfloat16, gate="eda", epi=epi, seed=131)
    alone = dict(opts, cu_seqlens=None)
    got = run(mk.chunk_delta_rule, lv, do, dht, opts, epi, vfirst=vfirst, grads=False)
    assert (got["o"][:, 179:] == 0).all()
    for n, (a, b) in enumerate(zip(cu[:-1], cu[1:])):
        if a == b:
            h0 = lv["h0"][n].transpose(-1, -2) if vfirst else lv["h0"][n]
            assert torch.equal(got["ht"][n], h0)
            continue
        sub = {m: (t[n:n + 1] if m == "h0" else t[:, a:b].contiguous() if t.dim() >= 3 else t) for m, t in lv.items()}
        one = run(mk.chunk_delta_rule, sub, do[:, a:b], dht[n:n + 1], alone, epi, vfirst=vfirst, grads=False)
        assert torch.equal(got["o"][:, a:b], one["o"]) and torch.equal(got["ht"][n:n + 1], one["ht"]), (n, b - a)
