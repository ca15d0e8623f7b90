"""GPU: mkda_intra_fwd over ragged chunks.  Sequences of 1, 15, 16, 17, 33, 63, 64, 65 and 100 tokens once (one item per
CTA) and thirty times over (several, all buffers reused): the same bits everywhere, the fp64 chunk algebra, and
nothing of a neighbour that holds infinities."""
import pytest
import torch

from mogankda_b200 import ops
from mogankda_b200.index import get_layout
from tests.common import unpack_chunk_tiles, unpack_quarter_tiles, unpack_row_tiles

pytestmark = pytest.mark.gpu
LENS, HK, HV, TIMES = (1, 15, 16, 17, 33, 63, 64, 65, 100), 2, 4, 30
# Operands carry 16 mantissa bits (2^-17 rounding each, three factors with A), sums of up to 64 terms with A: well below 2^-13 of the largest entry.
# Entries of Aqk are sums with cancellation: their error is that fraction of what the terms can add up to, scale |q| |k| = 128^-0.5.
TOL = 2.0 ** -13


def _call(lens, q, k, v, g, be, scalar):
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    lay = get_layout(1, sum(lens), cu, q.device)
    rq, rk = ops.l2norm_rstd(q), ops.l2norm_rstd(k)
    t = ops.intra_fwd(lay, q, k, v, rq, rk, g, be, 128 ** -0.5, HK, HV, scalar)
    TT = sum(lens)
    un = [unpack_quarter_tiles(t[0], lay, TT), unpack_quarter_tiles(t[1], lay, TT), unpack_chunk_tiles(t[2], lay, TT), unpack_chunk_tiles(t[3], lay, TT),
          unpack_row_tiles(t[4], lay, TT), unpack_row_tiles(t[5], lay, TT)]
    return lay, t, un


@pytest.mark.parametrize("scalar", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_rows_have_no_error_in_common(dtype, scalar):
    """Sequences of one token: u = beta v, nw = -beta (k 2^g).  Each of their 128 values is rounded twice (as an operand and as a result) to 16
    mantissa bits, 2^-17 at most: the part of the error that a row has in common is an average of 128 such, 2^-16 / 128^0.5 (root mean square over
    the rows, at most).  A beta that is itself rounded to 16 bits moves the whole row, and the norm behind it passes that on to dh0."""
    T, gen = 1200, torch.Generator(device="cuda").manual_seed(11)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")                        # noqa: E731
    q, k, v = r(1, T, HK, 128).to(dtype), r(1, T, HK, 128).to(dtype), r(1, T, HV, 128).to(dtype)
    be, g = torch.rand(T, HV, generator=gen, device="cuda"), -torch.rand(T, HV, *(() if scalar else (128,)), generator=gen, device="cuda")
    got = _call((1,) * T, q, k, v, g, be, scalar)[2]
    kn = k[0].double() * torch.rsqrt((k[0].double() ** 2).sum(-1, keepdim=True) + 1e-6)
    gd = g.double() if not scalar else g.double()[..., None]
    for x, y in ((got[2], -kn.repeat_interleave(HV // HK, 1) * torch.exp2(gd) * be[..., None]), (got[3], v[0].double() * be[..., None])):
        common = (x.double() * y).sum(-1) / (y * y).sum(-1) - 1
        assert common.square().mean().sqrt().item() <= 2.0 ** -16 / 128 ** 0.5


@pytest.mark.parametrize("scalar", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_ragged_chunks(dtype, scalar):
    T, gen = sum(LENS), torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")                        # noqa: E731
    q, k, v, be = r(1, T, HK, 128).to(dtype), r(1, T, HK, 128).to(dtype), r(1, T, HV, 128).to(dtype), 2 * torch.rand(T, HV, generator=gen, device="cuda")
    step = -torch.rand(T, HV, *(() if scalar else (128,)), generator=gen, device="cuda")
    g, at = torch.empty_like(step), 0
    chunks = []
    for n in LENS:
        for c in range(0, n, 64):
            chunks.append((at + c, min(64, n - c)))
            g[at + c:at + min(c + 64, n)] = step[at + c:at + min(c + 64, n)].cumsum(0)
        at += n
    lay, raw, got = _call(LENS, q, k, v, g, be, scalar)
    # the chunk algebra in fp64
    qn, kn = (x.double() * torch.rsqrt((x.double() ** 2).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    gd = g.double() if not scalar else g.double()[..., None].expand(T, HV, 128)
    for s, n in chunks:
        for h in range(HV):
            K, Q, V, G, b = kn[0, s:s + n, h // 2], qn[0, s:s + n, h // 2] * 128 ** -0.5, v[0, s:s + n, h].double(), gd[s:s + n, h], be[s:s + n, h].double()
            E = torch.exp2((G[:, None] - G[None]).clamp(max=0.))
            gam, aqk = torch.einsum("ic,jc,ijc->ij", K, K, E), torch.einsum("ic,jc,ijc->ij", Q, K, E).tril()
            A = torch.linalg.inv(torch.eye(n, device="cuda", dtype=torch.float64) + (b[:, None] * gam).tril(-1))
            up = torch.exp2(G)
            ref = [A, aqk, -A @ (b[:, None] * K * up), A @ (b[:, None] * V), K * torch.exp2(G[-1] - G), Q * up]
            for i, (x, y) in enumerate(zip(got, ref)):
                x = x[s:s + n, h, :n] if i < 2 else x[s:s + n, h]
                err, top = (x.double() - y).abs().max().item(), max(y.abs().max().item(), 128 ** -0.5 if i == 1 else 0.0)
                assert err <= TOL * top, (i, s, n, h, err, top)
    # many items, every second copy full of infinities
    rep = lambda x, d: torch.cat([x] * TIMES, d).contiguous()                           # noqa: E731
    Q, K, V = rep(q, 1), rep(k, 1), rep(v, 1)
    for c in range(1, TIMES, 2):
        for x in (Q, K, V):
            x[:, c * T:(c + 1) * T] = float("inf")
    lay2, raw2, _ = _call(LENS * TIMES, Q, K, V, rep(g, 0), rep(be, 0), scalar)
    assert lay2.NC == TIMES * lay.NC and lay2.NC * HV > 4 * 148
    for x, y in zip(raw, raw2):
        x, y = x.view(torch.int32), y.view(torch.int32).view(TIMES, *x.shape)
        for c in range(0, TIMES, 2):
            assert torch.equal(y[c], x)


@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("mode,x_dtype", [("eda", torch.float32), ("kimi", torch.bfloat16), ("gdn", torch.float16), ("precomputed", torch.float32)])
@pytest.mark.parametrize("dtype,scalar", [(torch.bfloat16, False), (torch.float16, False), (torch.float32, False), (torch.bfloat16, True), (torch.float32, True)])
def test_gate_in_the_kernel(dtype, scalar, mode, x_dtype, keep):
    """mkda_gate_intra_fwd gives the bits of mkda_gate_cumsum_fwd and mkda_intra_fwd, whether or not it leaves behind what a backward pass reads."""
    import ctypes
    from mogankda_b200 import _lib
    T, gen = sum(LENS), torch.Generator(device="cuda").manual_seed(7)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")                        # noqa: E731
    q, k, v, b = r(1, T, HK, 128).to(dtype), r(1, T, HK, 128).to(dtype), r(1, T, HV, 128).to(dtype), r(1, T, HV).to(x_dtype)
    x = r(1, T, HV, *(() if scalar else (128,)))
    x = (-x.abs() if mode == "precomputed" else x).to(x_dtype)
    A_log, bias = (None, None) if mode == "precomputed" else (0.1 * r(HV), 0.1 * r(*(x.shape[2:])).reshape(-1))
    cu = torch.tensor([0, *torch.tensor(LENS).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    lay = get_layout(1, T, cu, q.device)
    g_c, be = ops.gate_cumsum_fwd(lay, x, mode, A_log, bias, -5.0, HV, beta_raw=b, beta_sigmoid=True, beta_scale=2.0)
    want = ops.intra_fwd(lay, q, k, v, ops.l2norm_rstd(q), ops.l2norm_rstd(k), g_c, be, 128 ** -0.5, HK, HV, scalar)
    got = [torch.full_like(t, float("nan")) for t in want]
    g_out, b_out = torch.full_like(g_c, float("nan")), torch.full_like(be, float("nan"))
    rq, rk = ops.l2norm_rstd(q), ops.l2norm_rstd(k)
    g, p = _lib.STRUCTS["MkdaGateFwd"](), _lib.STRUCTS["MkdaIntraFwd"]()
    g.x, g.x_dtype, g.scalar_gate, g.mode, g.lower_bound = ops._ptr(x), ops._dt(x), int(scalar), ops.GATE_MODES[mode], -5.0
    g.A_log, g.dt_bias = ops._ptr(A_log), ops._ptr(bias)
    g.beta_raw, g.beta_dtype, g.beta_sigmoid, g.beta_scale = ops._ptr(b), ops._dt(b), 1, 2.0
    p.L = ops._layout_struct(lay, HK, HV)
    p.q, p.k, p.v, p.qkv_dtype, p.q_rstd, p.k_rstd = ops._ptr(q), ops._ptr(k), ops._ptr(v), ops._dt(q), ops._ptr(rq), ops._ptr(rk)
    p.scale, p.scalar_gate = 128 ** -0.5, int(scalar)
    p.Aqk, p.nw, p.u, p.kbar, p.qs, p.gl = (ops._ptr(t) for t in got[1:])
    if keep:
        p.A, g.g_c, g.beta_out = ops._ptr(got[0]), ops._ptr(g_out), ops._ptr(b_out)
    assert _lib.load().mkda_gate_intra_fwd(ctypes.byref(g), ctypes.byref(p), ops._stream()) == 0
    for a, c in zip((*got[not keep:], *((g_out, b_out) if keep else ())), (*want[not keep:], *((g_c, be) if keep else ()))):
        assert torch.equal(a.view(torch.int32), c.view(torch.int32))
    if not keep:
        assert g_out.isnan().all() and b_out.isnan().all() and got[0].isnan().all()
