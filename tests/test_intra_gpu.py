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
