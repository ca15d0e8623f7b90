"""GPU: the chunk backward over ragged chunks, with one item per CTA and with many (buffers, barriers and tensor memory reused): sequences of 1, 15, 16, 17,
33, 63, 64, 65 and 100 tokens have the same gradients, bit for bit, alone and in every copy of a batch of thirty of each.  Forward-only calls, which do
not keep A, have the outputs of the others."""
import pytest
import torch

import mogankda_b200 as mk
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
