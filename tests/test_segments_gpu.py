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
