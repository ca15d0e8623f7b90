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
    """dbeta is (dW Vd^T)_ii / beta_i; a chunk that holds a beta below 1e-12 forms it from v, k and the state instead.  Chunks without
    such a row, with one, with all rows zero, and a ragged last chunk."""
    lv, do, dht, opts, _ = make_inputs(B=2, T=64 * 3 + 21, HK=2, HV=4, dtype=dtype, gate="precomputed", scalar=scalar, beta="precomputed",
                                       epi=None, seed=41)
    lv["beta"][0, 70] = 0.0
    lv["beta"][0, 71] = 1e-13
    lv["beta"][1, 64:128] = 0.0
    lv["beta"][1, 64 * 3 + 20, 1] = 0.0
    compare(run(mk.chunk_delta_rule, lv, do, dht, opts, None),
            run(orc.chunked_delta_rule, lv, do, dht, opts, None, f64=True))
