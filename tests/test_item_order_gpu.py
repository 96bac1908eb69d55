"""Work dealt out in another order than one head after the other: causal calls whose heads form several groups (the last
one smaller).  Every item has to be done exactly once: against the oracle."""
import pytest
import torch

import mlx_flashattention_steel_b200 as fa
from oracle import sdpa_oracle as orc

from .util import LSE_TOL, assert_close, assert_close_grad, randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,N,S,D", [(7, 7, 300, 32768, 128), (7, 7, 32768, 300, 128), (14, 7, 20000, 333, 64), (16, 2, 900, 700, 128)])
def test_several_groups_of_heads(dev, Hq, Hkv, N, S, D):
    """48 MB a group: 3 heads of 32768 x 128 K / V (or Q / dO), 9 of 20000 x 64, all of the small ones."""
    dtype = torch.bfloat16
    q, k, v, do = (randn((1, h, n, D), dtype, 900 + i) for i, (h, n) in enumerate(((Hq, N), (Hkv, S), (Hkv, S), (Hq, N))))
    qg, kg, vg = (x.to(dev).requires_grad_(True) for x in (q, k, v))
    out, lse = fa.flash_attention(qg, kg, vg, causal=True, return_lse=True)
    out.backward(do.to(dev))
    O, L, _ = orc.sdpa(q, k, v, causal=True)
    assert_close(out, O, dtype)
    assert_close(lse, L, dtype, "lse", LSE_TOL[dtype])
    for name, got, ref in zip(("dQ", "dK", "dV"), (qg.grad, kg.grad, vg.grad), orc.backward(q, k, v, do, causal=True)):
        assert_close_grad(got, ref, dtype, name)
