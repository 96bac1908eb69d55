"""Packed rows that belong to no sequence: no gradient, whatever the memory held before."""
import pytest
import torch

import mlx_flashattention_steel_b200 as fa
from mlx_flashattention_steel_b200 import _lib
from mlx_flashattention_steel_b200 import attention as A

from .util import randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, _lib.FLAG_FORCE_MMA_SYNC])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Tq,Tk,cu_q,cu_k", [(200, 200, [0, 70, 130], [0, 70, 130]), (150, 400, [5, 70, 140], [9, 100, 390]),
                                             (300, 90, [0, 1, 300], [40, 41, 90]), (64, 64, [0, 32, 64], [0, 32, 64])])
def test_gradients_of_rows_of_no_sequence(dev, Tq, Tk, cu_q, cu_k, D, flags):
    q, k, v, do = (randn((1, h, n, D), torch.bfloat16, 10 + i).to(dev) for i, (h, n) in enumerate(((4, Tq), (2, Tk), (2, Tk), (4, Tq))))
    cq, ck = (torch.tensor(c, dtype=torch.int32, device=dev) for c in (cu_q, cu_k))
    old = A._set_force_flags(flags)
    try:
        t = [x.clone().requires_grad_(True) for x in (q, k, v)]
        out = fa.flash_attention_varlen(*t, cq, ck, Tq, Tk)
        junk = [torch.full_like(x, float("nan")) for x in (q, k, v) for _ in range(4)]
        del junk                                # what the gradients' memory holds
        got = torch.autograd.grad(out, t, do)
        want = [torch.zeros_like(x) for x in (q, k, v)]
        for a, b, c, d in zip(cu_q, cu_q[1:], cu_k, cu_k[1:]):
            s = [x[:, :, i:j].contiguous().requires_grad_(True) for x, i, j in ((q, a, b), (k, c, d), (v, c, d))]
            g = torch.autograd.grad(fa.flash_attention(*s), s, do[:, :, a:b].contiguous())
            for w, x, i in zip(want, g, (a, c, c)):
                w[:, :, i:i + x.shape[2]] = x
    finally:
        A._set_force_flags(old)
    for name, g, w, cu in zip(("dQ", "dK", "dV"), got, want, (cu_q, cu_k, cu_k)):
        # a packed call may cut its sums elsewhere: one step of bfloat16
        assert torch.allclose(g.double(), w.double(), rtol=2.0 ** -7, atol=2.0 ** -8), name
        assert not g[:, :, :cu[0]].any() and not g[:, :, cu[-1]:].any(), name
