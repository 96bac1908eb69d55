"""Backward calls with few (key tile, kv head) items, which the tcgen05 kernels cut into 2, 4 or 8 parts and sum: every
option of the kernels, rows and keys that are no multiple of a tile, keys that no query sees, parts without a step."""
import pytest
import torch

import mlx_flashattention_steel_b200 as fa
from oracle import sdpa_oracle as orc

from .util import assert_close_grad, randn

pytestmark = pytest.mark.gpu


def _run(dev, dtype, B, Hq, Hkv, N, S, D, seed, causal=True, softcap=0.0, window=None):
    q, k, v, do = (randn((B, h, n, D), dtype, seed + i) for i, (h, n) in enumerate(((Hq, N), (Hkv, S), (Hkv, S), (Hq, N))))
    qg, kg, vg = (x.to(dev).requires_grad_(True) for x in (q, k, v))
    out = fa.flash_attention(qg, kg, vg, causal=causal, softcap=softcap, window_size=None if window is None else (window, 0))
    grads = torch.autograd.grad(out, (qg, kg, vg), do.to(dev), retain_graph=True)
    # rows above the diagonal of the first key see nothing: no gradient, and the oracle's softmax of them is 0 / 0
    blind = max(0, N - S) if causal else 0
    refs = orc.backward(q[:, :, blind:], k, v, do[:, :, blind:], causal=causal, softcap=softcap, window_left=-1 if window is None else window)
    assert not grads[0][:, :, :blind].any()
    got_q = grads[0][:, :, blind:]
    for name, got, ref in zip(("dQ", "dK", "dV"), (got_q, grads[1], grads[2]), refs):
        assert_close_grad(got, ref, dtype, name)
    # the parts are summed in a fixed order
    again = torch.autograd.grad(out, (qg, kg, vg), do.to(dev))
    assert torch.equal(grads[1], again[1]) and torch.equal(grads[2], again[2])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,N,S,causal", [(1, 4, 2, 1100, 700, False), (2, 4, 1, 1100, 1100, True), (1, 8, 2, 2100, 130, True),
                                                 (1, 2, 2, 1200, 1900, True), (1, 6, 2, 700, 64, False)])
def test_parts(dev, dtype, D, B, Hq, Hkv, N, S, causal):
    _run(dev, dtype, B, Hq, Hkv, N, S, D, 930, causal=causal)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("softcap,window", [(30.0, None), (0.0, 600), (20.0, 300)])
def test_parts_with_cap_and_window(dev, D, softcap, window):
    _run(dev, torch.bfloat16, 1, 8, 1, 1500, 1500, D, 940, softcap=softcap, window=window)


@pytest.mark.parametrize("D", [64, 128])
def test_parts_with_a_block_mask(dev, D):
    N, dtype = 1200, torch.float16
    q, k, v, do = (randn((1, h, N, D), dtype, 950 + i) for i, h in enumerate((4, 2, 2, 4)))
    mask = fa.make_sliding_window_mask(N, 500, D, causal=True)
    qg, kg, vg = (x.to(dev).requires_grad_(True) for x in (q, k, v))
    out = fa.flash_attention_sparse(qg, kg, vg, mask.to(dev), causal=True)
    out.backward(do.to(dev))
    cells = mask.repeat_interleave(32, 0)[:N].repeat_interleave(32 if D == 64 else 16, 1)[:, :N]
    visible = cells & (torch.arange(N)[:, None] >= torch.arange(N)[None, :])
    qd, kd, vd = (x.double().requires_grad_(True) for x in (q, k, v))
    s = (qd @ kd.repeat_interleave(2, 1).transpose(-1, -2) * D ** -0.5).masked_fill(~visible, float("-inf"))
    (torch.softmax(s, -1) @ vd.repeat_interleave(2, 1)).backward(do.double())
    for name, got, ref in zip(("dQ", "dK", "dV"), (qg.grad, kg.grad, vg.grad), (qd.grad, kd.grad, vd.grad)):
        assert_close_grad(got, ref, dtype, name)
