"""apply_rope with positions from the host (in the launch's parameters up to 512, copied beyond) and from the device: the
same bits."""
import pytest
import torch

import mlx_flashattention_steel_b200 as fa

from .util import randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 3, 512, 513])
@pytest.mark.parametrize("interleaved", [False, True])
def test_positions_from_host_and_device_agree(dev, B, interleaved):
    x = randn((B, 2, 3, 64), torch.bfloat16, 960).to(dev).requires_grad_(True)
    ang = torch.rand((700, 32), device=dev) * 6.28
    pos = [(37 * b) % 697 for b in range(B)]
    do = randn((B, 2, 3, 64), torch.bfloat16, 961).to(dev)

    def run(offset):
        out = fa.apply_rope(x, ang.cos(), ang.sin(), offset, interleaved=interleaved)
        return out, torch.autograd.grad(out, x, do)[0]

    ref = run(torch.tensor(pos, dtype=torch.int32, device=dev))
    for offset in (pos, tuple(pos), torch.tensor(pos)):
        got = run(offset)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


def test_positions_from_the_host_are_checked(dev):
    x = randn((2, 2, 3, 64), torch.float16, 962).to(dev)
    cos, sin = torch.ones((10, 32), device=dev), torch.zeros((10, 32), device=dev)
    for bad in ([0, 8], [-1, 0], [0], [0, 1, 2]):
        with pytest.raises(ValueError):
            fa.apply_rope(x, cos, sin, bad, interleaved=False)
