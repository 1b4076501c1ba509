"""Gate kernels of the wrappers over the whole range of the activation (tiny steps to the linear branch, padding values,
infinities), on pointers that do not allow wide accesses, and with the gradient written in BF16, against FP64.  Softplus and
sigmoid carry about four FP32 roundings and the sums 64 terms: 2e-6 of the result."""
import math

import pytest
import torch

from gpu_util import nrmse
from rewy_b200 import elementwise as ew

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("offset", (0, 1))
@pytest.mark.parametrize("dtype", (torch.float32, torch.bfloat16))
def test_gate_activation_over_its_range(dtype, offset):
    B, T, H = 2, 128, 3
    gen = torch.Generator(device=DEV).manual_seed(4)
    flat = torch.empty(B * T * H * 128 + offset, device=DEV).uniform_(-30, 30, generator=gen).to(dtype)
    x = flat[offset:].view(B, T, H, 128)                                   # offset 1: two (four) bytes off an aligned address
    x[0, 0, 0, :4] = torch.tensor([-1e4, 1e4, -math.inf, 88.0], device=DEV).to(dtype)
    A_log = torch.randn(H, generator=gen, device=DEV)
    bias = torch.randn(H * 128, generator=gen, device=DEV)
    dg = torch.randn(B, T, H, 128, generator=gen, device=DEV)
    a = -A_log.double().exp().view(H, 1)
    arg = x.double() + bias.double().view(H, 128)
    act = a * torch.nn.functional.softplus(arg, threshold=40.0)
    want = act.view(B, T // 64, 64, H, 128).cumsum(2).view(B, T, H, 128) / math.log(2)
    assert nrmse(want, ew.gate_cumsum_fwd(x, A_log, bias)) < 2e-6
    small = arg.clamp(max=-8.0)                                             # steps of 1e-4 and less keep their relative precision
    got = ew.gate_cumsum_fwd((small - bias.double().view(H, 128)).float(), A_log, bias)
    ref = (a * torch.nn.functional.softplus(small)).view(B, T // 64, 64, H, 128).cumsum(2).view(B, T, H, 128) / math.log(2)
    assert nrmse(ref, got) < 2e-5                                           # the argument itself is rounded: 8 * 2^-23 and more
    ref = a * dg.double() * torch.sigmoid(arg)
    dx, dA, db = ew.gate_act_bwd(x, A_log, bias, dg)
    assert dx.dtype == torch.float32 and nrmse(ref, dx) < 2e-6
    assert nrmse((dg.double() * act).sum((0, 1, 3)), dA) < 2e-5 and nrmse(ref.sum((0, 1)).view(-1), db) < 2e-5
    half = ew.gate_act_bwd(x, A_log, bias, dg, torch.bfloat16)[0]
    assert torch.equal(half, dx.to(torch.bfloat16))
