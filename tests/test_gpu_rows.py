"""Row kernels around the operators (padding, cut, q/k front pass) against the same steps in torch: fixed batches and
packed sequences, row sizes down to two bytes, an unaligned input, grouped heads, with and without normalisation."""
import pytest
import torch

from gpu_util import nrmse
from rewy_b200 import elementwise as ew
from rewy_b200.functions import _Ragged

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SHAPES = [(1, 1, None), (3, 100, None), (2, 128, None), (1, 167, (37, 64, 66)), (1, 300, (1, 235, 64))]


def _ragged(T, lengths):
    cu = None if lengths is None else torch.cat([torch.zeros(1, dtype=torch.int64), torch.tensor(lengths).cumsum(0)])
    return _Ragged(T, DEV, cu)


@pytest.mark.parametrize("B,T,lengths", SHAPES)
def test_pad_and_cut_equal_the_tensor_operations(B, T, lengths):
    rg = _ragged(T, lengths)
    gen = torch.Generator(device=DEV).manual_seed(1)
    rn = lambda *s, dtype=torch.bfloat16: torch.randn(*s, generator=gen, device=DEV).to(dtype)
    wide = rn(B * T * 128 + 1)[1:].view(B, T, 1, 128)                      # rows start two bytes off an aligned address
    xs = [rn(B, T, 3, 128), rn(B, T, 1), rn(B, T, 3, dtype=torch.float32), rn(B, T, 5, dtype=torch.float16), wide,
          rn(B, T, 2, 4, dtype=torch.float64)]
    fills = [0.0, 0.0, -1e4, 2.0, 0.0, 1.5]
    got = rg.pad_rows(*zip(xs, fills))
    for x, f, y in zip(xs, fills, got):
        assert torch.equal(y, rg.pad(x, f)), x.dtype
    for x, y in zip(xs, rg.cut_rows(*got)):
        assert torch.equal(x, y), x.dtype


@pytest.mark.parametrize("dy_dtype", (torch.float32, torch.bfloat16))
@pytest.mark.parametrize("normalize", (True, False))
@pytest.mark.parametrize("groups", (1, 2, 3))
@pytest.mark.parametrize("B,T,lengths", SHAPES)
def test_qk_front_equals_its_steps(B, T, lengths, groups, normalize, dy_dtype):
    """Forward: bit for bit the library's l2norm on the padded rows, then repeat_interleave.  Backward: without groups bit for
    bit its backward (without normalisation one rounding), else the group sum and the normalisation backward in FP32 with one
    BF16 rounding (2^-9 of a value: 4e-3 covers it with the sum's own rounding)."""
    rg, H = _ragged(T, lengths), 3
    gen = torch.Generator(device=DEV).manual_seed(2)
    q, k = (torch.randn(B, T, H, 128, generator=gen, device=DEV).to(torch.bfloat16) for _ in range(2))
    yq, yk, rq, rk = ew.qk_front_fwd(q, k, rg.row_map(B), groups, normalize)
    for x, y, r in ((q, yq, rq), (k, yk, rk)):
        want = rg.pad(x)
        if normalize:
            want, rstd = ew.l2norm_fwd(want)
            assert torch.equal(rstd, r)
        assert torch.equal(want.repeat_interleave(groups, 2), y)
    dyq, dyk = (torch.randn(yq.shape, generator=gen, device=DEV).to(dy_dtype) for _ in range(2))
    for x, y, r, dy, dx in zip((q, k), (yq, yk), (rq, rk), (dyq, dyk),
                               ew.qk_front_bwd(yq, yk, rq, rk, dyq, dyk, rg.row_map(B), groups)):
        g = dy.double().view(B, rg.total, H, groups, 128).sum(3)
        if normalize:
            yd = y[:, :, ::groups].double()
            g = (g - yd * (g * yd).sum(-1, keepdim=True)) * r.double()[..., None]
        assert dx.shape == x.shape and dx.dtype == torch.bfloat16
        assert nrmse(rg.cut(g), dx) <= 4e-3
        if groups == 1:
            assert torch.equal(rg.cut(ew.l2norm_bwd(y, r, dy) if normalize else dy.to(torch.bfloat16)), dx)


def test_saved_tensor_hooks_may_change_the_layout():
    """Hooks that hand every saved tensor back head-first in memory: the gradients are those without hooks."""
    import rewy_b200 as fdr
    gen = torch.Generator(device=DEV).manual_seed(5)
    rn = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    xs = dict(q=rn(2, 100, 3, 128).bfloat16(), k=rn(2, 100, 3, 128).bfloat16(), v=rn(2, 100, 6, 128).bfloat16(),
              beta=torch.sigmoid(rn(2, 100, 6)).bfloat16())
    xs = {n: x.requires_grad_() for n, x in xs.items()}
    do = rn(2, 100, 6, 128).bfloat16()
    head_first = lambda t: t.transpose(1, 2).contiguous().transpose(1, 2) if t.ndim >= 3 else t

    def grads(unpack):
        with fdr.use_backend("optimized"), torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            o, _ = fdr.chunk_delta_rule(**xs, use_qk_l2norm_in_kernel=True)
            return torch.autograd.grad(o, tuple(xs.values()), do)

    for n, a, b in zip(xs, grads(lambda t: t), grads(head_first)):
        assert torch.equal(a, b), n


@pytest.mark.parametrize("name,T,lengths,groups", [("chunk_kda", 167, (100, 67), 1), ("chunk_kda", 100, None, 1),
                                                   ("chunk_gated_delta_rule", 128, None, 2), ("chunk_delta_rule", 167, (100, 67), 2)])
def test_second_derivatives_raise_through_the_row_kernels(name, T, lengths, groups):
    """A gradient taken with create_graph cannot be differentiated again: it raises and is never silently a constant."""
    import rewy_b200 as fdr
    gen, H = torch.Generator(device=DEV).manual_seed(4), 2
    rn = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    xs = dict(q=rn(1, T, H, 128).bfloat16(), k=torch.nn.functional.normalize(rn(1, T, H, 128), dim=-1).bfloat16(),
              v=rn(1, T, H * groups, 128).bfloat16(), beta=torch.sigmoid(rn(1, T, H * groups)).bfloat16())
    if name != "chunk_delta_rule":
        xs["g"] = -0.1 * torch.rand((1, T, H * groups) + ((128,) if name == "chunk_kda" else ()), generator=gen, device=DEV)
    xs = {n: x.requires_grad_() for n, x in xs.items()}
    cu = {} if lengths is None else dict(cu_seqlens=torch.tensor([0, lengths[0], T], device=DEV))
    with fdr.use_backend("optimized"):
        o, _ = getattr(fdr, name)(**xs, **cu)
    for loss in (o.float().sum(), o.float().pow(2).sum()):
        plain = torch.autograd.grad(loss, tuple(xs.values()), retain_graph=True)
        again = torch.autograd.grad(loss, tuple(xs.values()), create_graph=True)
        for n, a, b in zip(xs, plain, again):
            assert torch.equal(a, b), n
            with pytest.raises(RuntimeError, match="derivative for rewy_b200::family_bwd is not implemented"):
                torch.autograd.grad(b.float().sum(), tuple(xs.values()), retain_graph=True, allow_unused=True)
