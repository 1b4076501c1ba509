"""Per-channel gates whose span over a chunk lies on either side of the limit of the centred factors (200 log2 units):
forward and backward against the FP64 oracle, and which path the chunk kernel took.  The tolerance is that of every other
gradient (2e-3): a wider span changes the exponents of the operands, not their relative precision.  What keeps it so: the
gradient matrices are scaled per chunk (gradients of any size), and q or k of extreme size go to the pairwise sums."""
import pytest
import torch

from gpu_util import forward_saved, nrmse, oracle_backward
from rewy_b200 import _capi
from rewy_b200 import backward as bw
from rewy_b200.synthetic import make_inputs, operator_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(op, span, rising=False):
    xs = make_inputs(op, 1, 192, 3, seed=9, device=DEV, gate_scale=0.1)
    # chunk 1 of head 1: channels 0..39 decay evenly so that rows 0 and 63 of the chunk differ by `span`
    xs["g"][:, 64:128, 1, :40] = -span / 63 * 0.6931471805599453
    if rising:   # up by a few units in the middle of the decay: kept entries above 1
        xs["g"][:, 96, 1, :40] = 3.0
    return xs


def _forward_errors(op, xs, sv):
    from oracle import chunk_forward as oracle_forward
    fwd = oracle_forward(op, {n: (t.detach().cpu() if t is not None else None) for n, t in operator_inputs(op, xs).items()})
    return {n: nrmse(fwd[n].to(sv[n].dtype), sv[n]) for n in ("Aqk", "Akk", "o", "final_state")}


def _backward(op, xs, sv):
    """(gradients, number of chunks that went to the pairwise sums)"""
    ws = torch.empty(_capi.workspace_bytes(_capi.FAMILY_ID[op], _capi.SAVED, 1, 192, 3), dtype=torch.uint8, device=DEV)
    common = dict(q=xs["q"], k=xs["k"], v=xs["v"], scale=128 ** -0.5, initial_state=xs["initial_state"], do=xs["do"],
                  dht=xs["dht"], Aqk=sv["Aqk"], Akk=sv["Akk"], g=sv["g_cumsum"], disable_recompute=True, qg=sv["qg"],
                  kg=sv["kg"], v_new=sv["v_new"], h=sv["h"], out_dtype=torch.float32, workspace=ws, check_status=True)
    if op == "kda":
        r = bw.kda_backward(beta=xs["beta"], w=sv["w"], u=sv["u"], **common)
        out = dict(zip(("dq", "dk", "dv", "dbeta", "dg", "dh0"), r))
    else:
        r = bw.gdn2_backward(b=xs["b"], w_gate=xs["w"], w_wy=sv["w"], u_wy=sv["u"], **common)
        out = dict(zip(("dq", "dk", "dv", "db", "dw", "dg", "dh0"), r))
    return out, _capi.load().rewy_wide_chunk_count(_capi.ptr(ws), _capi.current_stream(torch.device(DEV)))


@pytest.mark.parametrize("op", ("kda", "gdn2"))
@pytest.mark.parametrize("span,rising,wide", [(79.0, False, False), (140.0, False, False), (199.0, False, False),
                                              (201.0, False, True), (160.0, True, False)])
def test_gate_spans_around_the_centred_limit(op, span, rising, wide):
    xs = _inputs(op, span, rising)
    sv = forward_saved(op, xs)
    g = sv["g_cumsum"][:, 64:128, 1]
    assert bool((g.amax(1) - g.amin(1)).max() >= 200.0) == wide
    errs = _forward_errors(op, xs, sv)
    assert all(e <= (3e-3 if n in ("Aqk", "Akk") else 6e-3) for n, e in errs.items()), errs   # as for every other forward
    ref = oracle_backward(op, xs, sv)
    out, count = _backward(op, xs, sv)
    assert count == int(wide)
    errs = {n: nrmse(ref[n].to(t.dtype), t) for n, t in out.items()}
    assert all(e <= 2e-3 for e in errs.values()), errs


@pytest.mark.parametrize("op", ("kda", "gdn2"))
@pytest.mark.parametrize("span,rising", [(79.0, False), (199.0, False), (160.0, True)])
def test_gradients_of_any_size_scale_with_the_output_gradient(op, span, rising):
    """The backward is linear in do and dht: scaled by a power of two they scale every gradient by it.  2^-50 .. 2^40, beyond
    what a mean over many tokens or a loss scale does; 1e-6 leaves room for single subnormal entries."""
    xs = _inputs(op, span, rising)
    sv = forward_saved(op, xs)
    base, _ = _backward(op, xs, sv)
    for power in (-50, -40, -30, 20, 40):
        f = 2.0 ** power
        out, count = _backward(op, dict(xs, do=xs["do"] * f, dht=xs["dht"] * f), sv)
        assert count == 0
        errs = {n: nrmse(base[n].double() * f, t) for n, t in out.items()}
        assert all(e <= 1e-6 for e in errs.values()), (power, errs)


@pytest.mark.parametrize("op", ("kda", "gdn2"))
def test_a_chunk_without_state_or_value_gradient_stays_finite(op):
    """Without state and values both gradient matrices are zero in the far chunk and nothing may be scaled by their size; with
    2^-40 of them they are tiny while do is not."""
    for v in (0.0, 2.0 ** -40):
        xs = _inputs(op, 199.0)
        xs["v"] = xs["v"] * v
        xs["initial_state"] = xs["initial_state"] * v
        sv = forward_saved(op, xs)
        ref = oracle_backward(op, xs, sv)
        out, _ = _backward(op, xs, sv)
        assert all(torch.isfinite(t).all() for t in out.values())
        errs = {n: nrmse(ref[n], t) for n, t in out.items() if ref[n].norm() > 0}
        assert all(e <= (2e-3 if n != "dv" else 4e-3) for n, e in errs.items()), (v, errs)


@pytest.mark.parametrize("op", ("kda", "gdn2"))
@pytest.mark.parametrize("q,k,wide", [(-30, -30, True), (-30, 0, True), (0, -30, True), (30, 0, True), (-16, -12, False)])
def test_far_chunks_with_q_or_k_of_extreme_size_are_summed_pairwise(op, q, k, wide):
    """q or k times 2^-30 or 2^30 on top of factors of 2^-100 and 2^100 would leave BF16's range; within 2^-20 .. 2^20 (largest
    entries here 2^-17 and 2^-13) the centred products keep their precision."""
    xs = _inputs(op, 199.0)
    xs["q"], xs["k"] = xs["q"] * 2.0 ** q, xs["k"] * 2.0 ** k
    sv = forward_saved(op, xs)
    errs = _forward_errors(op, xs, sv)
    assert all(e <= (3e-3 if n in ("Aqk", "Akk") else 6e-3) for n, e in errs.items()), errs
    one = _forward_errors_of_far_chunk(op, xs, sv)
    assert one <= 3e-3, one
    ref = oracle_backward(op, xs, sv)
    out, count = _backward(op, xs, sv)
    assert count == int(wide)
    errs = {n: nrmse(ref[n].to(t.dtype), t) for n, t in out.items()}
    assert all(e <= 2e-3 for e in errs.values()), errs


def _forward_errors_of_far_chunk(op, xs, sv):
    from oracle import chunk_forward as oracle_forward
    fwd = oracle_forward(op, {n: (t.detach().cpu() if t is not None else None) for n, t in operator_inputs(op, xs).items()})
    return nrmse(fwd["Aqk"].to(torch.bfloat16)[:, 64:128, 1], sv["Aqk"][:, 64:128, 1])
