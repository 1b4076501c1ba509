"""Per-channel gates whose span over a chunk lies on either side of the limit of the centred factors (200 log2 units):
forward and backward against the FP64 oracle, and which path the chunk kernel took.  The tolerance is that of every other
gradient (2e-3): a wider span changes the exponents of the operands, not their relative precision."""
import pytest
import torch

from gpu_util import forward_saved, nrmse, oracle_backward
from rewy_b200 import _capi
from rewy_b200 import backward as bw
from rewy_b200.synthetic import make_inputs, operator_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("op", ("kda", "gdn2"))
@pytest.mark.parametrize("span,rising,wide", [(79.0, False, False), (140.0, False, False), (199.0, False, False),
                                              (201.0, False, True), (160.0, True, False)])
def test_gate_spans_around_the_centred_limit(op, span, rising, wide):
    xs = make_inputs(op, 1, 192, 3, seed=9, device=DEV, gate_scale=0.1)
    # chunk 1 of head 1: channels 0..39 decay evenly so that rows 0 and 63 of the chunk differ by `span`
    xs["g"][:, 64:128, 1, :40] = -span / 63 * 0.6931471805599453
    if rising:   # up by a few units in the middle of the decay: kept entries above 1
        xs["g"][:, 96, 1, :40] = 3.0
    sv = forward_saved(op, xs)
    g = sv["g_cumsum"][:, 64:128, 1]
    assert bool((g.amax(1) - g.amin(1)).max() >= 200.0) == wide
    from oracle import chunk_forward as oracle_forward
    fwd = oracle_forward(op, {n: (t.detach().cpu() if t is not None else None) for n, t in operator_inputs(op, xs).items()})
    errs = {n: nrmse(fwd[n].to(sv[n].dtype), sv[n]) for n in ("Aqk", "Akk", "o", "final_state")}
    assert all(e <= (3e-3 if n in ("Aqk", "Akk") else 6e-3) for n, e in errs.items()), errs   # as for every other forward
    ref = oracle_backward(op, xs, sv)
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
    count = _capi.load().rewy_wide_chunk_count(_capi.ptr(ws), _capi.current_stream(torch.device(DEV)))
    assert count == int(wide)
    errs = {n: nrmse(ref[n].to(t.dtype), t) for n, t in out.items()}
    assert all(e <= 2e-3 for e in errs.values()), errs
