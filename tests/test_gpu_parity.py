"""GPU parity tests: every CUDA stage and the whole-family backward, called through the C ABI, against
the FP64 CPU oracle on the same seeded inputs.

Tolerances (normalised RMSE = ||got-ref||/||ref||):
  2e-3  for every gradient of the whole-family backward against the FP64 closed-form backward fed with the
        same (BF16) saved tensors — the bound the operator is specified to — including the cases that run the exact
        pairwise path on huge gate spans; 3e-3 only where dq/dk are compared after rounding to BF16 on a tiny problem
        (the rounding floor itself is measured at the benchmark shapes in test_gpu_shapes.py);
  8e-3 / 2e-2 (gate, beta and vector-gate gradients) for the public autograd path against the FP64 token
        recurrence on the raw inputs — the reference's own acceptance limits
        (src/fast_delta_rule/validation.py:68-71).
"""
import numpy as np
import pytest
import torch

from gpu_util import (base_args, call_stage, forward_saved, nrmse, oracle_backward, stage_buffers)
from rewy_b200 import _capi
from rewy_b200.synthetic import make_inputs, operator_inputs

pytestmark = pytest.mark.gpu

OPS = ("kda", "gdn2", "gdn", "delta")
DEV = "cuda:0"
TOL = 2e-3


def _inputs(op, B=1, T=256, H=2, seed=42, **kw):
    kw.setdefault("gate_scale", 0.1 if op != "gdn" else 1.0)
    kw.setdefault("gate", "softplus" if op != "gdn" else "head_exp")
    return make_inputs(op, B, T, H, seed=seed, device=DEV, **kw)


def _report(errs, tol):
    print("NRMSE", {n: float(f"{e:.3g}") for n, e in errs.items()}, "limit", tol)
    bad = {n: e for n, e in errs.items() if not (e <= (tol[n] if isinstance(tol, dict) else tol))}
    assert not bad, f"NRMSE above tolerance: {bad}; all: {errs}"


def _oracle_recompute(op, xs, saved):
    """FP64 statement of the recompute stage from the tensors the stage itself reads (BF16 q, k, v, gates, the saved
    BF16 Akk and the saved cumulative gate): w = Akk (b k gamma), u = Akk (w v), qg = q gamma, kg = k 2^(G_last - G),
    Aqk = scale tril(qg (k / gamma)^T).  Follows the oracle's chunked forward (oracle/chunked.py, chunk_forward)."""
    from oracle.chunked import _chunks, _gates, _unchunks
    f64 = torch.float64
    cpu = {n: (t.detach().cpu() if torch.is_tensor(t) else t) for n, t in xs.items()}
    cpu["g_cumsum"] = None if saved.get("g_cumsum") is None else saved["g_cumsum"].detach().cpu()
    q, k, v = (_chunks(cpu[n].to(f64), 64) for n in ("q", "k", "v"))
    G, b, w = _gates(op, cpu, 64, f64)
    gamma = torch.exp2(G)
    A = _chunks(saved["Akk"].detach().cpu().to(f64), 64)
    E, Z, Qg = b * k * gamma, w * v, q * gamma
    out = dict(w=A @ E, u=A @ Z, qg=Qg.expand_as(q), kg=(k * torch.exp2(G[..., -1:, :] - G)).expand_as(k),
               Aqk=128 ** -0.5 * torch.tril(Qg @ (k / gamma).transpose(-1, -2)))
    return {n: _unchunks(t) for n, t in out.items()}


@pytest.mark.parametrize("variant", ("tensor_core", "warp_mma"))
@pytest.mark.parametrize("op", OPS)
def test_stage_prepare(op, variant):
    """The recompute stage: the TMA + tcgen05 kernel (production) and the warp-MMA kernel (cross-check), on a problem
    with several chunks per persistent CTA slot."""
    xs = _inputs(op, B=2, T=512, H=3)
    saved = forward_saved(op, xs)
    a, keep = base_args(op, xs, saved)
    B, T, H, _ = xs["k"].shape
    mk = lambda d: torch.full((B, T, H, d), float("nan"), dtype=torch.bfloat16, device=DEV)
    w, u, qg, kg, aqk = mk(128), mk(128), mk(128), mk(128), mk(64)
    ctrl = torch.zeros(8, dtype=torch.int32, device=DEV)
    lib = _capi.load()
    try:
        assert lib.rewy_set_prepare_variant(1 if variant == "warp_mma" else 2) == 0
        before = lib.rewy_kernel_launch_count()
        call_stage("rewy_stage_prepare", a, stage_buffers(w=w, u=u, qg=qg, kg=kg, Aqk=aqk, ctrl=ctrl), DEV)
        assert lib.rewy_kernel_launch_count() == before + 1
    finally:
        lib.rewy_set_prepare_variant(0)
    assert ctrl[0].item() == 0, f"device status word {ctrl[0].item()}: a bounded wait gave up"
    # against the FP64 oracle, in the public dtype (BF16) of the stage's outputs: operands are rounded to BF16 before the
    # products (as the reference's recompute does), results once more on the way out
    ref = _oracle_recompute(op, xs, saved)
    got = dict(w=w, u=u, qg=qg, kg=kg)
    if op in ("gdn", "delta"):
        got["Aqk"] = aqk
    errs = {n: nrmse(ref[n].to(torch.bfloat16), t) for n, t in got.items()}
    print(f"prepare {op} vs FP64 oracle: {errs}")
    _report(errs, 4e-3)   # measured 2.7e-3 .. 2.9e-3 for w and u (two BF16 roundings), 0 for the elementwise outputs
    # and against the forward that produced the saved set (both sides BF16; identical up to accumulation order)
    errs = {n: nrmse(saved[n], t) for n, t in got.items()}
    _report(errs, 4e-3)


@pytest.mark.parametrize("op", OPS)
def test_stage_forward_scan(op):
    xs = _inputs(op)
    saved = forward_saved(op, xs)
    a, keep = base_args(op, xs, saved)
    h = torch.full_like(saved["h"], float("nan"))
    v_new = torch.full_like(saved["v_new"], float("nan"))
    ctrl = torch.zeros(8, dtype=torch.int32, device=DEV)
    call_stage("rewy_stage_fwd_scan", a, stage_buffers(w=saved["w"], u=saved["u"], kg=saved["kg"], h=h, v_new=v_new,
                                                       ctrl=ctrl), DEV)
    assert ctrl[0].item() == 0, f"device status word {ctrl[0].item()}: a bounded wait gave up"
    _report(dict(h=nrmse(saved["h"], h), v_new=nrmse(saved["v_new"], v_new)), 4e-3)


@pytest.mark.parametrize("op", OPS)
def test_stage_reverse_scan(op):
    xs = _inputs(op)
    saved = forward_saved(op, xs)
    ref = oracle_backward(op, xs, saved)
    a, keep = base_args(op, xs, saved)
    dh = torch.full_like(saved["h"], float("nan"))
    dR = torch.full_like(saved["v_new"], float("nan"))
    dR_lo = torch.full_like(saved["v_new"], float("nan"))
    dh0 = torch.full((xs["k"].shape[0], xs["k"].shape[2], 128, 128), float("nan"), device=DEV)
    a.dh0 = _capi.ptr(dh0)
    ctrl = torch.zeros(8, dtype=torch.int32, device=DEV)
    call_stage("rewy_stage_bwd_scan", a, stage_buffers(qg=saved["qg"], kg=saved["kg"], w=saved["w"], Aqk=saved["Aqk"],
                                                       dh=dh, dR=dR, dR_lo=dR_lo, ctrl=ctrl), DEV)
    assert ctrl[0].item() == 0, f"device status word {ctrl[0].item()}: a bounded wait gave up"
    # dh is stored in BF16 (inter-stage contract): compared in that dtype; dR is a BF16 hi/lo pair
    _report(dict(dh=nrmse(ref["dh"].to(torch.bfloat16), dh), dR=nrmse(ref["dR"], dR.float() + dR_lo.float()),
                 dh0=nrmse(ref["dh0"], dh0)), TOL)


def _split(x):
    hi = x.to(torch.bfloat16)
    return hi.to(DEV).contiguous(), (x - hi.to(x.dtype)).to(torch.bfloat16).to(DEV).contiguous()


def _run_chunk_adjoint(op, xs, saved, dh, dR, out_f32=True, passes=0, dR_lo=None):
    if dR_lo is None:
        dR_lo = torch.zeros_like(dR)
    a, keep = base_args(op, xs, saved, _capi.OUT_F32 if out_f32 else _capi.OUT_BF16, passes)
    B, T, H, _ = xs["k"].shape
    odt = torch.float32 if out_f32 else torch.bfloat16
    nan = lambda shape, dt: torch.full(shape, float("nan"), dtype=dt, device=DEV)
    out = dict(dq=nan((B, T, H, 128), odt), dk=nan((B, T, H, 128), odt), dv=nan((B, T, H, 128), torch.bfloat16))
    if op != "delta":
        out["dg"] = nan(tuple(saved["g_cumsum"].shape), torch.float32)
    if op == "gdn2":
        out["db_gate"], out["dw_gate"] = nan((B, T, H, 128), odt), nan((B, T, H, 128), odt)
    else:
        out["dbeta"] = nan((B, T, H), torch.float32)
    for n, t in out.items():
        setattr(a, n, _capi.ptr(t))
    ctrl = torch.zeros(2 + B * H * (T // 64), dtype=torch.int32, device=DEV)
    call_stage("rewy_stage_chunk_adjoint", a, stage_buffers(v_new=saved["v_new"], h=saved["h"], dh=dh, dR=dR, dR_lo=dR_lo,
                                                            ctrl=ctrl), DEV)
    assert ctrl[0].item() == 0, f"device status word {ctrl[0].item()}: a bounded wait gave up"
    return out


def _grad_errs(op, ref, out):
    """Errors in the public dtype of each output: the FP64 reference is rounded to that dtype first, as the
    reference's own regression does (scripts/npu950_intra_regression.py:66)."""
    def err(name_ref, name_out):
        got = out[name_out]
        return nrmse(ref[name_ref].to(got.dtype), got)
    errs = dict(dq=err("dq", "dq"), dk=err("dk", "dk"), dv=err("dv", "dv"))
    if op != "delta":
        errs["dg"] = err("dg", "dg")
    if op == "gdn2":
        errs["db"], errs["dw"] = err("db", "db_gate"), err("dw", "dw_gate")
    else:
        errs["dbeta"] = err("dbeta", "dbeta")
    return errs


@pytest.mark.parametrize("op", OPS)
def test_stage_chunk_adjoint(op):
    xs = _inputs(op)
    saved = forward_saved(op, xs)
    ref = oracle_backward(op, xs, saved)
    dh = ref["dh"].to(torch.bfloat16).to(DEV)
    dR, dR_lo = _split(ref["dR"])
    out = _run_chunk_adjoint(op, xs, saved, dh, dR, dR_lo=dR_lo)
    _report(_grad_errs(op, ref, out), TOL)


def _family_call(op, xs, saved, policy_saved, out_dtype=torch.float32, passes=None):
    from rewy_b200 import backward as bw
    common = dict(q=xs["q"], k=xs["k"], v=xs["v"], scale=128 ** -0.5, initial_state=xs.get("initial_state"),
                  do=xs["do"], dht=xs.get("dht"), out_dtype=out_dtype, intra_passes=passes, check_status=True)
    if op == "kda":
        r = bw.kda_backward(beta=xs["beta"], Aqk=saved["Aqk"], Akk=saved["Akk"], g=saved["g_cumsum"],
                            disable_recompute=policy_saved, w=saved["w"], u=saved["u"], qg=saved["qg"], kg=saved["kg"],
                            v_new=saved["v_new"], h=saved["h"], **common)
        return dict(dq=r[0], dk=r[1], dv=r[2], dbeta=r[3], dg=r[4], dh0=r[5])
    if op == "gdn2":
        r = bw.gdn2_backward(b=xs["b"], w_gate=xs["w"], Aqk=saved["Aqk"], Akk=saved["Akk"], g=saved["g_cumsum"],
                             disable_recompute=policy_saved, w_wy=saved["w"], u_wy=saved["u"], qg=saved["qg"],
                             kg=saved["kg"], v_new=saved["v_new"], h=saved["h"], **common)
        return dict(dq=r[0], dk=r[1], dv=r[2], db_gate=r[3], dw_gate=r[4], dg=r[5], dh0=r[6])
    if op == "gdn":
        r = bw.gdn_backward(g=saved["g_cumsum"], beta=xs["beta"], A=saved["Akk"], **common)
        return dict(dq=r[0], dk=r[1], dv=r[2], dbeta=r[3], dg=r[4], dh0=r[5])
    r = bw.delta_backward(beta=xs["beta"], A=saved["Akk"], **common)
    return dict(dq=r[0], dk=r[1], dv=r[2], dbeta=r[3], dh0=r[4])


@pytest.mark.parametrize("op,policy_saved", [("kda", True), ("kda", False), ("gdn2", True), ("gdn2", False),
                                             ("gdn", False), ("delta", False)])
def test_family_backward_matches_oracle(op, policy_saved):
    xs = _inputs(op, B=2, T=256, H=2, seed=7)
    saved = forward_saved(op, xs)
    ref = oracle_backward(op, xs, saved)
    out = _family_call(op, xs, saved, policy_saved)
    torch.cuda.synchronize()
    errs = _grad_errs(op, ref, out)
    errs["dh0"] = nrmse(ref["dh0"], out["dh0"])
    _report(errs, TOL)


@pytest.mark.parametrize("op", OPS)
def test_family_backward_bf16_outputs_and_no_states(op):
    """dq/dk written directly in BF16; no initial state, no final-state gradient."""
    xs = _inputs(op, T=128, H=1, seed=11, state=False)
    saved = forward_saved(op, xs)
    ref = oracle_backward(op, xs, saved)
    out = _family_call(op, xs, saved, op in ("kda", "gdn2"), out_dtype=torch.bfloat16)
    assert out["dh0"] is None and out["dq"].dtype == torch.bfloat16
    # two values that agree to 1e-3 can still round to neighbouring BF16 numbers (1 ulp = 4e-3..8e-3 relative),
    # so the comparison in the BF16 output domain carries that floor on top of the 2e-3 of the FP32 outputs
    _report(_grad_errs(op, ref, out), 3e-3)


def _tile_spans(saved):
    """The widest channel's span of the cumulative gate per (chunk, head), log2 units."""
    G = saved["g_cumsum"].float()
    G = G.reshape(G.shape[0], -1, 64, *G.shape[2:])
    return (G.amax(2) - G.amin(2)).amax(-1)


@pytest.mark.parametrize("case", ["zero_beta", "tiny_beta", "beta_over_one", "strong_gate", "far_gate", "weak_gate", "zero_gate",
                                  "mixed_tiles", "nonmonotonic_gate", "positive_gate", "dht_only", "h0_only"])
def test_kda_edge_cases(case):
    """The reference's named KDA acceptance grid (research/operators/gpu_matrix_20261024/run.py:52-78)."""
    state, grad_state = True, True
    if case == "dht_only":
        state = False
    if case == "h0_only":
        grad_state = False
    xs = _inputs("kda", T=192, H=2, seed=123, state=state, grad_state=grad_state)
    if case == "zero_beta":
        xs["beta"][:, ::3] = 0
    elif case == "tiny_beta":
        xs["beta"] = (xs["beta"].float() * 1e-8).to(torch.bfloat16)
    elif case == "beta_over_one":
        xs["beta"] = (xs["beta"].float() * 2).to(torch.bfloat16)
    elif case == "strong_gate":
        xs["g"] = xs["g"] * 40          # ~ -3 nat per step: every chunk spans 200 log2 units and more (pairwise)
    elif case == "far_gate":
        xs["g"] = xs["g"] * 20          # ~ -1.5 nat per step: every chunk between 80 and 200 (centred, scaled gradients)
    elif case == "weak_gate":
        xs["g"] = xs["g"] / 100
    elif case == "zero_gate":
        xs["g"] = torch.zeros_like(xs["g"])
    elif case == "mixed_tiles":
        xs["g"][:, 64:128, 0, :32] *= 30  # one chunk/head takes the pairwise path next to centred ones
    elif case == "nonmonotonic_gate":
        xs["g"] = xs["g"] * torch.where(torch.rand_like(xs["g"]) < 0.3, -1.0, 1.0)
    elif case == "positive_gate":
        xs["g"] = -xs["g"] * 0.2
    saved = forward_saved("kda", xs)
    spans = _tile_spans(saved)
    wide = dict(strong_gate=spans.numel(), far_gate=0, mixed_tiles=1).get(case)
    assert wide is None or int((spans >= 200).sum()) == wide, spans
    assert case != "far_gate" or bool((spans > 80).all()), spans
    ref = oracle_backward("kda", xs, saved)
    out = _family_call("kda", xs, saved, True)
    errs = _grad_errs("kda", ref, out)
    if state:
        errs["dh0"] = nrmse(ref["dh0"], out["dh0"])
    for n, t in out.items():
        if torch.is_tensor(t):
            assert torch.isfinite(t.float()).all(), f"{n} not finite"
    _report(errs, TOL)   # the pairwise path of strong_gate / mixed_tiles included (measured: dk 1.2e-3, dg 1.2e-3)


@pytest.mark.parametrize("op", ("gdn2", "gdn"))
def test_strong_gate_pairwise_path(op):
    xs = _inputs(op, T=128, H=2, seed=5)
    xs["g"] = xs["g"] * (50 if op == "gdn2" else 3)
    saved = forward_saved(op, xs)
    if op == "gdn2":
        assert bool((_tile_spans(saved) >= 200).all()), _tile_spans(saved)
    ref = oracle_backward(op, xs, saved)
    out = _family_call(op, xs, saved, op == "gdn2")
    errs = _grad_errs(op, ref, out)
    _report(errs, TOL)


@pytest.mark.parametrize("rising", (False, True))
def test_scalar_gate_strong_decay_keeps_the_tensor_core_path(rising):
    """Gated DeltaNet with a decay of far more than 80 log2 units per chunk: the pairwise factor is applied to the
    64x64 matrices, so a monotone gate needs no pairwise kernel; one rising step in such a chunk sends it there."""
    from rewy_b200 import backward as bw
    lib = _capi.load()
    xs = _inputs("gdn", T=128, H=2, seed=5)
    xs["g"] = xs["g"] * 3
    if rising:
        xs["g"][:, 70, 0] = 4.0
    saved = forward_saved("gdn", xs)
    span = (saved["g_cumsum"][:, 64:128].amax(1) - saved["g_cumsum"][:, 64:128].amin(1)).min().item()
    assert span > 80, span
    ref = oracle_backward("gdn", xs, saved)
    ws = torch.empty(_capi.workspace_bytes(_capi.GDN, _capi.RECOMPUTE, 1, 128, 2), dtype=torch.uint8, device=DEV)
    r = bw.gdn_backward(q=xs["q"], k=xs["k"], v=xs["v"], g=saved["g_cumsum"], beta=xs["beta"], A=saved["Akk"],
                        scale=128 ** -0.5, initial_state=xs["initial_state"], do=xs["do"], dht=xs["dht"],
                        out_dtype=torch.float32, workspace=ws, check_status=True)
    out = dict(dq=r[0], dk=r[1], dv=r[2], dbeta=r[3], dg=r[4], dh0=r[5])
    count = lib.rewy_wide_chunk_count(_capi.ptr(ws), _capi.current_stream(torch.device(DEV)))
    assert count == (1 if rising else 0), count
    _report(_grad_errs("gdn", ref, out), TOL)


@pytest.mark.parametrize("op", OPS)
def test_tensor_core_and_warp_mma_kernels_agree(op):
    """The production (tcgen05) scan and chunk kernels against the warp-MMA kernels on the same inputs."""
    xs = _inputs(op, B=2, T=192, H=3, seed=21)
    saved = forward_saved(op, xs)
    lib = _capi.load()
    try:
        assert lib.rewy_set_chunk_variant(1) == 0 and lib.rewy_set_scan_variant(1) == 0
        warp = _family_call(op, xs, saved, op in ("kda", "gdn2"))
    finally:
        lib.rewy_set_chunk_variant(0)
        lib.rewy_set_scan_variant(0)
    tc = _family_call(op, xs, saved, op in ("kda", "gdn2"))
    errs = {n: nrmse(warp[n], tc[n]) for n in warp if warp[n] is not None and n != "wide_chunks"}
    _report(errs, 1e-3)


def test_wide_span_chunks_are_counted():
    """Chunks whose gate span is too wide for centred factors are listed in the control block and handled by the
    exact pairwise path (the reference counts such tiles too: kernels/endpoint_intra.py:301-304)."""
    lib = _capi.load()
    for scale_block, expect in ((30.0, 1), (1.0, 0)):
        xs = _inputs("kda", T=192, H=2, seed=123)
        xs["g"][:, 64:128, 0, :32] *= scale_block
        saved = forward_saved("kda", xs)
        ws = torch.empty(_capi.workspace_bytes(_capi.KDA, _capi.SAVED, 1, 192, 2), dtype=torch.uint8, device=DEV)
        from rewy_b200 import backward as bw
        bw.kda_backward(q=xs["q"], k=xs["k"], v=xs["v"], beta=xs["beta"], Aqk=saved["Aqk"], Akk=saved["Akk"],
                        scale=128 ** -0.5, initial_state=xs["initial_state"], do=xs["do"], dht=xs["dht"],
                        g=saved["g_cumsum"], disable_recompute=True, w=saved["w"], u=saved["u"], qg=saved["qg"],
                        kg=saved["kg"], v_new=saved["v_new"], h=saved["h"], workspace=ws, check_status=True)
        assert lib.rewy_wide_chunk_count(_capi.ptr(ws), _capi.current_stream(torch.device(DEV))) == expect


def test_single_pass_intra_is_selectable_and_close():
    xs = _inputs("kda", T=128, H=2, seed=3)
    saved = forward_saved("kda", xs)
    ref = oracle_backward("kda", xs, saved)
    lib = _capi.load()
    try:
        lib.rewy_set_chunk_variant(1)      # the pass count is an option of the warp-MMA kernel
        out1 = _family_call("kda", xs, saved, True, passes=1)
        out3 = _family_call("kda", xs, saved, True, passes=3)
    finally:
        lib.rewy_set_chunk_variant(0)
    e1, e3 = _grad_errs("kda", ref, out1), _grad_errs("kda", ref, out3)
    _report(e3, TOL)
    _report(e1, 6e-3)


@pytest.mark.parametrize("family", ("kda", "gdn2"))
@pytest.mark.parametrize("scale", (1.0, 3.0))
def test_matrix_intra_on_reference_captured_inputs(golden_dir, family, scale):
    """The reference's captured matrix-intra inputs (validation/npu950_intra) pushed through the chunk
    kernel: Akk = I, dR = -dAkk (as P), v_new = unit rows and dO = dAqk/scale make the kernel's internal
    dAqk/dAkk equal the captured ones (up to BF16 rounding of those operands); h = dh = 0 removes every
    other term.  Limits are the reference's 0.008 / 0.02 (scripts/npu950_intra_regression.py:59-72)."""
    with np.load(golden_dir / f"intra_{family}_inputs.npz") as z:
        x = {n: torch.from_numpy(z[n].copy()) for n in z.files}
    with np.load(golden_dir / f"intra_{family}_expected.npz") as z:
        exp = {n: torch.from_numpy(z[f"scale{scale:g}_{n}"]) for n in ("dq", "dk", "db", "dg")}
    B, C, H, K = x["q"].shape
    sc = 128 ** -0.5
    L = torch.tril(x["dAqk"].permute(0, 2, 1, 3)).permute(0, 2, 1, 3)          # [B,C,H,C] rows i, cols j
    D = torch.tril(x["dAkk"].permute(0, 2, 1, 3), -1).permute(0, 2, 1, 3)
    z128 = lambda: torch.zeros(B, C, H, 128)
    dO, P, R = z128(), z128(), z128()
    dO[..., :C] = L / sc
    P[..., :C] = -D
    R[..., :C] = torch.eye(C)[None, :, None, :]
    eye = torch.eye(C)[None, :, None, :].expand(B, C, H, C)
    bf = lambda t: t.to(torch.bfloat16).to(DEV).contiguous()
    xs = dict(q=bf(x["q"]), k=bf(x["k"]), v=bf(z128()), do=bf(dO))
    if family == "kda":
        xs["beta"] = x["beta"].to(DEV)
    else:
        xs["b"], xs["w"] = bf(x["b"]), bf(z128())
    saved = dict(g_cumsum=(x["g"] * scale).to(DEV).contiguous(), Akk=bf(eye), v_new=bf(R),
                 h=torch.zeros(B, 1, H, 128, 128, dtype=torch.bfloat16, device=DEV))
    out = _run_chunk_adjoint(family, xs, saved, torch.zeros_like(saved["h"]), bf(P))
    # expected intra contribution = reference oracle output minus the partials it started from, with the
    # L/D operands as the kernel sees them (BF16-rounded) accounted for by the tolerance
    want = {n: exp[n].double() - x[n].double() for n in exp}
    want["dg"] = want["dg"].flip(1).cumsum(1).flip(1)   # the kernel also applies the reverse chunk cumsum
    got = dict(dq=out["dq"], dk=out["dk"], dg=out["dg"], db=out["dbeta"] if family == "kda" else out["db_gate"])
    errs = {n: nrmse(want[n], got[n]) for n in want}
    _report(errs, dict(dq=0.008, dk=0.008, db=0.02, dg=0.02))


@pytest.mark.parametrize("op", OPS)
def test_public_autograd_path_against_recurrence(op):
    """Public API end to end, like the reference's ``verify`` (validation.py:47-76): forward under
    use_backend('optimized'), backward after leaving the context, FP64 token recurrence as the oracle."""
    import rewy_b200 as fdr
    from oracle import recurrence_grads
    xs = _inputs(op, T=128, H=2, seed=42, gate_scale=0.05, gate="softplus")
    ins = {n: (x.detach().clone().requires_grad_() if x is not None else None) for n, x in operator_inputs(op, xs).items()}
    fdr.stats(reset=True)
    policies = (False, True) if op in ("kda", "gdn2") else (False,)
    ref, o_ref, fin_ref = recurrence_grads(op, {n: (x.detach().cpu() if x is not None else None) for n, x in ins.items()},
                                           xs["do"].cpu(), xs["dht"].cpu())
    for saved_policy in policies:
        kw = dict(ins, output_final_state=True)
        if op in ("kda", "gdn2"):
            kw["disable_recompute"] = saved_policy
        with fdr.use_backend("optimized", ops=(op,)):
            o, fin = getattr(fdr, {"kda": "chunk_kda", "gdn2": "chunk_gdn2", "gdn": "chunk_gated_delta_rule",
                                   "delta": "chunk_delta_rule"}[op])(**kw)
        leaves = [x for x in ins.values() if x is not None]
        grads = torch.autograd.grad((o, fin), leaves, (xs["do"], xs["dht"]))
        names = [n for n, x in ins.items() if x is not None]
        errs = {n: nrmse(ref[n], g) for n, g in zip(names, grads)}
        errs["o"] = nrmse(o_ref, o)
        errs["final_state"] = nrmse(fin_ref, fin)
        tol = {n: (0.02 if n in ("g", "beta", "b", "w") else 0.008) for n in errs}
        _report(errs, tol)
    fdr.assert_used((op,))
    assert fdr.stats()[f"{op}.optimized_backward"] == len(policies)


def test_rejections_and_error_codes():
    import rewy_b200 as fdr
    xs = _inputs("kda", T=128, H=1)
    with fdr.use_backend("optimized"):
        with pytest.raises(RuntimeError, match="custom scale"):
            fdr.chunk_kda(xs["q"], xs["k"], xs["v"], xs["g"], xs["beta"], scale=0.5)
    saved = forward_saved("kda", xs)
    a, keep = base_args("kda", xs, saved)
    lib = _capi.load()
    assert lib.rewy_kda_bwd(a, None) == 1 and b"NULL" in lib.rewy_last_error()     # outputs missing
    a.T = 100
    assert lib.rewy_kda_bwd(a, None) == 2                                           # bad shape


def test_full_size_headline_properties():
    """BASELINE headline shape (KDA B=8,T=8192,H=32) through size-independent properties:
    linearity of the backward in (dO, dht) and equality of one (batch, head) slice with the FP64 oracle run
    on that slice alone (the path is independent across batch and head)."""
    from rewy_b200.forward import chunk_forward
    B, T, H = 8, 8192, 32
    dev = torch.device(DEV)
    g = torch.Generator(device=dev); g.manual_seed(1)
    rn = lambda *s: torch.randn(*s, generator=g, device=dev)
    q = torch.nn.functional.normalize(rn(B, T, H, 128), dim=-1).to(torch.bfloat16)
    k = torch.nn.functional.normalize(rn(B, T, H, 128), dim=-1).to(torch.bfloat16)
    v = rn(B, T, H, 128).to(torch.bfloat16)
    gate = -torch.nn.functional.softplus(rn(B, T, H, 128)) * 0.1
    beta = torch.sigmoid(rn(B, T, H)).to(torch.bfloat16)
    do = rn(B, T, H, 128).to(torch.bfloat16)
    xs = dict(q=q, k=k, v=v, g=gate, beta=beta, do=do, initial_state=None, dht=None)
    saved = chunk_forward("kda", q, k, v, g=gate, beta=beta)
    out = _family_call("kda", xs, saved, True)
    xs2 = dict(xs, do=(do.float() * 2).to(torch.bfloat16))
    out2 = _family_call("kda", xs2, saved, True)
    for n in ("dq", "dk", "dv", "dg", "dbeta"):
        assert nrmse(out[n].float() * 2, out2[n]) < 5e-3, n
    b0, h0 = 5, 17
    sl = lambda t: None if t is None else t[b0:b0 + 1, :, h0:h0 + 1].contiguous()
    xs_s = {n: sl(t) for n, t in xs.items()}
    saved_s = {n: (sl(t) if n != "h" else t[b0:b0 + 1, :, h0:h0 + 1].contiguous()) for n, t in saved.items()
               if t is not None and n not in ("o", "final_state")}
    ref = oracle_backward("kda", xs_s, saved_s)
    got = {n: sl(t) for n, t in out.items() if torch.is_tensor(t)}
    _report(_grad_errs("kda", ref, got), TOL)


def test_custom_op_passes_opcheck():
    """torch.library.opcheck of the registered operator (schema, fake implementation against the real one) on a small
    KDA problem, through the same arguments the family function builds."""
    from rewy_b200 import backward as bw
    xs = _inputs("kda", T=128, H=2, seed=2)
    saved = forward_saved("kda", xs)
    ws = torch.empty(_capi.workspace_bytes(_capi.KDA, _capi.RECOMPUTE, 1, 128, 2), dtype=torch.uint8, device=DEV)
    args = (_capi.KDA, _capi.RECOMPUTE, True, 0, False, 128 ** -0.5, xs["q"], xs["k"], xs["v"], xs["do"], saved["Akk"], ws,
            saved["g_cumsum"], xs["beta"].float(), None, None, saved["Aqk"], xs["initial_state"], xs["dht"],
            None, None, None, None, None, None)
    torch.library.opcheck(torch.ops.rewy_b200.family_bwd.default, args,
                          test_utils=("test_schema", "test_faketensor"))


@pytest.mark.parametrize("op,policy_saved", [("kda", True), ("kda", False), ("gdn", False)])
def test_family_backward_replays_from_a_cuda_graph(op, policy_saved):
    """The whole backward is capturable (no host synchronisation, no shape-dependent host reads, fixed workspace):
    captured once after a warm-up call, replayed on new contents of the same buffers, it reproduces the eager results
    bit for bit.  The reference times its operators the same way (research/operators/delta_algebra_20261024/common.py:28-61)."""
    from rewy_b200 import backward as bw
    xs = _inputs(op, B=2, T=256, H=2, seed=31)
    saved = forward_saved(op, xs)
    B, T, H, _ = xs["k"].shape
    fam = _capi.FAMILY_ID[op]
    ws = torch.empty(_capi.workspace_bytes(fam, _capi.SAVED if policy_saved else _capi.RECOMPUTE, B, T, H),
                     dtype=torch.uint8, device=DEV)
    do_buf = xs["do"].clone()

    def call():
        common = dict(q=xs["q"], k=xs["k"], v=xs["v"], scale=128 ** -0.5, initial_state=xs["initial_state"], do=do_buf,
                      dht=xs["dht"], out_dtype=torch.bfloat16, workspace=ws)
        if op == "kda":
            return bw.kda_backward(beta=xs["beta"], Aqk=saved["Aqk"], Akk=saved["Akk"], g=saved["g_cumsum"],
                                   disable_recompute=policy_saved, w=saved["w"], u=saved["u"], qg=saved["qg"],
                                   kg=saved["kg"], v_new=saved["v_new"], h=saved["h"], **common)
        return bw.gdn_backward(g=saved["g_cumsum"], beta=xs["beta"], A=saved["Akk"], **common)

    side = torch.cuda.Stream(device=DEV)
    side.wait_stream(torch.cuda.current_stream(DEV))
    with torch.cuda.stream(side):
        call()                                        # warm-up outside the capture (first-use set-up of the kernels)
    torch.cuda.current_stream(DEV).wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = call()
    do_new = (xs["do"].float() * -0.5 + 0.25).to(torch.bfloat16)
    do_buf.copy_(do_new)
    graph.replay()
    torch.cuda.synchronize()
    replayed = [t.clone() for t in outs if t is not None]
    eager = [t for t in call() if t is not None]
    torch.cuda.synchronize()
    assert _capi.load().rewy_device_status(_capi.ptr(ws), _capi.current_stream(torch.device(DEV))) == 0
    for a, b in zip(replayed, eager):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)


@pytest.mark.parametrize("op", OPS)
def test_concurrent_scans_give_the_same_gradients_as_sequential_ones(op):
    """Recompute policy: the forward scan on the library's side stream (default) against every stage on the caller's
    stream; the two scans share no tensor, so the results are bitwise equal."""
    xs = _inputs(op, B=2, T=512, H=4, seed=77)
    saved = forward_saved(op, xs)
    lib = _capi.load()
    try:
        assert lib.rewy_set_scan_overlap(0) == 0
        seq = _family_call(op, xs, saved, False)
    finally:
        lib.rewy_set_scan_overlap(1)
    par = _family_call(op, xs, saved, False)
    par2 = _family_call(op, xs, saved, False)
    torch.cuda.synchronize()
    for n, t in seq.items():
        if torch.is_tensor(t):
            assert torch.equal(t, par[n]) and torch.equal(t, par2[n]), (op, n)


def test_a_workspace_of_the_caller_counts_as_written():
    """The schema says that the family backward writes its workspace: torch's version counter has to see it."""
    from rewy_b200 import backward as bw
    xs = _inputs("delta", T=128, H=2, seed=1, state=False)
    sv = forward_saved("delta", xs)
    ws = torch.empty(_capi.workspace_bytes(_capi.DELTA, _capi.RECOMPUTE, 1, 128, 2), dtype=torch.uint8, device=DEV)
    version = ws._version
    bw.delta_backward(xs["q"], xs["k"], xs["v"], xs["beta"], sv["Akk"], 128 ** -0.5, None, xs["do"], None, workspace=ws)
    assert ws._version > version
