"""The work this package is used for, as measurable cases.

Three entry points carry it:
  backward   ``rewy_b200.backward.{kda,gdn2,gdn,delta}_backward``: the whole-family backward, called with what a forward
             saved.  Lengths are multiples of the 64-token chunk, as at that boundary.
  train      the public operators under autograd, forward and backward of one layer call, with the options layers use:
             q/k normalisation, beta logits, the fused KDA gate, grouped value heads, packed sequences of any length.
  prefill    the public operators without autograd, from an incoming state to an outgoing one: a prompt, or the next
             piece of one, of any length.
Sizes are those of the benchmark configurations, of the published operator grid and of the tests.
"""
import math

import torch

import rewy_b200
from rewy_b200 import backward
from rewy_b200.forward import chunk_forward

D = 128  # key and value channels of a head
OPERATOR = {"kda": "chunk_kda", "gdn2": "chunk_gdn2", "gdn": "chunk_gated_delta_rule", "delta": "chunk_delta_rule"}


def _case(entry, family, B, T, H, *, groups=1, saved=False, state=False, options=False, sequences=0):
    return {"entry": entry, "family": family, "B": B, "T": T, "H": H, "groups": groups, "saved": saved, "state": state,
            "options": options, "sequences": sequences}


def listed():
    named = {
        # one short sequence with few heads: a test, a tiny model or a small shard; launches and host work count
        "backward_kda_smallest": _case("backward", "kda", 1, 512, 4, saved=True),
        # the largest shape of the published operator grid: one long sequence, fewer sequences than SMs
        "backward_kda_one_sequence": _case("backward", "kda", 1, 8192, 16, saved=True),
        # the headline training shape, everything saved by the forward
        "backward_kda_headline": _case("backward", "kda", 8, 8192, 32, saved=True),
        # scalar gate with states in and out: a segment of a longer sequence in training
        "backward_gdn_states": _case("backward", "gdn", 4, 4096, 16, state=True),
        # no gate, no state, many short sequences
        "backward_delta": _case("backward", "delta", 16, 2048, 16),
        # long-context training with vector gates; activations recomputed, states in and out
        "backward_gdn2_long": _case("backward", "gdn2", 2, 32768, 32, state=True),
        # a KDA layer's training step with everything fused into the operator, recompute policy (its default)
        "train_kda_layer": _case("train", "kda", 2, 4096, 16, options=True),
        # a gated DeltaNet layer with two value heads to each key head
        "train_gdn_grouped_heads": _case("train", "gdn", 2, 4096, 16, groups=2, options=True),
        # packed documents of arbitrary lengths, as a training batch without padding
        "train_delta_packed": _case("train", "delta", 1, 16001, 8, sequences=12, options=True),
        # a GDN2 layer on an odd length, activations kept
        "train_gdn2_odd_length": _case("train", "gdn2", 2, 2000, 8, saved=True),
        # a long prompt through a KDA layer with the fused gate
        "prefill_kda_prompt": _case("prefill", "kda", 1, 8192, 32, state=True, options=True),
        # the next short piece of a conversation: the smallest serving call
        "prefill_gdn_piece": _case("prefill", "gdn", 1, 77, 16, state=True, options=True),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _spread(rng, lo, hi):
    """Whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    entry = rng.choice(("backward", "train", "prefill"))
    family = rng.choice(tuple(OPERATOR))
    most = 1 << 20 if entry == "backward" else 1 << 18   # token-heads: below the largest listed case's cost
    H = _spread(rng, 2, 32)
    T = 64 * _spread(rng, 1, 256) if entry == "backward" else _spread(rng, 64 if entry == "train" else 1, 16384)
    B = _spread(rng, 1, 16)
    while B * T * H > most:
        B, T = (max(1, B // 2), T) if B > 1 else (1, T // 128 * 64 if entry == "backward" else T // 2)
    return _case(entry, family, B, T, H,
                 groups=rng.choice((1, 1, 2)) if entry != "backward" else 1,
                 saved=family in ("kda", "gdn2") and rng.random() < 0.5,
                 state=rng.random() < 0.5 if entry != "prefill" else True,
                 options=entry != "backward" and rng.random() < 0.7,
                 sequences=rng.randint(2, 9) if entry == "train" and B == 1 and T >= 512 and rng.random() < 0.5 else 0)


def _offsets(T, sequences, generator):
    """Offsets of `sequences` packed documents of uneven lengths that add up to T."""
    share = torch.rand(sequences, generator=generator, dtype=torch.float64) + 0.1
    cut = (torch.cumsum(share, 0) / share.sum() * T).round().to(torch.int64)
    cut[-1] = T
    return torch.cat([torch.zeros(1, dtype=torch.int64), cut])


def _inputs(case, seed):
    """Named inputs of the operator.  q, k unit length unless the operator normalises them; v ~ N(0, 1); beta in (0, 1)
    or its logits; natural-log decays as in the benchmark configurations, or the raw gate input of a layer whose
    decay rates and time steps are initialised over their usual ranges (rate 1..16, step 0.001..0.1)."""
    family, B, T, H, options = case["family"], case["B"], case["T"], case["H"], case["options"]
    HV = H * case["groups"]
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=gen, device=dev)
    uniform = lambda *s: torch.rand(*s, generator=gen, device=dev)
    softplus = torch.nn.functional.softplus
    fused = family == "kda" and options and case["groups"] == 1
    xs = {}
    for n in ("q", "k"):
        x = rn(B, T, H, D)
        xs[n] = (x if options else torch.nn.functional.normalize(x, dim=-1)).to(torch.bfloat16)
        del x
    xs["v"] = rn(B, T, HV, D).to(torch.bfloat16)
    if family == "gdn":
        xs["g"] = -torch.exp(uniform(HV)) * softplus(rn(B, T, HV))
    elif fused:
        xs["g"] = (0.5 * rn(B, T, HV, D)).to(torch.bfloat16)
        step = torch.exp(uniform(HV * D) * (math.log(0.1) - math.log(0.001)) + math.log(0.001))
        xs["A_log"] = torch.log(1 + 15 * uniform(HV))
        xs["dt_bias"] = step + torch.log(-torch.expm1(-step))     # softplus(dt_bias) = step
    elif family != "delta":
        xs["g"] = -softplus(rn(B, T, HV, D)) * (0.05 if family == "gdn2" else 0.1)
    if family == "gdn2":
        xs["b"] = torch.sigmoid(rn(B, T, HV, D)).to(torch.bfloat16)
        xs["w"] = torch.sigmoid(rn(B, T, HV, D)).to(torch.bfloat16)
    else:
        x = rn(B, T, HV)
        xs["beta"] = (x if options and family in ("kda", "gdn") else torch.sigmoid(x)).to(torch.bfloat16)
    states = case["sequences"] or B
    h0 = 0.1 * rn(states, HV, D, D) if case["state"] else None
    dht = 0.1 * rn(states, HV, D, D) if case["state"] else None
    do = rn(B, T, HV, D).to(torch.bfloat16)
    kw = {}
    if options:
        kw["use_qk_l2norm_in_kernel"] = True
        if family in ("kda", "gdn"):
            kw["use_beta_sigmoid_in_kernel"] = True
        if fused:
            kw["use_gate_in_kernel"] = True
    if family in ("kda", "gdn2"):
        kw["disable_recompute"] = case["saved"]
    if case["sequences"]:
        host = torch.Generator()
        host.manual_seed(seed)
        cu = _offsets(T, case["sequences"], host)
        kw["cu_seqlens"], kw["cu_seqlens_cpu"] = cu.to(dev, torch.int32), cu
    return xs, h0, do, dht, kw


def prepare(case, seed):
    rewy_b200.enable("optimized")
    xs, h0, do, dht, kw = _inputs(case, seed)
    entry, family = case["entry"], case["family"]
    if entry == "backward":
        f = chunk_forward(family, xs["q"], xs["k"], xs["v"], g=xs.get("g"), beta=xs.get("beta"), b=xs.get("b"), w=xs.get("w"),
                          initial_state=h0, output_final_state=False)
        args = dict(q=xs["q"], k=xs["k"], v=xs["v"], scale=D ** -0.5, initial_state=h0, do=do, dht=dht,
                    out_dtype=torch.bfloat16)
        if family != "delta":
            args["g"] = f["g_cumsum"]
        if family == "gdn2":
            args.update(b=xs["b"], w_gate=xs["w"])
        else:
            args["beta"] = xs["beta"].float()
        if family in ("kda", "gdn2"):
            args.update(Aqk=f["Aqk"], Akk=f["Akk"], disable_recompute=case["saved"])
            if case["saved"]:
                wy = ("w_wy", "u_wy") if family == "gdn2" else ("w", "u")
                args.update({wy[0]: f["w"], wy[1]: f["u"], "qg": f["qg"], "kg": f["kg"], "v_new": f["v_new"], "h": f["h"]})
        else:
            args["A"] = f["Akk"]
        return {"entry": entry, "call": getattr(backward, family + "_backward"), "args": args}
    call = getattr(rewy_b200, OPERATOR[family])
    if h0 is not None:
        kw.update(initial_state=h0, output_final_state=True)
    if entry == "train":
        leaves = {n: x.requires_grad_() for n, x in xs.items()}
        wrt = tuple(leaves.values()) + ((h0.requires_grad_(),) if h0 is not None else ())
        return {"entry": entry, "call": call, "args": {**leaves, **kw}, "wrt": wrt, "do": do, "dht": dht}
    return {"entry": entry, "call": call, "args": {**xs, **kw}}


def run(state):
    if state["entry"] == "backward":
        return state["call"](**state["args"])
    if state["entry"] == "prefill":
        with torch.no_grad():
            return state["call"](**state["args"])
    o, final = state["call"](**state["args"])
    if state["dht"] is None:
        return o, torch.autograd.grad(o, state["wrt"], state["do"])
    return o, final, torch.autograd.grad((o, final), state["wrt"], (state["do"], state["dht"]))


def work(case):
    """Boundary bytes (every input of the pass read once, every output written once, in their own types) and the dense
    products of the chunked algorithm (2 m n k each, chunk of 64 tokens; a causal 64x64 matrix counted whole)."""
    entry, family, H = case["entry"], case["family"], case["H"]
    HV = H * case["groups"]
    tokens = case["B"] * case["T"]
    n, nk = tokens * HV, tokens * H
    vector, fused = family in ("kda", "gdn2"), family == "kda" and case["options"] and case["groups"] == 1
    states = (case["sequences"] or case["B"]) * HV * D * D * 4 if case["state"] else 0
    gate = {"kda": 256 if fused else 512, "gdn2": 512, "gdn": 4, "delta": 0}[family]
    gates = 512 if family == "gdn2" else (4 if entry == "backward" else 2)       # b and w, or beta
    inputs = nk * 512 + n * (256 + gate + gates) + states                        # q, k; v, gates; h0
    C = 64
    forward_flops = n * 2 * (2 * C * D + C * C // 3 + 2 * C * D + 3 * D * D + C * D)
    recompute = n * 2 * (2 * C * D + 2 * D * D + (C * D if not vector else 0)) if not case["saved"] else 0
    backward_flops = n * 2 * (C * D + C * D + 2 * D * D + C * D + 2 * C * D + 3 * D * D + 4 * C * D) + recompute
    if entry == "prefill":
        return {"bytes": inputs + n * 256 + states, "flops": forward_flops}
    if entry == "train":   # inputs read and o written; do and dht read, a gradient written for every input
        return {"bytes": inputs + n * 256 + states + n * 256 + states + inputs, "flops": forward_flops + backward_flops}
    moved = inputs + n * 256 + states                                           # do, dht
    moved += n * (256 if vector else 128)                                       # Akk and, with vector gates, Aqk
    if case["saved"]:
        moved += n * (4 * 256 + 512)                                            # w, qg, kg, v_new; h
    return {"bytes": moved + inputs, "flops": backward_flops}


def tolerance(case):
    """Operands of every product are BF16, sums FP32.  Against the FP64 recurrence and the FP64 closed form the gradients
    are off by up to 2e-3 (the stored BF16 tensors) and up to 3.7e-3 through the whole autograd path; two implementations
    that sum in another order differ by 1e-4, and by up to 2e-3 where a BF16 state entry rounds the other way and stays."""
    return {"rel": 8e-3, "max": 0.4}
