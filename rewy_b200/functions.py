"""Autograd functions and public operators of the four families.

Same contracts as the reference's private autograd copies (src/fast_delta_rule/_compat/kda.py:23-210,
gdn.py:128-267, gdn2.py:43-201, delta.py:19-141): the forward saves FLA's tensor set (policy
``disable_recompute`` decides whether w,u,qg,kg,v_new,h are kept), the backward hands them to the
whole-family backward of ``rewy_b200.backward`` and casts to the input dtypes.  The wrapper-level options the
reference accepts for KDA on CUDA (fused gate activation, beta sigmoid, q/k L2 normalisation, value-first state
layout: docs/compatibility.md:12-13, tests/test_accelerator.py:65-83) run as CUDA passes of ``rewy_b200.elementwise``.  The backward stays bound
to this implementation after a ``use_backend`` context exits, like the reference's.
"""
import torch

from . import backward as _bwd
from .forward import chunk_forward


from . import elementwise as _ew


def _cumulative_gate(g, A_log=None, dt_bias=None):
    """Chunk-local cumulative gate in log2 units on the device (vector gates), optionally with the KDA gate activation."""
    return _ew.gate_cumsum_fwd(g, A_log, dt_bias)


def _first_order(grads):
    """Gradients that come out of the row kernels, which torch does not see: differentiating them again raises, as it does for
    the family backward (a torch operator without a derivative).  Called inside an autograd function's backward."""
    if not torch.is_grad_enabled():   # only a backward with create_graph runs with gradients enabled
        return tuple(grads)
    return tuple(torch.ops.rewy_b200.first_order.default(list(grads)))


def _front(q, k, rows, groups, normalize):
    """q and k as the kernels take them: L2-normalised (optional), padded, each head repeated to its value heads, in one
    pass.  Returns (q, k, q_rstd, k_rstd)."""
    plain = groups == 1 and not rows.needed
    if not normalize and (plain or q.dtype != torch.bfloat16):
        return q, k, None, None   # (other types are refused by the forward)
    if plain:   # every row where it is: the plain normalisation kernels are faster (B=2 T=4096 H=16: 31 + 47 against 35 + 58 us)
        (q, q_rstd), (k, k_rstd) = _ew.l2norm_fwd(q), _ew.l2norm_fwd(k)
        return q, k, q_rstd, k_rstd
    return _ew.qk_front_fwd(q, k, rows.row_map(q.shape[0]), groups, normalize)


def _front_backward(ctx, q, k, q_rstd, k_rstd, dq, dk):
    if q_rstd is None and ctx.groups == 1:
        return ctx.rows.cut_rows(dq, dk)
    if ctx.groups == 1 and not ctx.rows.needed:
        return _ew.l2norm_bwd(q, q_rstd, dq), _ew.l2norm_bwd(k, k_rstd, dk)
    grads = _ew.qk_front_bwd(q, k, q_rstd, k_rstd, dq, dk, ctx.rows.row_map(q.shape[0]), ctx.groups)
    return grads if q_rstd is not None else _first_order(grads)   # (the normalisation ends the graph, as its plain kernels do)


class ChunkKDAFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, g, beta, A_log, dt_bias, scale, initial_state, output_final_state, use_qk_l2norm_in_kernel,
                use_gate_in_kernel, use_beta_sigmoid_in_kernel, allow_neg_eigval, disable_recompute, state_v_first,
                cu_seqlens, rows, groups):
        q, k, q_rstd, k_rstd = _front(q, k, rows, groups, use_qk_l2norm_in_kernel)
        # a raw gate input goes through -exp(A_log) softplus(g + dt_bias): a very negative value gives decay 0
        v, beta, g = rows.pad_rows(v, beta, (g, -1e4 if use_gate_in_kernel else 0.0))
        beta_raw = beta
        if use_beta_sigmoid_in_kernel:
            beta = _ew.beta_sigmoid_fwd(beta_raw, 2.0 if allow_neg_eigval else 1.0)
        # with use_gate_in_kernel, g is the raw gate input: -exp(A_log) * softplus(g + dt_bias) and the chunk cumsum are
        # one pass; otherwise g is the per-step natural-log decay
        g_cumsum = _cumulative_gate(g, A_log if use_gate_in_kernel else None, dt_bias if use_gate_in_kernel else None)
        f = chunk_forward("kda", q, k, v, g=g_cumsum, beta=beta, scale=scale, initial_state=initial_state,
                          output_final_state=output_final_state, g_is_cumsum=True, state_v_first=state_v_first,
                          cu_seqlens=cu_seqlens)
        keep = (lambda x: x) if disable_recompute else (lambda x: None)
        ctx.save_for_backward(q, q_rstd, k, k_rstd, v, g_cumsum, g, beta_raw, beta, A_log, dt_bias, f["Aqk"], f["Akk"],
                              keep(f["w"]), keep(f["u"]), keep(f["qg"]), keep(f["kg"]), keep(f["v_new"]),
                              keep(f["h"]), initial_state, cu_seqlens)
        ctx.scale, ctx.disable_recompute = scale, disable_recompute
        ctx.use_qk_l2norm_in_kernel, ctx.use_beta_sigmoid_in_kernel = use_qk_l2norm_in_kernel, use_beta_sigmoid_in_kernel
        ctx.use_gate_in_kernel, ctx.allow_neg_eigval, ctx.state_v_first = use_gate_in_kernel, allow_neg_eigval, state_v_first
        ctx.rows, ctx.groups = rows, groups
        return rows.cut_output(f["o"].type_as(q)), f["final_state"]

    @staticmethod
    def backward(ctx, do, dht):
        (q, q_rstd, k, k_rstd, v, g_cumsum, g_input, beta_raw, beta, A_log, dt_bias, Aqk, Akk, w, u, qg, kg, v_new, h,
         initial_state, cu_seqlens) = ctx.saved_tensors
        dq, dk, dv, db, dg, dh0, _, _ = _bwd.kda_backward(
            q=q, k=k, v=v, beta=beta, Aqk=Aqk, Akk=Akk, scale=ctx.scale, initial_state=initial_state,
            do=ctx.rows.pad_output_grad(do), dht=dht, g=g_cumsum, state_v_first=ctx.state_v_first, cu_seqlens=cu_seqlens, disable_recompute=ctx.disable_recompute, w=w, u=u, qg=qg, kg=kg,
            v_new=v_new, h=h, out_dtype=torch.float32 if ctx.use_qk_l2norm_in_kernel else torch.bfloat16)
        dA = dbias = None
        if ctx.use_gate_in_kernel:
            dg, dA, dbias = _ew.gate_act_bwd(g_input, A_log, dt_bias, dg,
                                              torch.bfloat16 if g_input.dtype == torch.bfloat16 else torch.float32)
            dA = dA.view_as(A_log).to(A_log.dtype)
            dbias = None if dbias is None else dbias.view_as(dt_bias).to(dt_bias.dtype)
        dq, dk = _front_backward(ctx, q, k, q_rstd, k_rstd, dq, dk)
        if ctx.use_beta_sigmoid_in_kernel:
            db = _ew.beta_sigmoid_bwd(beta_raw, db, 2.0 if ctx.allow_neg_eigval else 1.0)
        dv, dg, db = ctx.rows.cut_rows(dv, dg, db)
        return (dq.to(q), dk.to(k), dv.to(v), dg.to(g_input), db.to(beta_raw), dA, dbias, None, dh0) + (None,) * 10


class ChunkGDN2Function(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, g, b, w, scale, initial_state, output_final_state, use_qk_l2norm_in_kernel,
                disable_recompute, state_v_first, cu_seqlens, rows, groups):
        q, k, q_rstd, k_rstd = _front(q, k, rows, groups, use_qk_l2norm_in_kernel)
        v, g, b, w = rows.pad_rows(v, g, b, w)
        g_cumsum = _cumulative_gate(g)
        f = chunk_forward("gdn2", q, k, v, g=g_cumsum, b=b, w=w, scale=scale, initial_state=initial_state,
                          output_final_state=output_final_state, g_is_cumsum=True, state_v_first=state_v_first,
                          cu_seqlens=cu_seqlens)
        keep = (lambda x: x) if disable_recompute else (lambda x: None)
        ctx.save_for_backward(q, q_rstd, k, k_rstd, v, g_cumsum, g, b, w, f["Aqk"], f["Akk"], keep(f["w"]),
                              keep(f["u"]), keep(f["qg"]), keep(f["kg"]), keep(f["v_new"]), keep(f["h"]), initial_state,
                              cu_seqlens)
        ctx.scale, ctx.disable_recompute, ctx.use_qk_l2norm_in_kernel = scale, disable_recompute, use_qk_l2norm_in_kernel
        ctx.state_v_first = state_v_first
        ctx.rows, ctx.groups = rows, groups
        return rows.cut_output(f["o"].type_as(q)), f["final_state"]

    @staticmethod
    def backward(ctx, do, dht):
        (q, q_rstd, k, k_rstd, v, g_cumsum, g_input, b, w, Aqk, Akk, w_wy, u_wy, qg, kg, v_new, h,
         initial_state, cu_seqlens) = ctx.saved_tensors
        dq, dk, dv, db, dw, dg, dh0, _, _ = _bwd.gdn2_backward(
            q=q, k=k, v=v, b=b, w_gate=w, Aqk=Aqk, Akk=Akk, scale=ctx.scale, initial_state=initial_state,
            do=ctx.rows.pad_output_grad(do),
            dht=dht, g=g_cumsum, state_v_first=ctx.state_v_first, cu_seqlens=cu_seqlens, w_wy=w_wy, u_wy=u_wy, qg=qg, kg=kg, v_new=v_new, h=h,
            disable_recompute=ctx.disable_recompute,
            out_dtype=torch.float32 if ctx.use_qk_l2norm_in_kernel else torch.bfloat16)
        dq, dk = _front_backward(ctx, q, k, q_rstd, k_rstd, dq, dk)
        dv, dg, db, dw = ctx.rows.cut_rows(dv, dg, db, dw)
        return (dq.to(q.dtype), dk.to(k.dtype), dv.to(v.dtype), dg.to(g_input.dtype), db.to(b.dtype), dw.to(w.dtype),
                None, dh0) + (None,) * 7


class ChunkGatedDeltaRuleFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, g, beta, scale, initial_state, output_final_state, use_qk_l2norm_in_kernel,
                use_beta_sigmoid_in_kernel, allow_neg_eigval, state_v_first, cu_seqlens, rows, groups):
        q, k, q_rstd, k_rstd = _front(q, k, rows, groups, use_qk_l2norm_in_kernel)
        v, g, beta = rows.pad_rows(v, g, beta)
        beta_raw = beta
        if use_beta_sigmoid_in_kernel:
            beta = _ew.beta_sigmoid_fwd(beta_raw, 2.0 if allow_neg_eigval else 1.0)
        f = chunk_forward("gdn", q, k, v, g=g, beta=beta, scale=scale, initial_state=initial_state,
                          output_final_state=output_final_state, state_v_first=state_v_first, cu_seqlens=cu_seqlens)
        ctx.save_for_backward(q, q_rstd, k, k_rstd, v, f["g_cumsum"], g, beta_raw, beta, f["Akk"], initial_state, cu_seqlens)
        ctx.scale, ctx.use_qk_l2norm_in_kernel = scale, use_qk_l2norm_in_kernel
        ctx.use_beta_sigmoid_in_kernel, ctx.allow_neg_eigval = use_beta_sigmoid_in_kernel, allow_neg_eigval
        ctx.state_v_first = state_v_first
        ctx.rows, ctx.groups = rows, groups
        return rows.cut_output(f["o"].to(q.dtype)), f["final_state"]

    @staticmethod
    def backward(ctx, do, dht):
        q, q_rstd, k, k_rstd, v, g, g_input, beta_raw, beta, A, initial_state, cu_seqlens = ctx.saved_tensors
        dq, dk, dv, db, dg, dh0, _, _ = _bwd.gdn_backward(
            q=q, k=k, v=v, g=g, beta=beta, A=A, scale=ctx.scale, initial_state=initial_state,
            do=ctx.rows.pad_output_grad(do), dht=dht,
            state_v_first=ctx.state_v_first, cu_seqlens=cu_seqlens,
            out_dtype=torch.float32 if ctx.use_qk_l2norm_in_kernel else torch.bfloat16)
        dq, dk = _front_backward(ctx, q, k, q_rstd, k_rstd, dq, dk)
        if ctx.use_beta_sigmoid_in_kernel:
            db = _ew.beta_sigmoid_bwd(beta_raw, db, 2.0 if ctx.allow_neg_eigval else 1.0)
        dv, dg, db = ctx.rows.cut_rows(dv, dg, db)
        return (dq.to(q), dk.to(k), dv.to(v), dg.to(g_input), db.to(beta_raw), None, dh0) + (None,) * 8


class ChunkDeltaRuleFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, beta, scale, initial_state, output_final_state, use_qk_l2norm_in_kernel, cu_seqlens, rows,
                groups):
        q, k, q_rstd, k_rstd = _front(q, k, rows, groups, use_qk_l2norm_in_kernel)
        v, beta = rows.pad_rows(v, beta)
        f = chunk_forward("delta", q, k, v, beta=beta, scale=scale, initial_state=initial_state,
                          output_final_state=output_final_state, cu_seqlens=cu_seqlens)
        ctx.save_for_backward(q, q_rstd, k, k_rstd, v, beta, f["Akk"], initial_state, cu_seqlens)
        ctx.scale, ctx.use_qk_l2norm_in_kernel = scale, use_qk_l2norm_in_kernel
        ctx.rows, ctx.groups = rows, groups
        return rows.cut_output(f["o"].to(q.dtype)), f["final_state"]

    @staticmethod
    def backward(ctx, do, dht):
        q, q_rstd, k, k_rstd, v, beta, A, initial_state, cu_seqlens = ctx.saved_tensors
        dq, dk, dv, db, dh0 = _bwd.delta_backward(
            q=q, k=k, v=v, beta=beta, A=A, scale=ctx.scale, initial_state=initial_state,
            do=ctx.rows.pad_output_grad(do), dht=dht,
            cu_seqlens=cu_seqlens,
            out_dtype=torch.float32 if ctx.use_qk_l2norm_in_kernel else torch.bfloat16)
        dq, dk = _front_backward(ctx, q, k, q_rstd, k_rstd, dq, dk)
        dv, db = ctx.rows.cut_rows(dv, db)
        return (dq.to(q.dtype), dk.to(k.dtype), dv.to(v.dtype), db.to(beta.dtype), None, dh0) + (None,) * 5


def _packed(cu_seqlens, q):
    """cu_seqlens as an int32 device tensor (the dispatch layer has already checked that every length is a multiple
    of 64), or None."""
    return None if cu_seqlens is None else cu_seqlens.to(device=q.device, dtype=torch.int32).contiguous()


class _Ragged:
    """Lengths that are not multiples of the chunk: every sequence is extended to the next multiple of 64 by neutral
    tokens (q = k = v = 0, no decay), which change neither the state nor any real token's output, and the results are
    cut back.  The autograd functions do both with the library's row kernels (``pad_rows``, ``cut_rows``, and the q/k
    front pass); ``pad`` and ``cut`` state the same as differentiable tensor operations for any device.  FLA handles
    such lengths by bounds checks inside its kernels (the reference's release envelope rejects them:
    src/fast_delta_rule/runtime.py:87-88)."""

    def __init__(self, T, device, cu_seqlens=None, cu_seqlens_cpu=None):
        self.T, self.cu, self._lengths = T, None, None
        if cu_seqlens is None:
            self.total = -(-T // 64) * 64
            self.needed = self.total != T
            return
        host = (cu_seqlens if cu_seqlens_cpu is None else cu_seqlens_cpu).detach().cpu().to(torch.int64)
        lengths = host[1:] - host[:-1]
        padded = (lengths + 63) // 64 * 64
        self.needed = bool((padded != lengths).any())
        if not self.needed:
            self.total = T
            return
        if bool((lengths < 0).any()) or int(lengths.sum()) != T:   # the row kernels go by these offsets
            raise ValueError(f"cu_seqlens must rise and cover the {T} tokens, got {host.tolist()}")
        self.total, self._lengths = int(padded.sum()), lengths
        both = torch.zeros(2, host.numel(), dtype=torch.int32)
        both[0, 1:] = torch.cumsum(lengths, 0)
        both[1, 1:] = torch.cumsum(padded, 0)
        self._cu_real, self.cu = both.to(device)

    def row_map(self, B):
        return _ew.row_map(B, self.T, self.total, None if self.cu is None else self._cu_real, self.cu)

    def pad_rows(self, *tensors):
        """[B, T, ...] tensors, or (tensor, fill value) pairs -> [B, padded T, ...]; one launch for all of them."""
        pairs = [t if isinstance(t, tuple) else (t, 0.0) for t in tensors]
        if not self.needed:
            out = [t for t, _ in pairs]
        else:
            out = _ew.rows_pad([t for t, _ in pairs], [f for _, f in pairs], self.row_map(pairs[0][0].shape[0]), self.total)
        return out[0] if len(out) == 1 else out

    def cut_rows(self, *tensors):
        """The inverse; for a fixed batch views of the padded tensors."""
        if not self.needed:
            out = tensors
        elif self.cu is None:
            out = _first_order(t[:, :self.T] for t in tensors)
        else:
            out = _first_order(_ew.rows_cut(tensors, self.row_map(1), self.T))
        return out[0] if len(out) == 1 else out

    # The output of a fixed batch is cut outside the autograd function, as a view that may be written in place like any
    # other; a packed one is gathered inside.
    def cut_output(self, o):
        return o if self.cu is None else self.cut_rows(o)

    def pad_output_grad(self, do):
        return do if self.cu is None else self.pad_rows(do)

    @property
    def index(self):
        """Padded row of every token of a packed batch."""
        if self._lengths is None:
            return None
        starts = self.cu[:-1].cpu().to(torch.int64)
        return torch.cat([torch.arange(int(n)) + int(s) for n, s in zip(self._lengths, starts)]).to(self.cu.device)

    def pad(self, x, fill=0.0):
        """x [B, T, ...] -> [B, padded T, ...]"""
        if x is None or not self.needed:
            return x
        if self.cu is None:
            tail = x.new_full((x.shape[0], self.total - self.T) + tuple(x.shape[2:]), fill)
            return torch.cat([x, tail], 1)
        return x.new_full((x.shape[0], self.total) + tuple(x.shape[2:]), fill).index_copy(1, self.index, x)

    def cut(self, o):
        if not self.needed:
            return o
        return o[:, :self.T] if self.cu is None else o.index_select(1, self.index)


def _common_checks(q, k, v, initial_state):
    if q.shape != k.shape:
        raise ValueError(f"q and k must have the same shape, got q={tuple(q.shape)} vs k={tuple(k.shape)}")
    if initial_state is not None and initial_state.dtype != torch.float32:
        raise ValueError("initial_state must be in float32.")
    if v.shape[2] != q.shape[2] and (v.shape[2] < q.shape[2] or v.shape[2] % q.shape[2] != 0):
        raise ValueError(f"the value heads ({v.shape[2]}) must be a multiple of the query/key heads ({q.shape[2]})")


class _Narrow:
    """Head dimensions below 128: the key and value channels are filled up with zeros (exact: a zero channel adds
    nothing to any product and its state rows stay zero) and outputs and states are cut back.  The scale keeps the
    caller's K.  Everything here is differentiable tensor code around the autograd function."""

    def __init__(self, q, v):
        self.K, self.V = q.shape[-1], v.shape[-1]
        if self.K > 128 or self.V > 128:
            raise ValueError(f"head dimensions above 128 are not supported (K={self.K}, V={self.V})")
        self.needed = self.K != 128 or self.V != 128

    def key(self, x):    # [..., K] -> [..., 128]
        return x if x is None or not self.needed else torch.nn.functional.pad(x, (0, 128 - self.K))

    def value(self, x):  # [..., V] -> [..., 128]
        return x if x is None or not self.needed else torch.nn.functional.pad(x, (0, 128 - self.V))

    def state(self, h, v_first=False):  # [N,H,K,V] (or [N,H,V,K]) -> [N,H,128,128]
        if h is None or not self.needed:
            return h
        last, first = (self.K, self.V) if v_first else (self.V, self.K)
        return torch.nn.functional.pad(h, (0, 128 - last, 0, 128 - first))

    def cut(self, o, final_state, v_first=False):
        if not self.needed:
            return o, final_state
        if final_state is not None:
            final_state = final_state[..., :self.V, :self.K] if v_first else final_state[..., :self.K, :self.V]
        return o[..., :self.V], final_state


def _groups(q, v):
    """Grouped value heads (HV = G * H; value head hv reads query/key head hv // G, as in FLA's kernels): the front pass
    repeats q and k to HV heads and its backward sums dq and dk over each group, so the kernels see equal head counts;
    the price is G copies of q and k."""
    return v.shape[2] // q.shape[2]


@torch.compiler.disable
def chunk_kda(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=False,
              use_qk_l2norm_in_kernel=False, use_gate_in_kernel=False, use_beta_sigmoid_in_kernel=False,
              allow_neg_eigval=False, safe_gate=False, lower_bound=None, disable_recompute=False,
              return_intermediate_states=False, state_v_first=False, cu_seqlens=None, cu_seqlens_cpu=None,
              cp_context=None, use_graph=False, max_num_seqs=None, **kwargs):
    """KDA (per-channel gated delta rule).  q,k [B,T,H,128] BF16, v [B,T,H,128], g [B,T,H,128] per-step
    natural-log decay (or, with ``use_gate_in_kernel``, the raw gate input together with ``A_log`` [H] and the optional
    ``dt_bias`` [H*128] keyword arguments), beta [B,T,H].  Returns (o, final_state)."""
    _common_checks(q, k, v, initial_state)
    if allow_neg_eigval and not use_beta_sigmoid_in_kernel:
        raise ValueError("`allow_neg_eigval=True` requires `use_beta_sigmoid_in_kernel=True`.")
    A_log, dt_bias = kwargs.get("A_log"), kwargs.get("dt_bias")
    if use_gate_in_kernel:
        if A_log is None:
            raise ValueError("A_log must be provided when use_gate_in_kernel=True.")
        if lower_bound is not None:
            raise ValueError("rewy_b200 chunk_kda: the lower_bound gate law belongs to safe_gate, which is not supported")
    if scale is None:
        scale = k.shape[-1] ** -0.5
    nw = _Narrow(q, v)
    if nw.needed:
        if use_gate_in_kernel:
            raise ValueError("rewy_b200 chunk_kda: the fused gate needs K = 128 (dt_bias is laid out per channel)")
        q, k, g, v, initial_state = nw.key(q), nw.key(k), nw.key(g), nw.value(v), nw.state(initial_state, state_v_first)
    rg = _Ragged(q.shape[1], q.device, cu_seqlens, cu_seqlens_cpu)
    if rg.needed:
        cu_seqlens = rg.cu
    o, final_state = ChunkKDAFunction.apply(q, k, v, g, beta, A_log, dt_bias, scale, initial_state, output_final_state,
                                            use_qk_l2norm_in_kernel, use_gate_in_kernel, use_beta_sigmoid_in_kernel,
                                            allow_neg_eigval, disable_recompute, state_v_first, _packed(cu_seqlens, q), rg,
                                            _groups(q, v))
    return nw.cut(o if rg.cu is not None else rg.cut(o), final_state, state_v_first)


@torch.compiler.disable
def chunk_gdn2(q, k, v, g, b, w, scale=None, initial_state=None, output_final_state=False,
               use_qk_l2norm_in_kernel=False, use_gate_in_kernel=False, cu_seqlens=None, cu_seqlens_cpu=None,
               safe_gate=False, lower_bound=None, disable_recompute=False, return_intermediate_states=False,
               state_v_first=False, cp_context=None, **kwargs):
    """GDN2 (vector erase gate b [B,T,H,128], vector write gate w [B,T,H,128]).  Returns (o, final_state)."""
    _common_checks(q, k, v, initial_state)
    if scale is None:
        scale = k.shape[-1] ** -0.5
    nw = _Narrow(q, v)
    if nw.needed:
        q, k, g, b = nw.key(q), nw.key(k), nw.key(g), nw.key(b)
        v, w, initial_state = nw.value(v), nw.value(w), nw.state(initial_state, state_v_first)
    rg = _Ragged(q.shape[1], q.device, cu_seqlens, cu_seqlens_cpu)
    if rg.needed:
        cu_seqlens = rg.cu
    o, final_state = ChunkGDN2Function.apply(q, k, v, g, b, w, scale, initial_state, output_final_state,
                                             use_qk_l2norm_in_kernel, disable_recompute, state_v_first,
                                             _packed(cu_seqlens, q), rg,
                                            _groups(q, v))
    return nw.cut(o if rg.cu is not None else rg.cut(o), final_state, state_v_first)


@torch.compiler.disable
def chunk_gated_delta_rule(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=False,
                           use_qk_l2norm_in_kernel=False, use_beta_sigmoid_in_kernel=False, allow_neg_eigval=False,
                           state_v_first=False, cu_seqlens=None, cu_seqlens_cpu=None, chunk_indices=None,
                           cp_context=None, **kwargs):
    """Gated DeltaNet (scalar per-head gate g [B,T,H]).  Returns (o, final_state)."""
    _common_checks(q, k, v, initial_state)
    if scale is None:
        scale = k.shape[-1] ** -0.5
    nw = _Narrow(q, v)
    if nw.needed:
        q, k, v, initial_state = nw.key(q), nw.key(k), nw.value(v), nw.state(initial_state, state_v_first)
    rg = _Ragged(q.shape[1], q.device, cu_seqlens, cu_seqlens_cpu)
    if rg.needed:
        cu_seqlens = rg.cu
    o, final_state = ChunkGatedDeltaRuleFunction.apply(q, k, v, g, beta, scale, initial_state, output_final_state,
                                                       use_qk_l2norm_in_kernel, use_beta_sigmoid_in_kernel,
                                                       allow_neg_eigval, state_v_first, _packed(cu_seqlens, q), rg,
                                            _groups(q, v))
    return nw.cut(o if rg.cu is not None else rg.cut(o), final_state, state_v_first)


@torch.compiler.disable
def chunk_delta_rule(q, k, v, beta, scale=None, initial_state=None, output_final_state=False,
                     use_qk_l2norm_in_kernel=False, cu_seqlens=None, cu_seqlens_cpu=None, **kwargs):
    """DeltaNet (ungated delta rule).  Returns (o, final_state)."""
    _common_checks(q, k, v, initial_state)
    if scale is None:
        scale = k.shape[-1] ** -0.5
    nw = _Narrow(q, v)
    if nw.needed:
        q, k, v, initial_state = nw.key(q), nw.key(k), nw.value(v), nw.state(initial_state)
    rg = _Ragged(q.shape[1], q.device, cu_seqlens, cu_seqlens_cpu)
    if rg.needed:
        cu_seqlens = rg.cu
    o, final_state = ChunkDeltaRuleFunction.apply(q, k, v, beta, scale, initial_state, output_final_state,
                                                  use_qk_l2norm_in_kernel, _packed(cu_seqlens, q), rg,
                                            _groups(q, v))
    return nw.cut(o if rg.cu is not None else rg.cut(o), final_state)
