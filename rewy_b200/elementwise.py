"""Element-wise stages of the autograd wrappers, bound to the CUDA library.

These are what the reference's autograd functions run around the core operator
(src/fast_delta_rule/_compat/kda.py:56-63 and :202-210: FLA ``l2norm_fwd`` / ``l2norm_bwd``,
``fused_beta_sigmoid`` / ``fused_beta_sigmoid_bwd``; ``kda_gate_chunk_cumsum`` / ``kda_gate_bwd`` inside
``chunk_kda_fwd`` / ``chunk_kda_bwd`` when ``use_gate_in_kernel`` is set).  One CUDA pass each; there is no
CPU or PyTorch fallback: non-CUDA tensors raise.
"""
import torch

from . import _capi


def _need_cuda(*tensors):
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise RuntimeError("rewy_b200 element-wise stages need CUDA tensors (there is no CPU fallback)")


def _stream(t):
    return _capi.current_stream(t.device)


def _as_input(x):
    """BF16 and FP32 are read directly; anything else is converted to FP32 first."""
    if x.dtype not in (torch.bfloat16, torch.float32):
        x = x.float()
    return x.contiguous(), int(x.dtype == torch.float32)


def _aligned(x):
    """Contiguous and 16-byte aligned."""
    x = x.contiguous()
    return x if x.data_ptr() % 16 == 0 else x.clone()


def l2norm_fwd(x, eps=1e-6):
    """x BF16 [..., 128] -> (y BF16, rstd FP32 [...])."""
    _need_cuda(x)
    if x.dtype != torch.bfloat16 or x.shape[-1] != 128:
        raise RuntimeError("rewy_b200 l2norm: expects BF16 rows of 128 values")
    x = x.contiguous()
    y = torch.empty_like(x)
    rstd = torch.empty(x.shape[:-1], dtype=torch.float32, device=x.device)
    with torch.cuda.device(x.device):
        _capi.check(_capi.load().rewy_l2norm_fwd(_capi.ptr(x), _capi.ptr(y), _capi.ptr(rstd), x.numel() // 128, eps,
                                                 _stream(x)), "rewy_l2norm_fwd")
    return y, rstd


def l2norm_bwd(y, rstd, dy):
    """Gradient of the normalisation, written in BF16 (the cast to the input dtype is part of the pass)."""
    _need_cuda(y, rstd, dy)
    if dy.dtype not in (torch.bfloat16, torch.float32):
        dy = dy.float()
    y, dy, rstd = y.contiguous(), dy.contiguous(), rstd.contiguous()
    dx = torch.empty_like(y)
    with torch.cuda.device(y.device):
        _capi.check(_capi.load().rewy_l2norm_bwd(_capi.ptr(y), _capi.ptr(rstd), _capi.ptr(dy),
                                                 int(dy.dtype == torch.float32), _capi.ptr(dx), y.numel() // 128,
                                                 _stream(y)), "rewy_l2norm_bwd")
    return dx


def beta_sigmoid_fwd(x, scale=1.0):
    """scale * sigmoid(x) in the dtype of x (BF16 logits give a BF16 beta, like the reference's fused sigmoid)."""
    _need_cuda(x)
    xin, is_f32 = _as_input(x)
    y16 = torch.empty_like(xin) if not is_f32 else None
    y32 = torch.empty(xin.shape, dtype=torch.float32, device=x.device) if is_f32 else None
    with torch.cuda.device(x.device):
        _capi.check(_capi.load().rewy_beta_sigmoid_fwd(_capi.ptr(xin), is_f32, _capi.ptr(y32), _capi.ptr(y16), xin.numel(),
                                                       float(scale), _stream(x)), "rewy_beta_sigmoid_fwd")
    return y32 if is_f32 else y16


def beta_sigmoid_bwd(x, dy, scale=1.0):
    """dx (FP32) for y = scale * sigmoid(x); dy FP32."""
    _need_cuda(x, dy)
    xin, is_f32 = _as_input(x)
    dy = dy.float().contiguous()
    dx = torch.empty(xin.shape, dtype=torch.float32, device=x.device)
    with torch.cuda.device(x.device):
        _capi.check(_capi.load().rewy_beta_sigmoid_bwd(_capi.ptr(xin), is_f32, _capi.ptr(dy), _capi.ptr(dx), xin.numel(),
                                                       float(scale), _stream(x)), "rewy_beta_sigmoid_bwd")
    return dx


def gate_cumsum_fwd(g, A_log=None, dt_bias=None):
    """g [B,T,H,128] (BF16 or FP32).  Returns the chunk-local cumulative gate in log2 units (FP32).  With ``A_log`` the KDA
    gate activation -exp(A_log[h]) * softplus(g + dt_bias[h*128+k]) is applied first (``dt_bias`` optional)."""
    _need_cuda(g, A_log, dt_bias)
    B, T, H, K = g.shape
    if K != 128 or T % 64:
        raise RuntimeError("rewy_b200 gate cumsum: expects [B,T,H,128] with T a multiple of 64")
    gin, is_f32 = _as_input(g)
    out = torch.empty(gin.shape, dtype=torch.float32, device=g.device)
    a = None if A_log is None else A_log.float().contiguous().view(-1)
    bias = None if dt_bias is None else dt_bias.float().contiguous().view(-1)
    if a is not None and a.numel() != H or bias is not None and bias.numel() != H * 128:
        raise RuntimeError("rewy_b200 gate cumsum: A_log must hold H values and dt_bias H*128")
    if a is None and bias is not None:
        raise RuntimeError("rewy_b200 gate cumsum: dt_bias needs A_log")
    with torch.cuda.device(g.device):
        _capi.check(_capi.load().rewy_gate_cumsum_fwd(_capi.ptr(gin), is_f32, _capi.ptr(a), _capi.ptr(bias), _capi.ptr(out),
                                                      None, B, T, H, _stream(g)), "rewy_gate_cumsum_fwd")
    return out


def gate_act_bwd(g_raw, A_log, dt_bias, dg, out_dtype=torch.float32):
    """Backward of the KDA gate activation.  dg: FP32 gradient of the activated per-step gate.
    Returns (dg_raw [B,T,H,128] in ``out_dtype``: FP32 or BF16, dA_log FP32 [H], ddt_bias FP32 [H*128] or None)."""
    _need_cuda(g_raw, A_log, dt_bias, dg)
    B, T, H, K = g_raw.shape
    gin, is_f32 = _as_input(g_raw)
    dg = dg.float().contiguous()
    a = A_log.float().contiguous().view(-1)
    bias = None if dt_bias is None else dt_bias.float().contiguous().view(-1)
    nt = T // 64
    dx = torch.empty(gin.shape, dtype=out_dtype, device=g_raw.device)
    fn = "rewy_gate_act_bwd_bf16" if out_dtype == torch.bfloat16 else "rewy_gate_act_bwd"
    dA_part = torch.empty(B * nt, H, dtype=torch.float32, device=g_raw.device)
    db_part = torch.empty(B * nt, H * 128, dtype=torch.float32, device=g_raw.device)
    with torch.cuda.device(g_raw.device):
        _capi.check(getattr(_capi.load(), fn)(_capi.ptr(gin), is_f32, _capi.ptr(a), _capi.ptr(bias), _capi.ptr(dg),
                                              _capi.ptr(dx), _capi.ptr(dA_part), _capi.ptr(db_part), B, T, H,
                                              _stream(g_raw)), fn)
    # the per-(batch, chunk) partial sums are added up in a fixed order (deterministic), as FLA's kda_gate_bwd does
    return dx, dA_part.sum(0), (db_part.sum(0) if dt_bias is not None else None)


def row_map(B, T, T_padded, cu=None, cu_padded=None):
    """Pairs B*T token rows with B*T_padded padded rows; ``cu``, ``cu_padded``: device int32 offsets of packed sequences."""
    m = _capi.RowMap()
    m.B, m.T, m.T_padded = B, T, T_padded
    if cu is not None:
        m.cu, m.cu_padded, m.num_seqs = _capi.ptr(cu), _capi.ptr(cu_padded), cu.numel() - 1
        m.keep = (cu, cu_padded)
    return m


def _pattern(fill, dtype):
    """8 bytes of the fill value in `dtype`."""
    if fill == 0:
        return 0
    one = torch.empty((), dtype=dtype).element_size()
    return int.from_bytes(bytes(torch.full((8 // one,), fill, dtype=dtype).view(torch.uint8).tolist()), "little")


def _need_rows(tensors, m, T):
    """The kernels take the number of rows from the map: a tensor with another one would be read past its end."""
    for t in tensors:
        if tuple(t.shape[:2]) != (m.B, T):
            raise RuntimeError(f"rewy_b200 rows: expected a tensor [{m.B}, {T}, ...], got {list(t.shape)}")


def _move_rows(fn, tensors, fills, m, T_in, T_out):
    _need_rows(tensors, m, T_in)
    _need_cuda(*tensors)
    src = [t.contiguous() for t in tensors]
    out = [torch.empty((t.shape[0], T_out) + tuple(t.shape[2:]), dtype=t.dtype, device=t.device) for t in src]
    items = (_capi.RowsItem * len(src))()
    for it, s, d, f in zip(items, src, out, fills):
        it.src, it.dst, it.fill = _capi.ptr(s), _capi.ptr(d), _pattern(f, s.dtype)
        it.row_bytes = s.numel() // (s.shape[0] * s.shape[1]) * s.element_size()
    with torch.cuda.device(src[0].device):
        _capi.check(getattr(_capi.load(), fn)(m, items, len(src), _stream(src[0])), fn)
    return out


def rows_pad(tensors, fills, m, T_padded):
    """[B, T, ...] tensors of any element type -> [B, T_padded, ...], `fills` in the added rows; one launch."""
    return _move_rows("rewy_rows_pad", tensors, fills, m, m.T, T_padded)


def rows_cut(tensors, m, T):
    """[B, T_padded, ...] -> [B, T, ...]; one launch."""
    return _move_rows("rewy_rows_cut", tensors, [0] * len(tensors), m, m.T_padded, T)


def qk_front_fwd(q, k, m, groups, normalize, eps=1e-6):
    """q, k BF16 [B,T,H,128] -> (BF16 [B,T_padded,H*groups,128] twice, rstd FP32 [B,T_padded,H] twice or None): L2
    normalisation, padding rows and the repeat of every head in one pass."""
    _need_rows((q, k), m, m.T)
    _need_cuda(q, k)
    if q.dtype != torch.bfloat16 or k.dtype != torch.bfloat16 or q.shape[-1] != 128:
        raise RuntimeError("rewy_b200 l2norm: expects BF16 rows of 128 values")
    if q.shape != k.shape:
        raise RuntimeError("rewy_b200 q/k front: q and k must have the same shape")
    q, k = _aligned(q), _aligned(k)
    B, _, H, _ = q.shape
    y = [torch.empty(B, m.T_padded, H * groups, 128, dtype=q.dtype, device=q.device) for _ in (q, k)]
    rstd = [torch.empty(B, m.T_padded, H, dtype=torch.float32, device=q.device) if normalize else None for _ in (q, k)]
    with torch.cuda.device(q.device):
        _capi.check(_capi.load().rewy_qk_front_fwd(m, _capi.ptr(q), _capi.ptr(k), _capi.ptr(y[0]), _capi.ptr(y[1]),
                                                   _capi.ptr(rstd[0]), _capi.ptr(rstd[1]), H, groups, eps, _stream(q)),
                    "rewy_qk_front_fwd")
    return (*y, *rstd)


def qk_front_bwd(yq, yk, rq, rk, dyq, dyk, m, groups):
    """Backward of qk_front_fwd: dy BF16 or FP32 [B,T_padded,H*groups,128] -> dq, dk BF16 [B,T,H,128]."""
    _need_rows((yq,), m, m.T_padded)
    if not yq.shape == yk.shape == dyq.shape == dyk.shape:
        raise RuntimeError("rewy_b200 q/k front backward: y and dy of q and k must have the same shape")
    _need_cuda(yq, yk, dyq, dyk)
    dyq, dyk = _aligned(dyq), _aligned(dyk)
    if rq is not None:   # read with the layout of the forward, which a saved-tensor hook need not give back
        yq, yk, rq, rk = _aligned(yq), _aligned(yk), rq.contiguous(), rk.contiguous()
    H = yq.shape[2] // groups
    dq, dk = (torch.empty(yq.shape[0], m.T, H, 128, dtype=torch.bfloat16, device=yq.device) for _ in range(2))
    with torch.cuda.device(yq.device):
        _capi.check(_capi.load().rewy_qk_front_bwd(m, _capi.ptr(yq), _capi.ptr(yk), _capi.ptr(rq), _capi.ptr(rk),
                                                   _capi.ptr(dyq), _capi.ptr(dyk), int(dyq.dtype == torch.float32),
                                                   _capi.ptr(dq), _capi.ptr(dk), H, groups, _stream(yq)),
                    "rewy_qk_front_bwd")
    return dq, dk
