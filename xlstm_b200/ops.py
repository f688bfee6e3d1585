"""Tensor-level entry points over the C ABI of ``include/xlstm_b200.h``.

PyTorch is used for device memory and streams only; all arithmetic happens in
the sm_100a kernels.  The host path of every call (argument checks, output
allocation, the parameter block, the launch on the current stream) is native
code, ``csrc/binding.cpp``; what is left here are the documented signatures and
the few cases that start from host data.  Nothing here falls back to PyTorch
math: unsupported inputs raise.
"""
from __future__ import annotations

from typing import Optional

import torch

from ._lib import native

_KERNELS = {"auto": 0, "chunkwise": 1, "recurrent": 2}
_CHUNKWISE_WHOLE = 3   # chunkwise, no document cut into parts


def status_word(device) -> torch.Tensor:
    """Per-device int32 word that kernels set when one of their bounded waits expires."""
    idx = torch.device(device).index
    if idx is None:
        idx = torch.cuda.current_device()
    return native().status_word(idx)


def _index(device) -> int:
    """CUDA device index of `device`; -1 for the host."""
    d = torch.device(device)
    return -1 if d.type != "cuda" else torch.cuda.current_device() if d.index is None else d.index


def check_device_status(device=None) -> None:
    """Synchronising check of the status word; raises if a kernel gave up on a wait."""
    w = status_word(device if device is not None else torch.cuda.current_device())
    v = int(w.item())
    if v != 0:
        w.zero_()
        raise RuntimeError(f"xlstm_b200 kernel reported device status {v} (a bounded wait expired)")


def prepare_cu_seqlens(cu_seqlens, B: int, S: int, device) -> tuple[torch.Tensor, int]:
    """Validate document offsets on the host and return (int32 device tensor, num_docs).

    Offsets index the flattened (B*S) token axis; they must start at 0, end at B*S, be
    non-decreasing, and no document may straddle two rows.  A tensor that already lives on
    the device is trusted as is (validating it would force a synchronisation).
    """
    if torch.is_tensor(cu_seqlens) and cu_seqlens.is_cuda:
        if cu_seqlens.dtype != torch.int32:
            raise ValueError("cu_seqlens on the device must be int32")
        return cu_seqlens.contiguous(), cu_seqlens.numel() - 1
    return native().document_offsets(cu_seqlens, B, S, _index(device))


def mlstm_sequence(q, k, v, i, f, c_initial=None, n_initial=None, m_initial=None, cu_seqlens=None,
                   eps: float = 1e-6, kernel: str = "auto"):
    """mLSTM over a sequence.  q,k (B,NH,S,DHQK), v (B,NH,S,DHV), i,f (B,NH,S).

    kernel: "chunkwise" (tcgen05), "recurrent" (fp32 recurrence) or "auto" (chunkwise when the
    shape/dtype is covered by it, else recurrent).  Returns h (B,NH,S,DHV) in q's dtype and the final
    fp32 state (c,n,m) with one row per document: c (N,NH,DHQK,DHV), n (N,NH,DHQK), m (N,NH,1).

    The chunkwise kernel cuts long documents into parts that run side by side, as many as the machine has room for.  A
    call gives the same bits from run to run, but the cut -- and with it the rounding of a document's h and state, within
    what bf16 operands give -- depends on the sizes of the whole call: B, S and the number of documents beside it.
    """
    code = _KERNELS.get(kernel)
    if code is None:
        raise ValueError(f"unknown kernel {kernel!r}")
    cu, nd = None, 0
    if cu_seqlens is not None and q.is_cuda:
        cu, nd = prepare_cu_seqlens(cu_seqlens, q.shape[0], q.shape[2], q.device)
    return native().mlstm_sequence(q, k, v, i, f, c_initial, n_initial, m_initial, cu, nd, eps, code)


_host_streams: dict[int, list] = {}


def mlstm_sequence_from_host(q, k, v, i, f, h_out, c_out, n_out=None, m_out=None, device=None, head_groups: Optional[int] = None,
                             eps: float = 1e-6):
    """Prefill whose inputs and outputs live in pinned HOST memory: q, k ``(B,NH,S,DHQK)``, v ``(B,NH,S,DHV)``, gates
    ``(B,NH,S)`` in, ``h_out (B,NH,S,DHV)``, ``c_out (B,NH,DHQK,DHV)`` (optionally n, m) out, zero initial state.

    Heads and batch rows are independent, so the call is cut into ``B x head_groups`` contiguous pieces that go round
    three streams: the upload of one piece overlaps the kernel and the download of the pieces before it (the link is
    full duplex), and the whole call takes about as long as its uploads alone.  Documents stay whole: the kernels hide
    behind the link either way, and cut into parts they slow the copies down (4 x 8192 tokens of 8 x 256/512: 11.95 ms,
    11.70 whole).  Returns when everything is enqueued; the caller's current stream waits for the last piece."""
    dev = torch.device(device if device is not None else "cuda")
    idx = dev.index if dev.index is not None else torch.cuda.current_device()
    dev = torch.device("cuda", idx)
    B, NH = q.shape[0], q.shape[1]
    if head_groups is None:   # pieces of a few tens of MB keep the link busy in both directions (measured: 4 groups of 2 heads at
        head_groups = next(g for g in (4, 2, 1) if NH % g == 0)   # the 7B head shape: 11.9 ms per 32 768 tokens; 2: 12.1; 8: 14.2)
    if NH % head_groups:
        raise ValueError(f"num_heads={NH} is not divisible by head_groups={head_groups}")
    for t in (q, k, v, i, f, h_out, c_out):
        if t.device.type != "cpu" or not t.is_pinned():
            raise ValueError("mlstm_sequence_from_host wants pinned host tensors")
    streams = _host_streams.setdefault(idx, [torch.cuda.Stream(device=dev) for _ in range(3)])
    cur = torch.cuda.current_stream(dev)
    for st in streams:
        st.wait_stream(cur)
    hg = NH // head_groups
    piece = 0
    for b in range(B):
        for g in range(head_groups):
            sl = (slice(b, b + 1), slice(g * hg, (g + 1) * hg))
            st = streams[piece % len(streams)]
            piece += 1
            with torch.cuda.stream(st):
                dq, dk, dv, di, df = [t[sl].to(dev, non_blocking=True) for t in (q, k, v, i, f)]
                h, (c, n, m) = native().mlstm_sequence(dq, dk, dv, di, df, None, None, None, None, 0, eps, _CHUNKWISE_WHOLE)
                h_out[sl].copy_(h, non_blocking=True)
                c_out[sl].copy_(c, non_blocking=True)
                if n_out is not None:
                    n_out[sl].copy_(n, non_blocking=True)
                if m_out is not None:
                    m_out[sl].copy_(m, non_blocking=True)
                for t in (dq, dk, dv, di, df, h, c, n, m):
                    t.record_stream(st)
    for st in streams:
        cur.wait_stream(st)


def prepare_slots(slot, B: int, n_slots: int, device) -> torch.Tensor:
    """Pool rows of the B decode streams as the int32 device vector the step kernel reads.

    A host tensor or list is checked here: one entry per stream, every entry below ``n_slots``, no row named by two
    active streams (negative entries mark inactive streams and may repeat).  A tensor that already lives on the device
    must be a (B,) integer vector; its values cannot be inspected without a synchronisation, so the kernel itself
    skips entries outside the pool and reports them through the status word (``check_device_status``)."""
    if torch.is_tensor(slot) and slot.is_cuda:
        if slot.dim() != 1 or slot.numel() != B or slot.dtype not in (torch.int32, torch.int64):
            raise ValueError(f"slot must be a ({B},) int32 (or int64) vector, got {tuple(slot.shape)} {slot.dtype}")
        if slot.device != torch.device(device):
            raise ValueError("slot lives on another device than the inputs")
        return slot.to(torch.int32).contiguous()
    return native().slot_vector(slot, B, n_slots, _index(device))


def _step_slots(slot, q, c):
    if slot is None or (torch.is_tensor(slot) and slot.is_cuda) or not q.is_cuda:
        return slot
    if c is None:
        raise ValueError("`slot` addresses rows of a state pool: pass c, n, m")
    return prepare_slots(slot, q.shape[0], c.shape[0], q.device)


def mlstm_step(q, k, v, i, f, c, n, m, slot=None, eps: float = 1e-6, inplace: bool = True):
    """One decode step.  q,k (B,NH,DHQK), v (B,NH,DHV), i,f (B,NH[,1]); state pool c (N,NH,DHQK,DHV),
    n (N,NH,DHQK), m (N,NH[,1]) fp32; ``slot`` (B,) selects each stream's pool row (default: row b; a negative
    entry marks an inactive stream whose pool rows stay untouched; see :func:`prepare_slots`).

    With ``inplace`` the large C state is updated where it lives and the SAME tensor object is returned,
    so a caller that copies the returned state back into its own buffers (xlstm_large/model.py:221-225)
    performs a no-op for C.  n and m are always returned as new small tensors (several thread blocks
    read the old values while one writes).  Without a pool (c is None) the state starts from zero.
    """
    return native().mlstm_step(q, k, v, i, f, c, n, m, slot if slot is None else _step_slots(slot, q, c), eps, bool(inplace))


def mlstm_decode_cell(q, k, v, gates_raw, gate_bias, gate_cap: float, ogate, norm_weight, c, n, m, slot=None,
                      eps: float = 1e-6, norm_eps: float = 1e-6):
    """The cell part of one decode step of the mLSTM layer in ONE kernel: soft cap of the gate pre-activations
    (xlstm/xlstm_large/model.py:389-394, fp32 arithmetic), the step of :func:`mlstm_step` (C updated in place), and the
    per-head norm + weight + output gate behind it (model.py:435-449).

    q,k (B,NH,DHQK), v (B,NH,DHV) as for the step; ``gates_raw`` (B, 2*NH): the projection's input-gate columns of all
    heads, then its forget-gate columns (a column slice of the stacked projection output is fine); ``gate_bias`` (2*NH)
    or None; ``ogate`` (B, NH*DHV); ``norm_weight`` (NH*DHV).  Returns (B, NH*DHV), the input of out_proj, and the
    state like :func:`mlstm_step`."""
    return native().mlstm_decode_cell(q, k, v, gates_raw, gate_bias, gate_cap, ogate, norm_weight, c, n, m,
                                      slot if slot is None else _step_slots(slot, q, c), eps, norm_eps)


def slstm_forward(wx, R, bias, state0=None, cu_seqlens=None, train_cache: bool = False):
    """sLSTM over a sequence.  wx (B,S,4*H) gate-major [i|f|z|o] each (NH,DH); R (NH,DH,4,DH); bias (NH,4,DH);
    state0 (4,B,H) ordered (h,c,n,m) or None.  Returns h (B,NH,S,DH) in wx's dtype and the final fp32 state; with
    ``train_cache`` also the opaque cache ``slstm_backward`` needs (no document offsets then)."""
    cu, nd = None, 0
    if cu_seqlens is not None and wx.is_cuda:
        cu, nd = prepare_cu_seqlens(cu_seqlens, wx.shape[0], wx.shape[1], wx.device)
    return native().slstm_forward(wx, R, bias, state0, cu, nd, bool(train_cache))


def slstm_backward(cache, R, dh, dstate_out=None, state0=None):
    """Backward through time of ``slstm_forward(..., train_cache=True)``: ``cache`` from that call, R (NH,DH,4,DH),
    dh (B,NH,S,DH) the gradient of its h, dstate_out (4,B,H) the gradient of its final state (m's entry is ignored)
    or None, state0 its initial state or None.  Returns dwx (B,S,4*H) in bf16 and dstate0 (4,B,H) fp32 (zero for m).
    Replaces sLSTMFunc.backward (xlstm/blocks/slstm/src/cuda/slstm.cc:137-254) up to the two sums ``slstm_weight_grads``
    forms."""
    return native().slstm_backward(cache, R, dh, dstate_out, state0)


def _weight_grads_native(dw, h, state0) -> bool:
    """Whether ``slstm_weight_grads`` runs on its kernel: contiguous, aligned bf16 tensors of one device, and nobody
    who would have to see the single operators (autograd in either direction, function transforms, dispatch modes)."""
    ts = [dw, h] + ([] if state0 is None else [state0])
    if any(type(t) is not torch.Tensor or t.device != h.device for t in ts) or not h.is_cuda or h.numel() == 0:
        return False
    if torch.is_grad_enabled() and any(t.requires_grad for t in ts):
        return False
    if torch._C._functorch.peek_interpreter_stack() is not None or torch._C._len_torch_dispatch_stack() or torch.autograd.forward_ad._current_level >= 0:
        return False
    return (h.shape[-1] in (64, 128, 256) and h.shape[1] <= 4096 and
            all(t.dtype == torch.bfloat16 and t.is_contiguous() and t.data_ptr() % 16 == 0 for t in (dw, h)))


def slstm_weight_grads(dwx, h, state0=None):
    """Gradients of the recurrent matrix and the bias from the backward kernel's output: with h_{t-1} the forward's h
    shifted by one step (h_{-1} from state0), dR[n,k,g,u] = sum_{b,t} h_{t-1}[b,n,k] dwx[b,t,g,n,u] and
    dbias[n,g,u] = sum_{b,t} dwx[b,t,g,n,u] (the reference forms the same products after its time loop,
    slstm_backward.cu).  fp32 results: (NH,DH,4,DH) and (NH,4,DH).  What the backward kernel writes goes through one
    tensor-core kernel; anything else (other devices, dtypes and head sizes, differentiable or traced calls) is formed by
    plain batched matrix products."""
    B, NH, S, DH = h.shape
    dw = dwx.reshape(B, S, 4, NH, DH)
    if _weight_grads_native(dw, h, state0):
        h0 = None if state0 is None else state0[0].reshape(B, NH, DH).to(torch.bfloat16).contiguous()
        return native().slstm_weight_grads(dw, h, h0)

    def mm(a, b):   # fp32 result; half-precision operands stay as they are where the GEMM library accumulates in fp32
        if a.is_cuda and a.dtype in (torch.bfloat16, torch.float16):
            try:
                return torch.bmm(a, b, out_dtype=torch.float32)
            except (TypeError, NotImplementedError, RuntimeError):
                pass
        return torch.bmm(a.float(), b.float())

    dR = torch.zeros(NH, DH, 4 * DH, dtype=torch.float32, device=dwx.device)
    if S > 1:   # steps 1 .. S-1 pair h_{t-1} = h[t-1] with dwx[t]: two shifted views, no shifted copy of h
        a = h[:, :, :-1].permute(1, 3, 0, 2).reshape(NH, DH, B * (S - 1)).to(dwx.dtype)      # (NH, DH_in, B*(S-1))
        b = dw[:, 1:].permute(3, 0, 1, 2, 4).reshape(NH, B * (S - 1), 4 * DH)                 # (NH, B*(S-1), 4*DH_out)
        dR = mm(a, b)
    if state0 is not None:   # step 0 pairs the initial h with dwx[0]
        a0 = state0[0].reshape(B, NH, DH).permute(1, 2, 0).to(dwx.dtype).contiguous()         # (NH, DH_in, B)
        b0 = dw[:, 0].permute(2, 0, 1, 3).reshape(NH, B, 4 * DH)                              # (NH, B, 4*DH_out)
        dR = dR + mm(a0, b0)
    db = dw.sum(dim=(0, 1), dtype=torch.float32).permute(1, 0, 2).contiguous()
    return dR.reshape(NH, DH, 4, DH), db


class SlstmFunction(torch.autograd.Function):
    """``slstm_forward`` with a backward pass: h, last = SlstmFunction.apply(wx, R, bias, state0)."""

    @staticmethod
    def forward(ctx, wx, R, bias, state0):
        h, last, cache = slstm_forward(wx, R, bias, state0, train_cache=True)
        ctx.save_for_backward(cache, R, h, state0 if state0 is not None else torch.empty(0, device=wx.device))
        ctx.has_state0 = state0 is not None
        ctx.dtypes = (wx.dtype, R.dtype, bias.dtype, None if state0 is None else state0.dtype)
        ctx.bias_shape = bias.shape
        return h, last

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dh, dlast):
        cache, R, h, s0 = ctx.saved_tensors
        s0 = s0 if ctx.has_state0 else None
        if dh is None:
            dh = torch.zeros_like(h)
        dwx, ds0 = slstm_backward(cache, R, dh, dlast, s0)
        dR = db = None
        if ctx.needs_input_grad[1] or ctx.needs_input_grad[2]:
            dR, db = slstm_weight_grads(dwx, h, s0)
            dR = dR.to(ctx.dtypes[1])
            db = db.reshape(ctx.bias_shape).to(ctx.dtypes[2])
        return (dwx.to(ctx.dtypes[0]), dR, db, ds0.to(ctx.dtypes[3]) if ctx.has_state0 else None)


def add_rmsnorm(x, weight, y=None, eps: float = 1e-6, inplace: bool = False):
    """``x_new = x + y`` (when ``y`` is given) and ``RMSNorm(x_new) * weight`` in one pass; returns
    ``(x_new, normed)``.  This is the residual add of one sub-block fused with the pre-norm of the next
    (xlstm/xlstm_large/model.py:499-510; RMSNorm: components.py:70-97), with the reference's rounding points.
    ``x`` is (..., D) with contiguous rows; ``inplace`` writes ``x_new`` over ``x``."""
    return native().add_rmsnorm(x, weight, y, eps, bool(inplace))


def headnorm_gate(h, o_preact, weight, eps: float = 1e-6):
    """``sigmoid(o_preact) * (LayerNorm over DH of h, per head) * weight`` -> (B, S, NH*DH).

    ``h`` is the cell output (B, NH, S, DH), read through its strides (no transpose copy); ``o_preact`` is
    (B, S, NH*DH), possibly a column slice of a wider projection output, or None: then the result is the plain
    per-head group norm ``(h - mean) * rstd * weight`` rounded once, the epilogue of the reference's sLSTM layer
    (``MultiHeadLayerNorm``, xlstm/components/ln.py:52-68; xlstm/blocks/slstm/layer.py:157).  Follows MultiHeadLayerNorm.forward
    and the output gate of the reference layer (components.py:188-242, xlstm_large/model.py:445-449)."""
    return native().headnorm_gate(h, o_preact, weight, eps)


def soft_cap(x, cap: float, out_float32: bool = False, float32_math: bool = False, bias=None):
    """``cap * tanh(x / cap)`` in one kernel with the rounding of the reference's eager ``soft_cap``
    (xlstm/xlstm_large/components.py:5-22).  ``out_float32`` returns the result (rounded to ``x.dtype``) as
    float32, the type the cell kernels take for gate pre-activations; with ``float32_math`` as well the
    quotient, tanh and product are not rounded to ``x.dtype`` in between (gates kept in fp32 in a bf16 model).
    ``x`` may be a column slice of a wider matrix (last dimension contiguous, one row stride); ``bias`` (last-dimension
    sized) is added first, which lets the gate projection ride in the q/k/v/o GEMM without its own launch."""
    if float32_math and not out_float32:
        raise ValueError("soft_cap: float32_math needs out_float32")
    return native().soft_cap(x, cap, 2 if float32_math else int(bool(out_float32)), bias)


def swiglu(gz):
    """``silu(gz[..., :F]) * gz[..., F:]`` in one kernel, the feed-forward's gating on the output of one projection that
    stacks ``proj_up_gate`` on ``proj_up`` (xlstm/xlstm_large/model.py:268-277), with the eager sequence's rounding."""
    return native().swiglu(gz)


def causal_conv1d(x, weight, bias=None, cu_seqlens=None, silu: bool = True):
    """Depthwise causal convolution over time and (by default) SiLU, the front of the reference's sLSTM layer
    (``CausalConv1d.forward``, xlstm/components/conv.py:110-129; activation xlstm/blocks/slstm/layer.py:133-142).

    x (B, S, F); weight (F, K) or the ``nn.Conv1d`` weight (F, 1, K); bias (F) or None.  With ``cu_seqlens`` (offsets on
    the flattened (B*S) axis) no tap reaches across a document boundary -- the reference's module knows rows only."""
    cu, nd = None, 0
    if cu_seqlens is not None and x.is_cuda and x.dim() == 3:
        cu, nd = prepare_cu_seqlens(cu_seqlens, x.shape[0], x.shape[1], x.device)
    return native().causal_conv1d(x, weight, bias, cu, nd, bool(silu))


def headwise_proj(inputs, weights, in_sel=None):
    """Up to four headwise (block-diagonal) projections in one launch, stacked in the sLSTM cell's input layout: the
    reference's ``LinearHeadwiseExpand.forward`` per gate (xlstm/components/linear_headwise.py:75-82, bias-free as the layer
    builds them) and the ``torch.cat`` of xlstm/blocks/slstm/layer.py:145-154.

    ``inputs``: one or two (..., NH*DH) bfloat16 tensors; ``weights``: list of (NH, DH, DH) parameters, slot order;
    ``in_sel[s]``: which input slot s projects (default: all the first).  Returns (..., len(weights) * NH * DH): slot-major,
    then head, then feature -- what the cell views as (.., 4, NH, DH)."""
    inputs = [inputs] if isinstance(inputs, torch.Tensor) else list(inputs)
    weights = list(weights)
    return native().headwise_proj(inputs, weights, [0] * len(weights) if in_sel is None else [int(i) for i in in_sel])


ROWS_LINEAR_MAX = 16   # rows of x that ``rows_linear`` takes


def rows_linear(x, w, w_ahead: bool = False):
    """``F.linear(x, w)`` for at most 16 rows of x (decoding): bf16 x (..., K) and w (N, K), K a multiple of 8, fp32
    accumulation; bound by the stream of w.  ``w_ahead`` is for a caller who knows every launch on the stream: w is then read
    ahead of the end of the kernel directly in front, which must not be the one that writes w (a weight that stays as it is
    between steps; a w computed, cast or copied on the line before is not one)."""
    return native().rows_linear(x, w, bool(w_ahead))


def softcap_argmax(logits, cap: float):
    """Greedy tokens of un-capped logits: ``argmax(soft_cap(logits, cap), dim=-1)`` with the reference's rounding and
    tie rule (xlstm/xlstm_large/model.py:149-151, generate.py:13-15) in one kernel.  ``logits`` is (..., V) with
    contiguous rows; returns int64 of shape ``logits.shape[:-1]``.  The kernel's scratch area is allocated once per
    device (and grown when more rows come) and shared by all calls on that device's streams in issue order."""
    return native().softcap_argmax(logits, cap)
