"""Python API of the sm_100a gdn_chunk forward, mirroring the reference project's
``gdn_qsa_sm80/gdn_chunk_interface.py`` (same names, argument order and error behaviour).

Differences from the reference, all additive:
  * ``initial_state`` keyword (fp32 or bf16 ``[B,Hv,128,128]``) and an fp32 ``final_state``,
    as in the reference's torch definition (``reference/gdn_chunk_ref.py:20-31``);
  * ``GDN_CHUNK`` is 64 (the reference's CUDA path uses 16, its torch definition 64);
  * g and beta may be bf16 or fp32;
  * the result is exact for every gate distribution (the reference's production fast path
    is an approximation that holds only under strong decay, ``csrc/gdn_chunk/gdn_ops.cu:845-848``).

PyTorch is used only for device memory and the current stream; all arithmetic happens in the
CUDA library behind the C ABI.  There is no CPU or eager fallback.
"""

from __future__ import annotations

import os
import threading

import torch

from . import _lib

__all__ = ["gdn_chunk", "gdn_chunk_host", "gdn_chunk_varlen", "rmsnorm_gated", "gdn_chunk_twolevel", "gdn_chunk_reference", "scan_transfers", "GDN_D", "GDN_CHUNK"]

GDN_D = 128      # head dim (compile-time constant in the kernels)
GDN_CHUNK = 64   # intra-chunk size (compile-time constant)

_scratch = {}
_scratch_lock = threading.Lock()   # growing one: this dictionary and the front end hold the same buffer


def _check_inputs(q, k, v, g, beta):
    # same checks and messages as the reference's _check_inputs (gdn_chunk_interface.py:19-32)
    if q.dim() != 4 or q.size(3) != GDN_D:
        raise ValueError(f"q must be [B,S,Hk,{GDN_D}], got {tuple(q.shape)}")
    if k.shape != q.shape:
        raise ValueError(f"k must match q, got q={tuple(q.shape)} k={tuple(k.shape)}")
    B, S, Hk, _ = q.shape
    if v.dim() != 4 or v.size(3) != GDN_D or v.shape[:2] != (B, S):
        raise ValueError(f"v must be [B,S,Hv,{GDN_D}], got {tuple(v.shape)}")
    Hv = v.size(2)
    if g.shape != (B, S, Hv) or beta.shape != (B, S, Hv):
        raise ValueError("g and beta must be [B,S,Hv]")
    if Hv % Hk != 0:
        raise ValueError(f"Hv must be a multiple of Hk, got Hk={Hk} Hv={Hv}")
    return B, S, Hk, Hv


def _check_output_gate(output_gate, out_shape, dev):
    if len(output_gate) == 2:
        z, weight = output_gate
        eps = 1e-6
    else:
        z, weight, eps = output_gate
    if tuple(z.shape) != tuple(out_shape):
        raise ValueError(f"output_gate z must be {tuple(out_shape)}, got {tuple(z.shape)}")
    if weight.numel() != GDN_D:
        raise ValueError(f"output_gate weight must have {GDN_D} elements")
    z = z.to(device=dev, dtype=torch.bfloat16).contiguous()
    weight = weight.to(device=dev, dtype=torch.bfloat16).contiguous()
    return z, weight, float(eps)


def rmsnorm_gated(y, z, weight, eps=1e-6, out=None):
    """out[i] = RMSNorm(y)[i] * weight[i] * silu(z[i]) per 128-wide row: the reference's operator of the same name
    (gdn_qsa_sm80/output_gate_interface.py:15-27).  y, z: [N, 128] (any leading shape) bf16 CUDA tensors;
    weight: [128] bf16.  `out` may be y (in place)."""
    if y.shape != z.shape or y.size(-1) != GDN_D or weight.numel() != GDN_D:
        raise ValueError(f"y and z must be [..., {GDN_D}] with equal shapes and weight [{GDN_D}]")
    if not y.is_cuda:
        raise RuntimeError("rmsnorm_gated needs CUDA tensors (sm_100a); there is no CPU path")
    y, z, weight = (x.to(torch.bfloat16).contiguous() for x in (y, z, weight))
    if out is None:
        out = torch.empty_like(y)
    elif out.shape != y.shape or out.dtype != torch.bfloat16 or not out.is_contiguous():
        raise ValueError("out must be a contiguous bf16 tensor shaped like y")
    with torch.cuda.device(y.device):
        st = _lib.load().gdn_rmsnorm_gated_sm100(y.data_ptr(), z.data_ptr(), weight.data_ptr(), out.data_ptr(),
                                                 y.numel() // GDN_D, float(eps),
                                                 torch.cuda.current_stream(y.device).cuda_stream)
    _lib.check(st, "gdn_rmsnorm_gated_sm100")
    return out


def _scratch_for(device, nbytes):
    # one buffer per (device, stream): calls on different streams may overlap on the GPU and must not share scratch
    key = (device.index, torch.cuda.current_stream(device).cuda_stream)
    with _scratch_lock:
        buf = _scratch.get(key)
        if buf is None or buf.numel() < nbytes:
            buf = torch.empty(max(nbytes, 256), dtype=torch.uint8, device=device)
            _scratch[key] = buf
            front = _lib.frontend()
            if front is not None:
                front.note_scratch(*key, buf)
    return buf


_native_forward = None


def _native():
    """The front end's forward(): the plain call (CUDA tensors of the current device, contiguous, in the kernels' dtypes)
    without this module's interpreter time; it returns None for everything else, which then takes _forward()."""
    global _native_forward
    if _native_forward is None:
        front = _lib.frontend()
        if front is None:
            _native_forward = lambda *args: None
            return _native_forward
        front.set_grow_scratch(lambda index, nbytes: _scratch_for(torch.device("cuda", index), nbytes))
        _native_forward = front.forward
    return _native_forward


def _flags(l2norm, gate_act):
    return (_lib.FLAG_QK_L2NORM if l2norm else 0) | (_lib.FLAG_GATE_ACTIVATIONS if gate_act else 0)


def _forward(q, k, v, g, beta, output_final_state, initial_state, path, l2norm=False, gate_act=False,
             output_gate=None, out_buf=None, state_buf=None):
    q, k, v, g, beta = (x.contiguous() for x in (q, k, v, g, beta))
    B, S, Hk, Hv = _check_inputs(q, k, v, g, beta)
    if not q.is_cuda:
        raise RuntimeError("gdn_chunk needs CUDA tensors (sm_100a); there is no CPU path")
    lib = _lib.load()
    dev = q.device
    for name, x in (("k", k), ("v", v), ("g", g), ("beta", beta)):
        if x.device != dev:
            raise ValueError(f"{name} is on {x.device}, q on {dev}")
    q, k, v = (x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16) for x in (q, k, v))
    if g.dtype == torch.bfloat16 and beta.dtype == torch.bfloat16:
        gate = _lib.GATE_BF16
    else:
        g, beta = g.float(), beta.float()
        gate = _lib.GATE_F32
    h0 = None
    if initial_state is not None:
        if tuple(initial_state.shape) != (B, Hv, GDN_D, GDN_D):
            raise ValueError(f"initial_state must be [B,Hv,{GDN_D},{GDN_D}], got {tuple(initial_state.shape)}")
        h0 = initial_state.to(device=dev, dtype=torch.float32).contiguous()
    # out_buf / state_buf: contiguous views the results are written into directly (used by the packed-batch driver)
    out = torch.empty((B, S, Hv, GDN_D), dtype=torch.bfloat16, device=dev) if out_buf is None else out_buf
    hT = None
    if output_final_state:
        hT = torch.empty((B, Hv, GDN_D, GDN_D), dtype=torch.float32, device=dev) if state_buf is None else state_buf
    code = _lib.PATHS[path]
    with torch.cuda.device(dev):
        nbytes = int(lib.gdn_chunk_scratch_bytes(B, S, Hk, Hv, code))
        scratch = _scratch_for(dev, nbytes)
        stream = torch.cuda.current_stream(dev).cuda_stream
        if output_gate is None:
            st = lib.gdn_chunk_fwd_sm100_ex(
                q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(),
                h0.data_ptr() if h0 is not None else None, out.data_ptr(),
                hT.data_ptr() if hT is not None else None, scratch.data_ptr(), scratch.numel(),
                B, S, Hk, Hv, gate, code, _flags(l2norm, gate_act), stream)
            _lib.check(st, "gdn_chunk_fwd_sm100_ex")
        else:
            z, weight, eps = _check_output_gate(output_gate, (B, S, Hv, GDN_D), dev)
            st = lib.gdn_chunk_fwd_gated_sm100(
                q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(),
                h0.data_ptr() if h0 is not None else None, z.data_ptr(), weight.data_ptr(), eps, out.data_ptr(),
                hT.data_ptr() if hT is not None else None, scratch.data_ptr(), scratch.numel(),
                B, S, Hk, Hv, gate, code, _flags(l2norm, gate_act), stream)
            _lib.check(st, "gdn_chunk_fwd_gated_sm100")
        if os.environ.get("GDN_CHUNK_CHECK_STATUS", "0") == "1":
            check_device_status(dev)
    return out, hT


def _forward_packed(q, k, v, g, beta, cu, output_final_state, initial_state, l2norm, gate_act):
    """One pass over a packed batch (checked by the caller): [1, T, ...] tensors, cu the list of boundaries."""
    import ctypes
    lib = _lib.load()
    dev = q.device
    for name, x in (("k", k), ("v", v), ("g", g), ("beta", beta)):
        if x.device != dev:
            raise ValueError(f"{name} is on {x.device}, q on {dev}")
    q, k, v = (x.to(torch.bfloat16).contiguous() for x in (q, k, v))
    if g.dtype == torch.bfloat16 and beta.dtype == torch.bfloat16:
        g, beta = g.contiguous(), beta.contiguous()
        gate = _lib.GATE_BF16
    else:
        g, beta = g.float().contiguous(), beta.float().contiguous()
        gate = _lib.GATE_F32
    Hk, Hv, T, n_seq = q.size(2), v.size(2), q.size(1), len(cu) - 1
    h0 = None if initial_state is None else initial_state.to(device=dev, dtype=torch.float32).contiguous()
    out = torch.empty((1, T, Hv, GDN_D), dtype=torch.bfloat16, device=dev)
    hT = torch.empty((n_seq, Hv, GDN_D, GDN_D), dtype=torch.float32, device=dev) if output_final_state else None
    bounds = (ctypes.c_int * (n_seq + 1))(*cu)
    with torch.cuda.device(dev):
        scratch = _scratch_for(dev, int(lib.gdn_chunk_varlen_scratch_bytes(bounds, n_seq, Hv)))
        st = lib.gdn_chunk_fwd_varlen_sm100(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(), None if h0 is None else h0.data_ptr(),
            out.data_ptr(), None if hT is None else hT.data_ptr(), scratch.data_ptr(), scratch.numel(), bounds, n_seq,
            Hk, Hv, gate, _flags(l2norm, gate_act), torch.cuda.current_stream(dev).cuda_stream)
        _lib.check(st, "gdn_chunk_fwd_varlen_sm100")
        if os.environ.get("GDN_CHUNK_CHECK_STATUS", "0") == "1":
            check_device_status(dev)
    return out, hT


def check_device_status(device=None):
    """Synchronise every stream of `device` this module has launched on and raise if a kernel on any of them
    reported a bounded wait that ran out (its result is then undefined).  Callers that launch asynchronously and
    never come here should call this before they trust a result; the module's own synchronising calls do."""
    import ctypes
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    if device.index is None:
        device = torch.device("cuda", torch.cuda.current_device())
    lib = _lib.load()
    for (index, stream), buf in list(_scratch.items()):
        if index != device.index:
            continue
        word = ctypes.c_int(0)
        with torch.cuda.device(device):
            st = lib.gdn_chunk_read_status(buf.data_ptr(), stream, ctypes.byref(word))
        if st != _lib.GDN_OK:
            raise _lib.GdnLibraryError(f"device status 0x{word.value:x}: {_lib.error_string(st)}")


def gdn_chunk(q, k, v, g, beta, output_final_state=True, initial_state=None, path="auto",
              use_qk_l2norm_in_kernel=False, gate_activations=False, output_gate=None):
    """GDN forward (chunked gated delta rule).

    Args:
        q, k: [B, S, Hk, D] bf16 - QK heads.
        v:    [B, S, Hv, D] bf16 - V heads (Hv must be a multiple of Hk).
        g, beta: [B, S, Hv] bf16 or fp32 - log-decay (<= 0) and update gate.
        output_final_state: whether to return the final state.
        initial_state: optional [B, Hv, D, D] state to start from (zeros when None).
        path: "auto", or a key of `_lib.PATHS` to force a kernel.
        use_qk_l2norm_in_kernel: L2-normalise every q and k head vector inside the kernels, the switch of the
            reference's torch definition (reference/gdn_chunk_ref.py:29, :43-45).
        gate_activations: g and beta are raw projections; the kernels apply g = -softplus(g), beta = sigmoid(beta).
        output_gate: (z, weight) or (z, weight, eps): `out` becomes rmsnorm_gated(out, z, weight), the layer's next
            step (reference: output_gate_interface.py:15-27), applied in place right behind the forward pass.

    Returns:
        out [B, S, Hv, D] bf16, and final_state [B, Hv, D, D] fp32 (None when not requested).
    """
    done = (_native_forward or _native())(q, k, v, g, beta, output_final_state, initial_state, _lib.PATHS[path],
                                          _flags(use_qk_l2norm_in_kernel, gate_activations), output_gate)
    if done is not None:
        return done
    return _forward(q, k, v, g, beta, output_final_state, initial_state, path, bool(use_qk_l2norm_in_kernel),
                    bool(gate_activations), output_gate)


_arena = {}    # (device index, stream slot) -> uint8 device tensor for gdn_chunk_host


def gdn_chunk_host(q, k, v, g, beta, output_final_state=True, initial_state=None, out=None, final_state_out=None,
                   device=None, seg_tokens=0, use_qk_l2norm_in_kernel=False, gate_activations=False, synchronize=True,
                   arena_slot=0):
    """gdn_chunk for inputs and results in HOST memory, with the copies pipelined against the kernels.

    q, k, v (bf16), g, beta (bf16 or fp32) and initial_state (fp32) are CPU tensors, contiguous; page-locked
    tensors (`pin_memory()`) are needed for the overlap.  The sequence is cut into segments; while segment i runs
    on the GPU the inputs of segment i+1 travel in and the outputs of segment i-1 travel out (C ABI:
    gdn_chunk_fwd_host_sm100).  Results land in `out` [B,S,Hv,D] bf16 and `final_state_out` [B,Hv,D,D] fp32
    (pinned CPU tensors, allocated when not given).  With synchronize=False the call returns while copies are
    still in flight on the current stream: synchronise that stream before reading the results.  Calls that may
    be in flight at the same time (different streams) must use different `arena_slot` values.
    """
    B, S, Hk, Hv = _check_inputs(q, k, v, g, beta)
    for name, x in (("q", q), ("k", k), ("v", v), ("g", g), ("beta", beta)):
        if x.is_cuda:
            raise ValueError(f"{name} is a CUDA tensor: use gdn_chunk for device tensors")
    lib = _lib.load()
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    q, k, v = (x.contiguous() if x.dtype == torch.bfloat16 else x.to(torch.bfloat16).contiguous() for x in (q, k, v))
    if g.dtype == torch.bfloat16 and beta.dtype == torch.bfloat16:
        gate = _lib.GATE_BF16
        g, beta = g.contiguous(), beta.contiguous()
    else:
        g, beta = g.float().contiguous(), beta.float().contiguous()
        gate = _lib.GATE_F32
    h0 = None
    if initial_state is not None:
        if tuple(initial_state.shape) != (B, Hv, GDN_D, GDN_D):
            raise ValueError(f"initial_state must be [B,Hv,{GDN_D},{GDN_D}], got {tuple(initial_state.shape)}")
        h0 = initial_state.to(torch.float32).contiguous()
    if out is None:
        out = torch.empty((B, S, Hv, GDN_D), dtype=torch.bfloat16).pin_memory()
    elif tuple(out.shape) != (B, S, Hv, GDN_D) or out.dtype != torch.bfloat16 or out.is_cuda or not out.is_contiguous():
        raise ValueError("out must be a contiguous CPU bf16 tensor [B,S,Hv,D]")
    hT = None
    if output_final_state:
        hT = final_state_out
        if hT is None:
            hT = torch.empty((B, Hv, GDN_D, GDN_D), dtype=torch.float32).pin_memory()
        elif tuple(hT.shape) != (B, Hv, GDN_D, GDN_D) or hT.dtype != torch.float32 or hT.is_cuda or not hT.is_contiguous():
            raise ValueError("final_state_out must be a contiguous CPU fp32 tensor [B,Hv,D,D]")
    with torch.cuda.device(dev):
        nbytes = int(lib.gdn_chunk_host_arena_bytes(B, S, Hk, Hv, gate, int(seg_tokens)))
        key = (dev.index, int(arena_slot))
        arena = _arena.get(key)
        if arena is None or arena.numel() < nbytes:
            arena = torch.empty(max(nbytes, 256), dtype=torch.uint8, device=dev)
            _arena[key] = arena
        stream = torch.cuda.current_stream(dev)
        st = lib.gdn_chunk_fwd_host_sm100(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(),
            h0.data_ptr() if h0 is not None else None, out.data_ptr(), hT.data_ptr() if hT is not None else None,
            arena.data_ptr(), arena.numel(), B, S, Hk, Hv, gate, int(seg_tokens),
            _flags(use_qk_l2norm_in_kernel, gate_activations), stream.cuda_stream)
        _lib.check(st, "gdn_chunk_fwd_host_sm100")
        if synchronize:
            stream.synchronize()
            if os.environ.get("GDN_CHUNK_CHECK_STATUS", "0") == "1":
                import ctypes
                word = ctypes.c_int(0)
                if lib.gdn_chunk_read_status(arena.data_ptr(), stream.cuda_stream, ctypes.byref(word)) != _lib.GDN_OK:
                    raise _lib.GdnLibraryError(f"device status 0x{word.value:x}")
    return out, hT


_varlen_streams = {}


def gdn_chunk_varlen(q, k, v, g, beta, cu_seqlens, output_final_state=True, initial_state=None, n_streams=4,
                     strategy="auto", **options):
    """gdn_chunk over a packed batch of sequences of different lengths.

    q, k: [1, T, Hk, D] (or [T, Hk, D]); v: [1, T, Hv, D]; g, beta: [1, T, Hv]; cu_seqlens: the n_seq + 1 cumulative
    sequence boundaries 0 = c_0 < c_1 < ... < c_n = T as a list or CPU tensor (a CUDA tensor is read back, which
    synchronises).  Sequence i is tokens [c_i, c_{i+1}).
    strategy:
      "packed"  all sequences in one pass of the kernels, which find each chunk's sequence through small tables (no
                padding, no copies; C ABI: gdn_chunk_fwd_varlen_sm100); sequences of at most 8 tokens share a launch of the
                decode kernel.  What "auto" does.
      "views"   every sequence as an ordinary forward pass on its slice, neighbours of equal length as one regular batch, the
                launches spread round-robin over `n_streams` streams that are ordered after, and joined back into, the
                current one.
      "padded"  all sequences gathered into one regular batch [n_seq, L_max, ...] whose padding tokens carry g = 0 and
                beta = 0 (they leave the state untouched and their outputs are dropped, so the result is exact), one forward
                pass, the outputs scattered back: two extra passes over the data.
    With a forced path, or contiguous tensors at an address that is no multiple of 16 bytes, "auto" is "padded" when there
    are more than 8 launches to make and padding at most doubles the token count, else "views".  The reference has no
    variable-length entry; its recurrent torch definition (reference/gdn_chunk_ref.py:103-147) applied per sequence
    defines the result.  initial_state / returned final state: [n_seq, Hv, D, D]; `options` are gdn_chunk's keywords
    (path, use_qk_l2norm_in_kernel, gate_activations).
    Returns (out [1, T, Hv, D] bf16 (or [T, Hv, D] when the inputs had no batch axis), final_state or None).
    """
    squeeze = q.dim() == 3
    if squeeze:
        q, k, v, g, beta = (x.unsqueeze(0) for x in (q, k, v, g, beta))
    _, T, Hk, Hv = _check_inputs(q, k, v, g, beta)
    if q.size(0) != 1:
        raise ValueError("packed tensors must have batch size 1")
    cu = cu_seqlens.tolist() if torch.is_tensor(cu_seqlens) else list(cu_seqlens)
    if len(cu) < 2 or cu[0] != 0 or cu[-1] != T or any(b <= a for a, b in zip(cu, cu[1:])):
        raise ValueError(f"cu_seqlens must rise strictly from 0 to T={T}, got {cu}")
    n_seq = len(cu) - 1
    if initial_state is not None and tuple(initial_state.shape) != (n_seq, Hv, GDN_D, GDN_D):
        raise ValueError(f"initial_state must be [n_seq,Hv,{GDN_D},{GDN_D}], got {tuple(initial_state.shape)}")
    if not q.is_cuda:
        raise RuntimeError("gdn_chunk_varlen needs CUDA tensors (sm_100a); there is no CPU path")
    dev = q.device
    if strategy not in ("auto", "views", "packed", "padded"):
        raise ValueError(f"unknown strategy {strategy!r}")
    # (the kernels want 16-byte aligned tensors; strided or converted ones are copied, a view at an odd offset is not and
    # takes the routes below, which gather it or refuse it)
    aligned = all(x is None or x.data_ptr() % 16 == 0 for x in (q, k, v, initial_state))
    if strategy == "packed" or (strategy == "auto" and aligned and options.get("path", "auto") == "auto"):
        out, states = _forward_packed(q, k, v, g, beta, cu, output_final_state, initial_state,
                                      bool(options.get("use_qk_l2norm_in_kernel", False)),
                                      bool(options.get("gate_activations", False)))
        return (out[0] if squeeze else out), states
    q, k, v, g, beta = (x.contiguous() for x in (q, k, v, g, beta))
    out = torch.empty((1, T, Hv, GDN_D), dtype=torch.bfloat16, device=dev)
    states = torch.empty((n_seq, Hv, GDN_D, GDN_D), dtype=torch.float32, device=dev) if output_final_state else None
    main = torch.cuda.current_stream(dev)
    n_streams = max(1, min(int(n_streams), n_seq))
    streams = _varlen_streams.setdefault(dev.index, [])
    while len(streams) < n_streams:
        streams.append(torch.cuda.Stream(dev))
    runs = []                       # (first sequence, number of sequences, length): neighbours of equal length
    for i in range(n_seq):
        n = cu[i + 1] - cu[i]
        if runs and runs[-1][2] == n:
            runs[-1][1] += 1
        else:
            runs.append([i, 1, n])
    l_max = max(r[2] for r in runs)
    if strategy == "padded" or (strategy == "auto" and len(runs) > 8 and n_seq * l_max <= 2 * T):
        import numpy as np
        lens = np.diff(np.asarray(cu, dtype=np.int64))
        pos = np.arange(l_max, dtype=np.int64)[None, :]
        valid_np = pos < lens[:, None]                                                  # [n_seq, l_max]
        idx_np = np.minimum(np.asarray(cu[:-1], dtype=np.int64)[:, None] + pos, T - 1)  # token of (sequence, position)
        idx = torch.from_numpy(idx_np).to(dev)
        valid = torch.from_numpy(valid_np).to(dev)
        take = lambda x: x[0][idx]                                                      # [n_seq, l_max, ...]
        gates = [take(x) * valid.unsqueeze(-1).to(x.dtype) for x in (g, beta)]
        if options.get("gate_activations", False):    # raw gates: the values the activations map to g = 0, beta = 0
            gates = [torch.where(valid.unsqueeze(-1), take(x), torch.full((), float("-inf"), dtype=x.dtype, device=dev))
                     for x in (g, beta)]
        ob, sb = _forward(take(q), take(k), take(v), gates[0], gates[1], output_final_state, initial_state,
                          options.get("path", "auto"), bool(options.get("use_qk_l2norm_in_kernel", False)),
                          bool(options.get("gate_activations", False)))
        out[0][idx[valid]] = ob[valid]
        return (out[0] if squeeze else out), sb
    ready = main.record_event()
    n_streams = min(n_streams, len(runs))
    for j, (i, cnt, n) in enumerate(runs):
        a, b = cu[i], cu[i + cnt]
        s = streams[j % n_streams]
        if j < n_streams:
            s.wait_event(ready)
        as_batch = lambda x: x[0, a:b].reshape(cnt, n, *x.shape[2:])      # [1, cnt*n, ...] -> [cnt, n, ...], a view
        with torch.cuda.stream(s):
            h0 = None if initial_state is None else initial_state[i:i + cnt]
            _forward(as_batch(q), as_batch(k), as_batch(v), as_batch(g), as_batch(beta), output_final_state, h0,
                     options.get("path", "auto"), bool(options.get("use_qk_l2norm_in_kernel", False)),
                     bool(options.get("gate_activations", False)), None, as_batch(out),
                     None if states is None else states[i:i + cnt])
    for s in streams[:n_streams]:
        main.wait_stream(s)
    for x in (q, k, v, g, beta, out):      # the side streams read and wrote these: keep the allocator informed
        for s in streams[:n_streams]:
            x.record_stream(s)
    return (out[0] if squeeze else out), states


def scan_transfers(A, Bm, h0=None):
    """Second scan level on the GPU: groups g of each sequence map S_in -> A[:, g] @ S_in + Bm[:, g].

    A, Bm: fp32 [n_seq, G, 128, 128]; h0: fp32 [n_seq, 128, 128] or None.  Returns (s_in, s_final): the state
    every group starts from, fp32 [n_seq, G, 128, 128], and the state after the last group [n_seq, 128, 128].
    """
    n_seq, G = A.shape[:2]
    A, Bm = A.contiguous(), Bm.contiguous()
    s_in = torch.empty_like(A)
    s_final = torch.empty((n_seq, GDN_D, GDN_D), dtype=torch.float32, device=A.device)
    h = None if h0 is None else h0.to(torch.float32).contiguous()
    with torch.cuda.device(A.device):
        st = _lib.load().gdn_chunk_scan_transfers(
            A.data_ptr(), Bm.data_ptr(), h.data_ptr() if h is not None else None, s_in.data_ptr(),
            s_final.data_ptr(), n_seq, G, torch.cuda.current_stream(A.device).cuda_stream)
    _lib.check(st, "gdn_chunk_scan_transfers")
    return s_in, s_final


def gdn_chunk_twolevel(q, k, v, g, beta, group_chunks=64, eps=1e-6, frac=1.0, gt_eps=1e-2, initial_state=None,
                       decay_early_out=True):
    """Explicit two-level chunk scan (same name and leading arguments as the reference's
    gdn_chunk_interface.py:53-62).

    The sequence is cut into groups of `group_chunks` 64-token chunks.  Pass 1 runs every group as an independent
    sequence twice - from a zero state (giving B_g) and, with zero values, from an identity state (giving A_g) - so
    that S_out = A_g S_in + B_g; the scan kernel chains these maps in fp32; pass 2 runs every group from its true
    incoming state and writes the output.  Always exact: eps / frac / gt_eps, which steer the reference's
    approximate reset path, are accepted and ignored.  Returns (out, final_state, info); info holds the number of
    groups
    and the number of passes made.  S must be a multiple of 64 * group_chunks (otherwise the serial path is used).

    decay_early_out: when the decay makes every group forget its incoming state within its first p tokens (the bound
    ||A|| <= exp(sum of g), see distributed.forgetting_horizon; one host read), pass 1 already gives the right
    outputs from token p of each group on and the right outgoing states; the A_g are not computed and pass 2 reruns
    only the first p tokens of every group from the previous group's B_g: 1 + p / (64 * group_chunks) passes
    instead of three, same result.  This is the exact counterpart of the reference's approximate reset path
    (csrc/gdn_chunk/gdn_ops.cu:774-963).
    """
    q, k, v, g, beta = (x.contiguous() for x in (q, k, v, g, beta))
    B, S, Hk, Hv = _check_inputs(q, k, v, g, beta)
    seg = GDN_CHUNK * int(group_chunks)
    G = S // seg if seg > 0 else 0
    if G < 2 or S % seg != 0:
        out, hT = _forward(q, k, v, g, beta, True, initial_state, "auto")
        return out, hT, torch.ones(1, dtype=torch.float32, device=out.device)
    dev = q.device

    def fold(x):      # [B, G*seg, ...] -> [B*G, seg, ...]: every group becomes a batch element
        return x.reshape(B * G, seg, *x.shape[2:])

    qg, kg, vg, gg, bg = (fold(x) for x in (q, k, v, g, beta))
    out1, Bm = _forward(qg, kg, vg, gg, bg, True, None, "auto")                    # [B*G, Hv, 128, 128]
    from .distributed import forgetting_horizon
    p = forgetting_horizon(kg, gg, bg) if decay_early_out else None
    if p is not None:
        # every group has forgotten its incoming state after p tokens: pass 1 is right from there on, and group j
        # really starts from B_{j-1} (the first from the initial state)
        Bg = Bm.reshape(B, G, Hv, GDN_D, GDN_D)
        first = (torch.zeros_like(Bg[:, :1]) if initial_state is None
                 else initial_state.to(device=dev, dtype=torch.float32).reshape(B, 1, Hv, GDN_D, GDN_D))
        s_in = torch.cat([first, Bg[:, :-1]], dim=1).reshape(B * G, Hv, GDN_D, GDN_D)
        head, _ = _forward(qg[:, :p], kg[:, :p], vg[:, :p], gg[:, :p], bg[:, :p], False, s_in, "auto")
        out1[:, :p] = head
        info = torch.tensor([float(G), 1.0 + p / seg], dtype=torch.float32, device=dev)
        return out1.reshape(B, S, Hv, GDN_D), Bg[:, -1].contiguous(), info
    else:
        eye = torch.eye(GDN_D, dtype=torch.float32, device=dev).expand(B * G, Hv, GDN_D, GDN_D).contiguous()
        _, A = _forward(qg, kg, torch.zeros_like(vg), gg, bg, True, eye, "auto")
        # [B*G, Hv, ...] -> [B*Hv, G, ...]
        to_seq = lambda x: x.reshape(B, G, Hv, GDN_D, GDN_D).permute(0, 2, 1, 3, 4).reshape(B * Hv, G, GDN_D, GDN_D)
        h0 = None if initial_state is None else initial_state.to(device=dev, dtype=torch.float32).reshape(B * Hv, GDN_D, GDN_D)
        s_in, s_final = scan_transfers(to_seq(A), to_seq(Bm), h0)
        s_in = s_in.reshape(B, Hv, G, GDN_D, GDN_D).permute(0, 2, 1, 3, 4).reshape(B * G, Hv, GDN_D, GDN_D)
        passes = 3.0
    out, _ = _forward(qg, kg, vg, gg, bg, False, s_in, "auto")
    info = torch.tensor([float(G), passes], dtype=torch.float32, device=dev)
    return out.reshape(B, S, Hv, GDN_D), s_final.reshape(B, Hv, GDN_D, GDN_D), info


def gdn_chunk_reference(q, k, v, g, beta, chunk_size=64, mode="chunk"):
    """Pure-torch definition of the operator, for callers that want the correctness anchor the
    reference exposes under this name (gdn_chunk_interface.py:65-72).  Runs on the inputs'
    device in fp32; q/k must already be expanded to Hv heads, as in the reference."""
    from .torch_definition import chunk_gated_delta_rule, recurrent_gated_delta_rule
    if mode == "chunk":
        return chunk_gated_delta_rule(q, k, v, g, beta, chunk_size=chunk_size, output_final_state=True)
    return recurrent_gated_delta_rule(q, k, v, g, beta, output_final_state=True)
