"""``chunk_kda``: the KDA chunkwise gated delta rule, forward and backward, on B200.

Drop-in for the call the reference makes at k3mini/model.py:197-216
(``fla.ops.kda.chunk_kda``): same arguments, same gate / beta / initial-state /
final-state / ``cu_seqlens`` meaning, same return value ``(o, final_state_or_None)``.
The arithmetic runs in ``libkda_b200.so`` (hand-written CUDA for sm_100a) through the C ABI
of include/kda_b200.h; PyTorch only owns the memory and the stream.
"""

from __future__ import annotations

import threading
from functools import lru_cache

import torch

from . import _lib

_DTYPES = {torch.float32: _lib.DTYPE_F32, torch.bfloat16: _lib.DTYPE_BF16}


@lru_cache(maxsize=64)
def _chunk_tables_cached(cu: tuple, device_index: int):
    lens = [cu[i + 1] - cu[i] for i in range(len(cu) - 1)]
    if any(l < 0 for l in lens):
        raise ValueError("cu_seqlens must be non-decreasing")
    counts = [(l + _lib.CHUNK - 1) // _lib.CHUNK for l in lens]
    off = [0]
    for c in counts:
        off.append(off[-1] + c)
    seq = [n for n, c in enumerate(counts) for _ in range(c)]
    # per chunk: sequence, chunk inside the sequence, first flattened token, valid rows
    tab = [(n, j, cu[n] + j * _lib.CHUNK, min(_lib.CHUNK, lens[n] - j * _lib.CHUNK))
           for n, c in enumerate(counts) for j in range(c)]
    dev = torch.device("cuda", device_index)
    return (torch.tensor(seq if seq else [0], dtype=torch.int32, device=dev),
            torch.tensor(off, dtype=torch.int32, device=dev), off[-1],
            torch.tensor(tab if tab else [(0, 0, 0, 0)], dtype=torch.int32, device=dev), max(counts, default=0))


def _chunk_tables(cu_seqlens, cu_seqlens_cpu, device, tokens):
    """Per-chunk sequence index and per-sequence first chunk.  Chunks never straddle a
    document boundary, so the table depends on the lengths; it is built on the host
    (``cu_seqlens_cpu`` avoids the device-to-host copy) and cached per length tuple."""
    host = cu_seqlens_cpu if cu_seqlens_cpu is not None else cu_seqlens.cpu()
    cu = tuple(int(x) for x in host.tolist())
    if cu and (cu[0] < 0 or cu[-1] > tokens):
        raise ValueError(f"cu_seqlens must stay within the {tokens} tokens of the batch, got {cu[0]} to {cu[-1]}")
    return _chunk_tables_cached(cu, device.index or 0)


def _packed_tables(cu_seqlens, cu_seqlens_cpu, x):
    """(cu_seqlens, chunk_seq, seq_chunk_off, chunk_tab, number of chunks, chunks of the longest document) as the native
    calls take them, for documents packed into the [B, T, ...] tensor x."""
    if cu_seqlens is None:
        return None, None, None, None, 0, 0
    seq, off, nt, tab, longest = _chunk_tables(cu_seqlens, cu_seqlens_cpu, x.device, x.shape[:2].numel())
    return cu_seqlens.to(device=x.device, dtype=torch.int64).contiguous(), seq, off, tab, nt, longest


class _DeviceStatus:
    """One int32 status word per device, mirrored in pinned host memory.  A kernel whose bounded wait
    gives up ORs a code into the device word (``KdaParams.status``) and stores the word into the pinned
    mirror (``KdaParams.status_host``, device-mapped) itself, so the next
    call on that device (or ``check_device_status``) notices it by reading host memory: no copy engine,
    no synchronisation on the hot path."""

    _per_device: dict = {}
    _lock = threading.Lock()  # a word that kernels and the native path know is never replaced

    def __init__(self, device):
        self.dev = torch.zeros(1, dtype=torch.int32, device=device)
        self.host = torch.zeros(1, dtype=torch.int32).pin_memory()  # device-mapped under unified addressing
        _lib.host().set_status(device.index, self.dev.data_ptr(), self.host.data_ptr())

    @classmethod
    def get(cls, device):
        key = device.index if device.index is not None else torch.cuda.current_device()
        st = cls._per_device.get(key)
        if st is None:
            with cls._lock:
                st = cls._per_device.get(key)
                if st is None:
                    st = cls._per_device[key] = cls(torch.device("cuda", key))
        return st

    @classmethod
    def of_index(cls, index):
        cls.get(torch.device("cuda", index))

    @classmethod
    def report(cls, index):
        cls.get(torch.device("cuda", index)).poll()

    def poll(self, sync=False):
        if sync:
            self.host.copy_(self.dev)
        code = int(self.host[0])
        if code:
            self.dev.zero_()
            self.host.zero_()
            msg = _lib.load().kda_status_string(_lib.ERR_DEVICE_WAIT).decode()
            raise RuntimeError(f"chunk_kda: {msg} (stage bits 0x{code:x}); the results of the affected call are invalid")


def check_device_status(device=None, sync=True):
    """Raise if a KDA kernel on ``device`` reported a bounded wait that gave up.  ``sync=True``
    reads the status word now (blocking); ``sync=False`` only looks at copies already finished."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    _DeviceStatus.get(dev).poll(sync=sync)


_warned = set()


def _warn_once(msg):
    if msg not in _warned:
        _warned.add(msg)
        import warnings
        warnings.warn(msg, RuntimeWarning, stacklevel=3)


def _require_cuda(t):
    if not t.is_cuda:
        raise RuntimeError("chunk_kda runs only on a CUDA device (sm_100a); there is no CPU fallback")


@torch.compiler.disable
def chunk_kda(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=False,
              use_qk_l2norm_in_kernel=False, use_gate_in_kernel=False, use_beta_sigmoid_in_kernel=False,
              cu_seqlens=None, cu_seqlens_cpu=None, safe_gate=False, lower_bound=None, disable_recompute=False,
              state_v_first=False, A_log=None, dt_bias=None, chunk_size=64, fp32_math=False,
              short_conv_weights=None, **kwargs):
    """Kimi Delta Attention, chunkwise (k3mini/model.py:200-216).

    q, k, g: [B, T, H, K]; v: [B, T, H, V]; beta: [B, T, H].  With
    ``use_gate_in_kernel`` g is the raw gate input and the op applies
    ``-exp(A_log) * softplus(g + dt_bias)`` (k3mini/model.py:220-222), otherwise g is the
    natural-log decay per token.  ``use_qk_l2norm_in_kernel`` normalises q and k as
    k3mini/model.py:218-219 does; ``use_beta_sigmoid_in_kernel`` treats beta as logits.
    ``initial_state`` / the returned final state are FP32 ``[N, H, K, V]`` (``[N, H, V, K]``
    with ``state_v_first``).  ``cu_seqlens`` ([N+1], batch 1) packs N documents; chunks and
    the state restart at every document.  ``disable_recompute=True`` keeps the per-chunk
    records between forward and backward, ``False`` rebuilds them in the backward.
    ``fp32_math=True`` forces FP32 CUDA-core arithmetic in every stage (validation mode;
    FP32 inputs always run that way).  Returns ``(o, final_state or None)``.

    ``short_conv_weights=(wq, wk, wv)`` (each ``[H*K, 1, ksize]``, ksize <= 4; an extension, the
    reference has no such argument) says that q, k, v are the projections BEFORE the three
    causal depthwise convolutions + SiLU of k3mini/model.py:181-185.  For BF16 with K = 128 the
    forward kernel applies the filter while it loads the chunk (three halo rows included, the
    window restarting at every sequence start) and the backward kernels run the convolution
    backward on the gradient rows while they are still on chip; otherwise the stand-alone
    convolution kernels run first.  Both routes give the same bits as ``ShortConvolution`` followed
    by ``chunk_kda`` (the filter gradients agree to FP32 summation accuracy).
    """
    state_v_first = bool(kwargs.pop("transpose_state_layout", state_v_first))
    for name in ("return_intermediate_states", "cp_context"):
        if kwargs.pop(name, None):
            raise NotImplementedError(f"chunk_kda: {name} is not supported by the B200 kernels")
    if kwargs:
        raise TypeError(f"chunk_kda: unexpected arguments {sorted(kwargs)}")
    for t in (q, k, v, g, beta):
        _require_cuda(t)
    if safe_gate or lower_bound is not None:
        raise NotImplementedError("chunk_kda: safe_gate/lower_bound are not part of the reference path "
                                  "(k3mini/model.py:212 always passes safe_gate=False)")
    if chunk_size != 64:
        raise ValueError(f"`chunk_size` must be 64 for the B200 KDA kernels, got {chunk_size}.")
    host = _lib.host()
    # environment switches for debugging and A-B measurement: OPENKIMI_B200_FP32_MATH=1 (as fp32_math),
    # OPENKIMI_B200_ROW_COPIES=1 (row copies instead of bulk-tensor tile copies), and OPENKIMI_B200_FP32_STAGES, whose bit
    # s runs stage s (0 fwd_intra, 1 fwd_state, 2 bwd_state, 3 bwd_chunk as one fused kernel, 4 bwd_wy) with FP32
    # CUDA-core arithmetic instead of tensor cores
    flags = host.env_flags()
    if flags & (31 << 5):
        _warn_once(f"OPENKIMI_B200_FP32_STAGES={flags >> 5 & 31}: the selected KDA stages run the FP32 CUDA-core "
                   "validation kernels instead of the tensor-core kernels (debugging switch, much slower)")
    if fp32_math:
        flags |= _lib.FLAG_FORCE_SIMT
    flags |= ((_lib.FLAG_QK_L2NORM if use_qk_l2norm_in_kernel else 0) | (_lib.FLAG_GATE if use_gate_in_kernel else 0)
              | (_lib.FLAG_BETA_SIGMOID if use_beta_sigmoid_in_kernel else 0)
              | (_lib.FLAG_STATE_V_FIRST if state_v_first else 0))
    wq = wk = wv = None
    if short_conv_weights is not None:
        wq, wk, wv = short_conv_weights
        if q.dim() != 4:
            raise ValueError(f"q and k must have the same shape [B,T,H,K], got q={tuple(q.shape)} vs k={tuple(k.shape)}")
        B, T, H, K = q.shape
        for w in (wq, wk, wv):
            if w.dim() != 3 or w.shape[0] != H * K or w.shape[1] != 1 or not 1 <= w.shape[2] <= 4 or w.shape != wq.shape:
                raise ValueError(f"short_conv_weights must be three [H*K, 1, ksize<=4] filters, got {tuple(w.shape)}")
        if not (q.dtype == torch.bfloat16 and K == 128 and not flags & ~15):
            # FP32 validation mode and d = 64: same arithmetic, separate kernels
            from .modules import short_convolution
            cu = None if cu_seqlens is None else cu_seqlens.to(device=q.device, dtype=torch.int64).contiguous()
            q, k, v = (short_convolution(x.reshape(B, T, H * K), w, cu).view(B, T, H, K)
                       for x, w in zip((q, k, v), (wq, wk, wv)))
            wq = wk = wv = None
    return host.chunk_kda(q, k, v, g, beta, A_log, dt_bias, initial_state, wq, wk, wv, scale, flags, output_final_state,
                          disable_recompute, *_packed_tables(cu_seqlens, cu_seqlens_cpu, q))


def recurrent_kda_step(q, k, v, g, beta, state, *, scale=None, A_log=None, dt_bias=None,
                       use_qk_l2norm_in_kernel=False, use_gate_in_kernel=False, use_beta_sigmoid_in_kernel=False,
                       state_v_first=False, inplace=False):
    """One decoding step of KDA: the recurrence of k3mini/model.py:121-128 for a single token.

    q, k, g: [N, H, K]; v: [N, H, V]; beta: [N, H]; ``state``: FP32 ``[N, H, K, V]`` (``[N, H, V, K]``
    with ``state_v_first``), e.g. the final state ``chunk_kda`` returned for the prompt.  The prologue
    switches mean what they mean in ``chunk_kda``.  Returns ``(o [N, H, V], new_state)``; with
    ``inplace=True`` the state tensor itself is updated and returned.  Inference only (no autograd).
    """
    return _lib.host().recurrent(q, k, v, g, beta, state, A_log, dt_bias, scale, use_qk_l2norm_in_kernel, use_gate_in_kernel,
                                 use_beta_sigmoid_in_kernel, state_v_first, inplace, False, True)


def fused_recurrent_kda(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=False, *, A_log=None,
                        dt_bias=None, use_qk_l2norm_in_kernel=False, use_gate_in_kernel=False,
                        use_beta_sigmoid_in_kernel=False, state_v_first=False):
    """Token-by-token KDA over ``[B, T, H, K]`` inputs (the decoding counterpart of ``chunk_kda``, same prologue
    keywords; meant for the few tokens of a decode loop): the recurrence of ``recurrent_kda_step`` in one launch,
    the state on chip from the first token to the last.  Returns ``(o [B, T, H, V], final_state or None)``."""
    return _lib.host().recurrent(q, k, v, g, beta, initial_state, A_log, dt_bias, scale, use_qk_l2norm_in_kernel,
                                 use_gate_in_kernel, use_beta_sigmoid_in_kernel, state_v_first, False, True, output_final_state)
