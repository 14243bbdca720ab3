"""Tensor-level wrapper over the C ABI (torch provides device memory only).  The checks of a call, its
allocations and its parameter block are native (csrc/torch_native.cpp)."""
from __future__ import annotations

import ctypes
import math

import torch

from . import build, capi

_native = build.load_native()

_DTYPES = {torch.float16: capi.DTYPE_FP16, torch.bfloat16: capi.DTYPE_BF16}


class Fa3Error(RuntimeError):
    def __init__(self, entry: str, code: int):
        super().__init__(f"{entry} returned {code} ({capi.status_string(code)})")
        self.code = code


_native.set_error_type(Fa3Error)  # (what the torch ops raise)


class Fa3DeviceError(RuntimeError):
    """A kernel gave up a bounded wait (1) or found its shared memory misaligned (2): its outputs are
    not valid."""


def _raise_on_device_error(lib, entry: str):
    """After a synchronous call: read and clear the device-side error flag (the C entry points return
    SUCCESS once the work is enqueued; a kernel that ran into trouble can only say so through the flag)."""
    flag = lib.shaobo_fa3_b200_device_error(1)
    if flag != 0:
        raise Fa3DeviceError(f"{entry}: device error flag {flag}")


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _seqused_ptr(t):
    if t is None:
        return None
    if t.dtype != torch.int32 or not t.is_cuda:
        raise TypeError("seqused must be an int32 CUDA tensor")
    return t.data_ptr()


def make_params(q: torch.Tensor, k: torch.Tensor, causal: bool, softmax_scale=None, layout: str = "bhsd",
                seqused_q=None, seqused_k=None, **extra) -> capi.Params:
    """layout "bhsd": q [B,Hq,Sq,D], k [B,Hkv,Sk,D]; "bshd": q [B,Sq,Hq,D], k [B,Sk,Hkv,D].
    seqused_q / seqused_k: optional int32 [B] device tensors, the used length of every batch entry."""
    if layout == "bhsd":
        (b, hq, s, d), hkv, sk = q.shape, k.shape[1], k.shape[2]
    elif layout == "bshd":
        (b, s, hq, d), hkv, sk = q.shape, k.shape[2], k.shape[1]
    else:
        raise ValueError(f"unknown layout {layout!r}")
    p = capi.new_params(batch=b, seqlen_q=s, seqlen_k=sk, num_heads_q=hq, num_heads_kv=hkv,
                        head_dim_qk=d, head_dim_v=d, causal=int(causal), dtype=_DTYPES[q.dtype],
                        layout=capi.LAYOUT_BSHD if layout == "bshd" else capi.LAYOUT_BHSD)
    if softmax_scale is not None:
        p.softmax_scale = float(softmax_scale)
        p.softmax_scale_is_set = 1
    p.seqused_q, p.seqused_k = _seqused_ptr(seqused_q), _seqused_ptr(seqused_k)
    for key, val in extra.items():
        setattr(p, key, val)
    return p


def _result(r):
    """What a native call returned: its tensors, or (entry, status) when the C ABI refused the call."""
    if type(r[0]) is str:
        raise Fa3Error(*r)
    return r


def fa3_bwd(dout, q, k, v, out, softmax_lse, causal: bool, softmax_scale=None, deterministic=False,
            workspace=None, return_delta=False, sync=False, layout: str = "bhsd", window=(-1, -1),
            seqused_q=None, seqused_k=None, outputs=None, softcap: float = 0.0):
    """dq, dk, dv (and delta) = backward of softmax(q k^T * scale) v.

    layout "bhsd": q, out, dout [B,Hq,Sq,D]; k, v [B,Hkv,Sk,D].  layout "bshd": [B,Sq,Hq,D] and
    [B,Sk,Hkv,D].  fp16 or bf16; softmax_lse: fp32 [B,Hq,Sq] natural log in both layouts.  With
    causal=True and Sq != Sk the diagonal is aligned bottom-right.  window = (left, right): query i
    sees keys i+off-left .. i+off+right (off = Sk - Sq), -1 = unbounded; causal forces right = 0.
    seqused_q / seqused_k (int32 [B]): only the first seqused[b] rows of batch entry b take part; the
    gradient rows behind them are zero.  outputs = (dq, dk, dv): write into these tensors instead of
    allocating.  Calls shaobo_fa3_bwd_v2.
    """
    r = _result(_native.bwd(dout, q, k, v, out, softmax_lse, causal, softmax_scale, deterministic, workspace, return_delta,
                            sync, layout, window, seqused_q, seqused_k, outputs, softcap))
    if sync:
        _raise_on_device_error(capi.load(), "shaobo_fa3_bwd_v2")
    return r


def fa3_fwd(q, k, v, causal: bool, softmax_scale=None, layout: str = "bhsd", window=(-1, -1), sync=False,
            seqused_q=None, seqused_k=None, softcap: float = 0.0):
    """out, softmax_lse = forward of softmax(q k^T * scale) v (shaobo_fa3_b200_fwd).  Shapes, layouts,
    masks as in fa3_bwd; softmax_lse is fp32 [B,Hq,Sq] natural log."""
    return _result(_native.fwd(q, k, v, causal, softmax_scale, layout, window, sync, seqused_q, seqused_k, softcap))


def fa3_fwd_varlen(q, k, v, cu_seqlens_q, cu_seqlens_k, max_seqlen_q: int, max_seqlen_k: int, causal: bool,
                   softmax_scale=None, window=(-1, -1), sync=False):
    """Forward over packed sequences: q [total_q,Hq,D], k/v [total_k,Hkv,D] -> out [total_q,Hq,D],
    softmax_lse fp32 [Hq,total_q]."""
    return _result(_native.fwd_packed(q, k, v, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, causal,
                                      softmax_scale, window, sync))


def fa3_bwd_varlen(dout, q, k, v, out, softmax_lse, cu_seqlens_q, cu_seqlens_k, max_seqlen_q: int,
                   max_seqlen_k: int, causal: bool, softmax_scale=None, deterministic=False, window=(-1, -1),
                   return_delta=False, sync=False):
    """Backward over packed sequences.  q, out, dout: [total_q, Hq, D]; k, v: [total_k, Hkv, D];
    softmax_lse: fp32 [Hq, total_q]; cu_seqlens_*: int32 device tensors of batch+1 row offsets.
    Returns dq, dk, dv in the shapes of q, k, v (and delta [Hq, total_q]).  Calls shaobo_fa3_bwd_v2."""
    r = _result(_native.bwd_packed(dout, q, k, v, out, softmax_lse, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k,
                                   causal, softmax_scale, deterministic, window, return_delta, sync))
    if sync:
        _raise_on_device_error(capi.load(), "shaobo_fa3_bwd_v2")
    return r


class HostBackward:
    """The backward for callers whose tensors live in host memory ([B,H,S,D], pinned for full speed).

    A call copies the inputs to the GPU, runs shaobo_fa3_bwd_v2 and copies dq, dk, dv back.  Large
    problems are cut into contiguous (batch, KV head) shards (the backward has no reduction across
    them) that go round-robin over a few CUDA streams, so that the host-to-device copy of one shard,
    the kernels of another and the device-to-host copy of a third overlap: over PCIe the copies, not
    the kernels, bound such a call.  Device staging tensors, workspaces and the parameter blocks of
    every shard are built once, here; a call itself only issues copies and launches.
    """

    def __init__(self, batch, heads_q, heads_kv, seqlen, head_dim, dtype, causal, softmax_scale=None,
                 shards=None, streams=3, device="cuda"):
        from . import sharding
        self.group = heads_q // heads_kv
        units = batch * heads_kv
        if shards is None:
            # a shard per ~8 MB of traffic: below that the per-shard host work (copies, launches)
            # costs more than the overlap gains (measured on B=1,H=4,S=2048,D=128, 16.8 MB: one shard
            # 389 us, two 370 us, four 419 us)
            elem = torch.empty((), dtype=dtype).element_size()
            total = (5 * batch * heads_q + 4 * batch * heads_kv) * seqlen * head_dim * elem
            shards = max(1, min(8, total // (8 << 20)))
        n = max(1, min(int(shards), units))
        self.shards = [sh for part in sharding.plan(batch, heads_kv, n) for sh in part]
        self._slice = sharding.slice_tensors
        mk = lambda *shape, dt=dtype: torch.empty(shape, dtype=dt, device=device)
        q_shape, kv_shape = (batch, heads_q, seqlen, head_dim), (batch, heads_kv, seqlen, head_dim)
        self.q, self.dout, self.out, self.dq = mk(*q_shape), mk(*q_shape), mk(*q_shape), mk(*q_shape)
        self.k, self.v, self.dk, self.dv = mk(*kv_shape), mk(*kv_shape), mk(*kv_shape), mk(*kv_shape)
        self.lse = mk(batch, heads_q, seqlen, dt=torch.float32)
        self.streams = [torch.cuda.Stream(device=device) for _ in range(max(1, min(streams, len(self.shards))))]
        self.lib = capi.load()
        # per shard: device views, parameter block (workspace and stream filled in), C arguments
        self.plans = []
        need = 0
        for i, sh in enumerate(self.shards):
            d_q, d_kv, d_row = self._slice(sh, self.group, [self.q, self.dout, self.out, self.dq],
                                           [self.k, self.v, self.dk, self.dv], [self.lse])
            p = make_params(d_q[0], d_kv[0], causal, softmax_scale)
            need = max(need, self.lib.shaobo_fa3_bwd_v2_workspace_bytes(ctypes.byref(p)))
            self.plans.append((sh, d_q, d_kv, d_row, p))
        if need == 0:
            raise Fa3Error("shaobo_fa3_bwd_v2_validate", capi.STATUS_UNSUPPORTED)
        self.workspaces = [torch.empty(need, dtype=torch.uint8, device=device) for _ in self.streams]
        self.calls = []
        for i, (sh, d_q, d_kv, d_row, p) in enumerate(self.plans):
            lane = i % len(self.streams)
            p.workspace, p.workspace_bytes = self.workspaces[lane].data_ptr(), need
            p.reserved_ptr[capi.RESERVED_PTR_STREAM] = self.streams[lane].cuda_stream
            args = tuple(_ptr(t) for t in (d_q[1], d_q[0], d_kv[0], d_kv[1], d_q[2], d_row[0], d_q[3], d_kv[2], d_kv[3]))
            self.calls.append(args + (None, ctypes.byref(p)))
        self._host_key, self._host_views = None, None
        self.h2d_bytes = sum(t.numel() * t.element_size() for t in (self.q, self.k, self.v, self.dout, self.out, self.lse))
        self.d2h_bytes = sum(t.numel() * t.element_size() for t in (self.dq, self.dk, self.dv))

    def __call__(self, dout, q, k, v, out, softmax_lse, dq, dk, dv):
        """All nine arguments are host tensors; dq, dk, dv are written.  Returns when the work has been
        queued: the caller's current stream waits for it (synchronise that stream before reading)."""
        main = torch.cuda.current_stream()
        start = torch.cuda.Event()
        start.record(main)
        # the per-shard views of the host tensors are kept for the next call with the same tensors
        key = tuple(t.data_ptr() for t in (dout, q, k, v, out, softmax_lse, dq, dk, dv))
        if key != self._host_key:
            if len(self.plans) == 1:
                self._host_views = [([q, dout, out, dq], [k, v, dk, dv], [softmax_lse])]
            else:
                self._host_views = [self._slice(sh, self.group, [q, dout, out, dq], [k, v, dk, dv], [softmax_lse])
                                    for sh, *_ in self.plans]
            self._host_key = key
        for i, (sh, d_q, d_kv, d_row, _) in enumerate(self.plans):
            st = self.streams[i % len(self.streams)]
            st.wait_event(start)
            h_q, h_kv, h_row = self._host_views[i]
            with torch.cuda.stream(st):
                d_q[0].copy_(h_q[0], non_blocking=True)
                d_kv[0].copy_(h_kv[0], non_blocking=True)
                d_kv[1].copy_(h_kv[1], non_blocking=True)
                d_q[1].copy_(h_q[1], non_blocking=True)
                d_q[2].copy_(h_q[2], non_blocking=True)
                d_row[0].copy_(h_row[0], non_blocking=True)
                code = self.lib.shaobo_fa3_bwd_v2(*self.calls[i])
                if code != capi.STATUS_SUCCESS:
                    raise Fa3Error("shaobo_fa3_bwd_v2", code)
                h_q[3].copy_(d_q[3], non_blocking=True)
                h_kv[2].copy_(d_kv[2], non_blocking=True)
                h_kv[3].copy_(d_kv[3], non_blocking=True)
        for st in self.streams:
            main.wait_stream(st)


class HostBackwardC:
    """The same call as HostBackward, with the shard pipeline inside the library
    (shaobo_fa3_b200_bwd_v2_host): one C call per backward, no per-copy Python overhead.  [B,H,S,D],
    fixed lengths.  The device staging buffer is allocated once, here."""

    def __init__(self, batch, heads_q, heads_kv, seqlen, head_dim, dtype, causal, softmax_scale=None,
                 device="cuda", seqlen_k=None):
        self.lib = capi.load()
        self.p = capi.new_params(batch=batch, seqlen_q=seqlen, seqlen_k=seqlen if seqlen_k is None else seqlen_k,
                                 num_heads_q=heads_q, num_heads_kv=heads_kv, head_dim_qk=head_dim,
                                 head_dim_v=head_dim, causal=int(causal), dtype=_DTYPES[dtype])
        if softmax_scale is not None:
            self.p.softmax_scale = float(softmax_scale)
            self.p.softmax_scale_is_set = 1
        need = self.lib.shaobo_fa3_b200_bwd_v2_host_staging_bytes(ctypes.byref(self.p))
        if need == 0:
            raise Fa3Error("shaobo_fa3_b200_bwd_v2_host_staging_bytes", capi.STATUS_UNSUPPORTED)
        self.staging = torch.empty(need, dtype=torch.uint8, device=device)
        elem = torch.empty((), dtype=dtype).element_size()
        nq, nkv = batch * heads_q * seqlen * head_dim * elem, batch * heads_kv * self.p.seqlen_k * head_dim * elem
        self.h2d_bytes = 3 * nq + 2 * nkv + batch * heads_q * seqlen * 4
        self.d2h_bytes = nq + 2 * nkv

    def __call__(self, dout, q, k, v, out, softmax_lse, dq, dk, dv):
        """Nine host tensors; dq, dk, dv are written once the current stream has been synchronised."""
        for t in (dout, q, k, v, out, softmax_lse, dq, dk, dv):
            if t.is_cuda or not t.is_contiguous():
                raise RuntimeError("contiguous host tensors are required")
        with torch.cuda.device(self.staging.device):
            self.p.reserved_ptr[capi.RESERVED_PTR_STREAM] = torch.cuda.current_stream().cuda_stream or None
            code = self.lib.shaobo_fa3_b200_bwd_v2_host(
                _ptr(dout), _ptr(q), _ptr(k), _ptr(v), _ptr(out), _ptr(softmax_lse), _ptr(dq), _ptr(dk), _ptr(dv),
                _ptr(self.staging), self.staging.numel(), ctypes.byref(self.p))
        if code != capi.STATUS_SUCCESS:
            raise Fa3Error("shaobo_fa3_b200_bwd_v2_host", code)


def default_scale(d: int) -> float:
    return 1.0 / math.sqrt(d)
