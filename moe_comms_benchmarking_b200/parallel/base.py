"""Dispatcher interface shared by every transport.

The reference's benchers are duck-typed (README.md:157, bench_*.py); here the protocol is a
small base class: ``build`` (collective allocation), ``setup_batch`` (load one step's
inputs), ``dispatch`` / ``combine`` / ``step`` / ``decode_step`` (the timed operations),
``validate`` (known-value checks -> ``[(name, ok, detail)]``), ``functional_roundtrip``
(dispatch -> identity expert -> combine on given tokens) and ``destroy``.
"""
from __future__ import annotations

import ctypes as C

import torch

from ..config import Config
from ..ops import _ext

_Tensor = torch.Tensor


class Dispatcher:
    name = "base"
    num_sms = -1          # CTA-count knob reported in the CSV (-1 = not applicable)

    def __init__(self, cfg: Config, group, device=None):
        self.cfg = cfg
        self.group = group
        if device is None:
            device = torch.device("cuda", cfg.local_rank) if torch.cuda.is_available() else torch.device("cpu")
        self.device = torch.device(device)
        self._built = False
        self.kernel_launches_per_step = lambda num_layers: 0

    # collective, once
    def build(self):
        raise NotImplementedError

    def setup_batch(self, hidden, topk_idx, topk_weights):
        raise NotImplementedError

    def dispatch(self):
        raise NotImplementedError

    def combine(self):
        raise NotImplementedError

    def step(self):
        self.dispatch()
        self.combine()

    def decode_step(self, num_layers: int):
        for _ in range(num_layers):
            self.step()

    def validate(self):
        return []

    def set_num_sms(self, num_sms: int):
        pass

    def check_health(self):
        """Raise if a kernel of this dispatcher reported an error (host-synchronising)."""

    def destroy(self):
        pass

    # loading one step's inputs into in_hidden / in_routing / in_probs / n_local ------------------------------------
    def _load_rows(self, hidden, topk_idx, topk_weights, pinned: bool = False):
        """This rank's rows for the next step, stream-ordered: one kernel launch when the three tensors have the
        buffers' types, are contiguous and lie on this GPU (or, with ``pinned``, in pinned host memory); copies
        otherwise (other types, strides, devices, negated views or subclasses, which ``copy_`` resolves; or another
        GPU is current, to whose stream the launch would go)."""
        n = hidden.shape[0]
        if n > self.cap:
            raise ValueError(f"{n} local tokens exceed the per-rank capacity {self.cap}")
        self.local_tokens = n
        bufs = (self.in_hidden, self.in_routing, self.in_probs)
        if getattr(self, "_load_for", None) is not self.in_hidden:       # first call since build()
            self._load_for = self.in_hidden
            a = _ext.McbLoadArgs()
            for t, b in enumerate(bufs):
                a.dst[t] = b.data_ptr()
            a.n_local = self.n_local.data_ptr()
            self._load_args, self._load_ref, self._load_src, self._load_bytes = a, C.byref(a), a.src, a.bytes
            self._load_device = self.in_hidden.device.index
            self._load_row = tuple(enumerate((b.dtype, b.device, b.shape[1], b.shape[1] * b.element_size()) for b in bufs))
        a, src, nbytes = self._load_args, self._load_src, self._load_bytes
        rows = (hidden, topk_idx, topk_weights)
        if _ext.current_device() == self._load_device:
            for t, (dtype, device, cols, row_bytes) in self._load_row:
                s = rows[t]
                if (s.dtype is not dtype or s.shape != (n, cols) or not s.is_contiguous() or s.is_neg() or type(s) is not _Tensor
                        or not (s.is_pinned() if pinned else s.device == device)):
                    break
                ptr = s.data_ptr()
                if ptr & 3:
                    break
                src[t], nbytes[t] = ptr, n * row_bytes
            else:
                a.n = n
                err = _ext.require().mcb_launch_load_batch(self._load_ref, int(self.pdl), _ext.stream_handle())
                _ext.check(err, "load_batch")
                return
        if n:
            for b, s in zip(bufs, rows):
                b[:n].copy_(s, non_blocking=True)
        self.n_local.fill_(n)

    # helpers -----------------------------------------------------------------------------------
    def _validation_counts(self, global_b: int):
        w = self.cfg.ep_size
        return [global_b // w + (1 if r < global_b % w else 0) for r in range(w)]
