"""Loading one step's inputs into a dispatcher's buffers: which inputs the one-launch loader takes (CPU: the launch is
recorded, the copies run), and that both ways leave exactly the rows and the count (GPU)."""
import types

import pytest
import torch

from moe_comms_benchmarking_b200.ops import _ext
from moe_comms_benchmarking_b200.parallel.base import Dispatcher


class _Buffers(Dispatcher):
    def __init__(self, cap, H, K, device):
        self.cap, self.pdl, self.device = cap, False, torch.device(device)
        self.in_hidden = torch.full((cap, H), -7.0, dtype=torch.bfloat16, device=device)
        self.in_routing = torch.full((cap, K), -7, dtype=torch.int64, device=device)
        self.in_probs = torch.full((cap, K), -7.0, device=device)
        self.n_local = torch.full((1,), -7, dtype=torch.int32, device=device)

    def check(self, h, i, w):
        n = h.shape[0]
        assert self.local_tokens == n and int(self.n_local) == n
        for buf, rows in ((self.in_hidden, h), (self.in_routing, i), (self.in_probs, w)):
            assert torch.equal(buf[:n], rows.to(buf.device, buf.dtype)) and bool((buf[n:] == -7).all())


def _inputs(n, H, K, device):
    return (torch.randn(n, H, device=device).to(torch.bfloat16), torch.randint(0, 512, (n, K), device=device),
            torch.rand(n, K, device=device))


def _shifted(t, by):
    """The same rows `by` elements behind the start of an allocation."""
    s = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)[by:].view(t.shape)
    return s.copy_(t)


def _pinned(t):
    """The same rows in pinned memory, as far behind a 16-byte boundary as they are."""
    by = t.data_ptr() % 16 // t.element_size()
    return torch.empty(t.numel() + by, dtype=t.dtype).pin_memory()[by:].view(t.shape).copy_(t)


FORMS = {
    "plain": lambda h, i, w: (h, i, w),
    "shifted_4_8_4": lambda h, i, w: (_shifted(h, 2), _shifted(i, 1), _shifted(w, 1)),
    "shifted_12_8_12": lambda h, i, w: (_shifted(h, 6), _shifted(i, 1), _shifted(w, 3)),
    "shifted_8_0_8": lambda h, i, w: (_shifted(h, 4), i, _shifted(w, 2)),
    "shifted_2": lambda h, i, w: (_shifted(h, 1), i, w),
    "hidden_fp32": lambda h, i, w: (h.float(), i, w),
    "ids_int32": lambda h, i, w: (h, i.int(), w),
    "weights_fp64": lambda h, i, w: (h, i, w.double()),
    "strided": lambda h, i, w: (h.t().contiguous().t(), torch.cat([i, i], 1)[:, :i.shape[1]], w),
    "negated": lambda h, i, w: (h, i, torch._neg_view(-w)),
    "parameter": lambda h, i, w: (torch.nn.Parameter(h, requires_grad=False), i, w),
}
LAUNCHED = ("plain", "shifted_4_8_4", "shifted_12_8_12", "shifted_8_0_8")


@pytest.mark.parametrize("form", list(FORMS) + ["other_device"])
def test_loader_takes_only_rows_it_can_read(monkeypatch, form):
    """Contiguous rows of the buffers' types, 4-byte aligned, while the buffers' GPU is the current one; the rest is copied."""
    d = _Buffers(8, 16, 3, "cpu")
    launched = []
    fake = types.SimpleNamespace(mcb_launch_load_batch=lambda ref, pdl, stream: launched.append(d._load_args.n) or 0)
    monkeypatch.setattr(_ext, "require", lambda: fake)
    monkeypatch.setattr(_ext, "stream_handle", lambda: 0)
    monkeypatch.setattr(_ext, "current_device", lambda: 1 if form == "other_device" else None)     # None: the index of "cpu"
    rows = FORMS.get(form, FORMS["plain"])(*_inputs(5, 16, 3, "cpu"))
    d._load_rows(*rows)
    if form in LAUNCHED:
        assert launched == [5] and list(d._load_args.bytes) == [5 * 32, 5 * 24, 5 * 12]
        assert [d._load_args.src[t] for t in range(3)] == [t.data_ptr() for t in rows]
    else:
        assert not launched
        d.check(*rows)


def test_loader_refuses_more_rows_than_the_capacity():
    with pytest.raises(ValueError):
        _Buffers(8, 16, 3, "cpu")._load_rows(*_inputs(9, 16, 3, "cpu"))


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1, 5, 7, 22])
@pytest.mark.parametrize("form", list(FORMS))
def test_load_rows_on_the_gpu(lib, form, K):
    for n in (0, 1, 3, 31, 40):
        for host, pinned in ((False, False), (True, True), (True, False)):
            rows = FORMS[form](*_inputs(n, 24, K, "cpu" if host else "cuda:0"))
            if pinned and form in LAUNCHED:
                rows = tuple(_pinned(r) for r in rows)
            d = _Buffers(40, 24, K, "cuda:0")
            d._load_rows(*rows, pinned=host)
            torch.cuda.synchronize()
            d.check(*rows)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 2])
def test_load_rows_larger_than_one_round_of_the_grid(lib, shift):
    """More packs than the loader's blocks take in one round (592 blocks x 256 threads x 4 packs are 9.7 MB)."""
    n, H, K = 6001, 1032, 5
    d = _Buffers(n + 2, H, K, "cuda:0")
    h, i, w = _inputs(n, H, K, "cuda:0")
    rows = (_shifted(h, shift), i, _shifted(w, shift))
    d._load_rows(*rows)
    torch.cuda.synchronize()
    d.check(*rows)
