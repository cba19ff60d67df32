"""Plan.cg_unrolled / cg_unrolled_adjoint on the host: what they allocate, check, order and hand
to the library, with CPU tensors that pass for device tensors, named streams and a library that
records its calls."""
import ctypes
from contextlib import contextmanager
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

from torch.overrides import TorchFunctionMode  # noqa: E402

from trajsparsenufft_b200 import autograd as tad  # noqa: E402
from trajsparsenufft_b200 import operator as op  # noqa: E402

N, C, M = 4, 4, 10


class _Device(TorchFunctionMode):
    """CPU tensors pass for device tensors; every torch call is logged with its stream."""

    def __init__(self):
        super().__init__()
        self.log = []
        self.stream = self.main = SimpleNamespace(name="main", cuda_stream=1)
        self.side = SimpleNamespace(name="side", cuda_stream=2)
        for s in (self.main, self.side):
            s.wait_stream = lambda other, s=s: self.log.append(("wait", s.name, other.name))

    def __torch_function__(self, func, types, args=(), kwargs=None):
        if func == torch.Tensor.is_cuda.__get__:
            return True
        out = func(*args, **(kwargs or {}))
        self.log.append((getattr(func, "__name__", str(func)), self.stream.name, out))
        return out

    @contextmanager
    def on(self, stream):
        before, self.stream = self.stream, stream
        yield
        self.stream = before

    def native(self, name):
        def call(*args):
            self.log.append((name, {1: "main", 2: "side"}[args[-1].value], args))
            return 0
        return call


@pytest.fixture
def device(monkeypatch):
    d = _Device()
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: d.stream)
    monkeypatch.setattr(torch.cuda, "stream", d.on)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: d.log.append(("record", t.data_ptr(), s.name)))
    fake = SimpleNamespace(**{n: d.native(n) for n in ("tsn_cg_unrolled", "tsn_cg_unrolled_adjoint")})
    monkeypatch.setattr(op, "lib", lambda: fake)
    with d:
        yield d


def _plan():
    p = object.__new__(op.Plan)
    p._h, p.im_size, p.dims, p.coils, p.samples = None, N, 2, C, M
    return p


def _img(*lead):
    return torch.zeros(lead + (N, N), dtype=torch.complex64)


def _arguments(iters, checkpoint):
    """x0, r0, rho0, maps, density, lam, iters, checkpoint, coils of Plan.cg_unrolled"""
    return [_img(), _img(), torch.zeros((), dtype=torch.float64), _img(C), torch.zeros(M), 1e-4, iters, checkpoint, True]


def test_arrays_are_made_on_the_stream_of_the_call(device):
    """Fills and copies that the native loop reads, and the work array that outlives the call only
    in the allocator, belong to the stream of the loop, which first waits for the caller's; what
    comes back is recorded on the caller's stream and the caller's tensors on the call's."""
    plan, args = _plan(), _arguments(3, 2)
    _, saved = plan.cg_unrolled(*args)
    xb, sb, maps, density = _img(), _img(C), args[3], args[4]
    for name, call, ins in (
            ("tsn_cg_unrolled", lambda: plan.cg_unrolled(*args, stream=device.side), args[:5]),
            ("tsn_cg_unrolled_adjoint", lambda: plan.cg_unrolled_adjoint(saved, maps, density, 1e-4, 3, 2, xb, sb,
                                                                         stream=device.side), (*saved, maps, density, xb, sb))):
        device.log.clear()
        out = call()
        made = [e for e in device.log if e[0] in ("empty", "zeros", "zeros_like", "__setitem__", name)]
        assert len(made) > 4 and {e[1] for e in made} == {"side"}, name
        waits = [e for e in device.log if e[0] == "wait"]
        assert waits == [("wait", "side", "main")] and device.log.index(waits[0]) < device.log.index(made[0])
        back = [out[0], *out[1]] if name == "tsn_cg_unrolled" else out
        recorded = {e[1:] for e in device.log if e[0] == "record"}
        assert {(t.data_ptr(), "main") for t in back} | {(t.data_ptr(), "side") for t in ins} == recorded


@pytest.mark.parametrize("checkpoint", [4, 50, 1 << 40])
def test_interval_beyond_the_solve_costs_no_memory(device, checkpoint):
    """A segment holds at most the solve's steps: an interval beyond them allocates what the solve's
    own length does and reaches the library as that."""
    plan, args = _plan(), _arguments(4, checkpoint)
    _, saved = plan.cg_unrolled(*args)
    plan.cg_unrolled_adjoint(saved, args[3], None, 1e-4, 4, checkpoint, _img(), _img(C))
    work = [e[2].numel() for e in device.log if e[0] == "empty" and e[2].dtype == torch.uint8]
    n = N * N
    assert work == [8 * 7 * n + 8 * 296, 8 * n * (3 * 4 + 3 + (4 + 1) * C) + 8 * (2 * 296 + 2)]
    for name in ("tsn_cg_unrolled", "tsn_cg_unrolled_adjoint"):
        assert [e for e in device.log if e[0] == name][0][2][4:6] == (4, 4)


@pytest.mark.parametrize("change", ["iters", "checkpoint", "shape", "dtype", "strides", "conj", "no coil images"])
def test_reverse_pass_checks_what_was_saved(device, change):
    """Arrays saved by another solve, or changed since, are refused before the library reads them."""
    plan, args = _plan(), _arguments(4, 2)
    saved = list(plan.cg_unrolled(*args)[1])
    iters, checkpoint = 4, 2
    if change == "iters":
        iters = 5
    elif change == "checkpoint":
        checkpoint = 1
    elif change == "shape":
        saved[3] = saved[3][:, :2].contiguous()
    elif change == "dtype":
        saved[1] = saved[1].to(torch.float32)
    elif change == "strides":
        saved[4] = saved[4].transpose(-1, -2)
    elif change == "conj":
        saved[0] = saved[0].conj()
    else:
        saved = saved[:4]
    with pytest.raises((TypeError, ValueError)):
        plan.cg_unrolled_adjoint(saved, args[3], None, 1e-4, iters, checkpoint, _img(), _img(C))
    assert not [e for e in device.log if e[0] == "tsn_cg_unrolled_adjoint"]


def test_start_image_may_be_a_conjugated_view(device):
    """The step-by-step solve starts from a copy of x0, which resolves a lazy conjugation; so does the
    native one (tad.PlanOps)."""
    args = _arguments(3, 2)
    want = torch.complex(torch.rand(N, N), torch.rand(N, N))
    for view in (want.conj().resolve_conj().conj(), want.T.contiguous().T):
        states = tad.PlanOps(_plan()).unrolled(view, *args[1:])[1][0]
        assert torch.equal(states[0, 0], want)
