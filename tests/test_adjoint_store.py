"""The pressures that a forward pass keeps for its backward pass, on a solver whose
device is the CPU and whose kernels only note what they are given."""
import types

import pytest

torch = pytest.importorskip("torch")

from strata_fdtd_gb300 import adjoint  # noqa: E402

SHAPE, N = (4, 3, 5), 60
DEVICE_BYTES = 16 * 60000  # a sixteenth of it holds 60000 bytes


class _Lib:
    """Notes (what, steps, address of the stored pressures) per call."""

    def __init__(self):
        self.calls = []

    def sf_diff_forward(self, desc, cv, s0, s1, cur, n, src, trace, store, stream):
        self.calls.append(("forward", n, store))
        return 0

    def sf_diff_adjoint(self, desc, cv, l0, l1, cur, n, store, trace, target, w, grad, stream):
        self.calls.append(("adjoint", n, store))
        return 0

    def sf_diff_grad_fields(self, *a):
        return 0


class _Torch:
    """torch with a device of DEVICE_BYTES."""

    def __init__(self):
        self.cuda = types.SimpleNamespace(
            get_device_properties=lambda dev: types.SimpleNamespace(total_memory=DEVICE_BYTES),
            current_stream=lambda: types.SimpleNamespace(cuda_stream=None),
            OutOfMemoryError=torch.cuda.OutOfMemoryError)

    def __getattr__(self, name):
        return getattr(torch, name)


def _solver(K):
    s = adjoint.DifferentiableSolver.__new__(adjoint.DifferentiableSolver)
    s.torch, s.lib, s.dev, s.K = _Torch(), _Lib(), torch.device("cpu"), K
    s.shape, s.n, s.precision = SHAPE, N, "f64"
    s.dtype = s.ext_dtype = torch.float64
    s.probe_pos = [(0, 0, 0)]
    s._desc = lambda occ=None: adjoint._Desc()
    s.coefficients = lambda theta, occ=None: [torch.zeros(SHAPE, dtype=s.dtype) for _ in range(3)]
    s._source_table = lambda n: torch.zeros(n, dtype=s.dtype)
    s.stores = {}
    plain = s._segment_store

    def store(*a):
        t = plain(*a)
        s.stores[t.data_ptr()] = t.shape[0]
        return t

    s._segment_store = store
    return s


def _loss(s, steps):
    theta = torch.zeros(SHAPE, dtype=torch.float64, requires_grad=True)
    return s.loss(theta, torch.zeros((steps, 1), dtype=torch.float64), steps), theta


@pytest.mark.parametrize("after", [3, 10, 40])
def test_a_backward_pass_keeps_the_segments_of_its_forward_pass(after):
    """checkpoint spacing changed between the two: every call's steps fit the store it
    is given, and the segments are the ones the checkpoints were made at."""
    s = _solver(10)
    loss, _ = _loss(s, 25)
    first = list(s.lib.calls)
    s.K = after
    loss.backward()
    assert [c[:2] for c in first] == [("forward", 10), ("forward", 10), ("forward", 5)]
    assert [c[:2] for c in s.lib.calls[3:]] == [("adjoint", 5), ("forward", 10), ("adjoint", 10),
                                                ("forward", 10), ("adjoint", 10)]
    assert all(n <= s.stores[at] for _, n, at in s.lib.calls if at is not None)


def test_losses_that_wait_share_one_bound():
    """24000 bytes each, 60000 for all: the third loss keeps nothing, a loss that was
    dropped or has had its backward pass makes room for the next."""
    s = _solver(50)
    kept = lambda: s.lib.calls[-1][2] is not None  # noqa: E731
    losses = []
    for expect in (True, True, False, False):
        losses.append(_loss(s, 60))
        assert kept() == expect
    del losses[0]
    losses.append(_loss(s, 60))
    assert kept()
    losses[0][0].backward()
    assert losses[0][1].grad is not None
    losses.append(_loss(s, 60))
    assert kept()
    losses.append(_loss(s, 60))
    assert not kept()


def test_a_solve_that_runs_out_of_memory_takes_the_waiting_pressures():
    """Forward and backward passes run again without them, and the losses that lost
    theirs recompute them."""
    s = _solver(50)
    waiting, _ = _loss(s, 60)
    plain, left = s._zeros4, [1]

    def short():
        if left[0]:
            left[0] -= 1
            raise torch.cuda.OutOfMemoryError("no room")
        return plain()

    s._zeros4 = short
    other, _ = _loss(s, 60)
    assert s.lib.calls[-1][2] is None  # (its own were dropped too)
    del s.lib.calls[:]
    waiting.backward()
    assert [c[:2] for c in s.lib.calls] == [("forward", 10), ("adjoint", 10), ("forward", 50),
                                            ("adjoint", 50)]
    again, _ = _loss(s, 60)
    left[0] = 1
    del s.lib.calls[:]
    other.backward()
    assert [c[0] for c in s.lib.calls] == ["forward", "adjoint"] * 2
    with pytest.raises(torch.cuda.OutOfMemoryError):
        left[0] = 2
        _loss(s, 60)
