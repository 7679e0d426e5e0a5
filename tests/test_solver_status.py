"""What a solver does with a run that failed on the device (a bounded wait of the
state-on-chip kernel that ran out), on a solver whose device is the CPU: fields are
CPU tensors and the library's status is scripted."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import strata_fdtd_gb300 as S  # noqa: E402
from strata_fdtd_gb300 import _native  # noqa: E402

FIELDS = ("p", "vx", "vy", "vz")
SHAPE = (4, 3, 5)


class _Lib:
    """sf_plan_status answers from `status`, one value per call, then 0."""

    def __init__(self, *status):
        self.status = list(status)

    def sf_plan_status(self, plan):
        return self.status.pop(0) if self.status else 0

    def sf_plan_current(self, plan):
        return 0

    def sf_energy_scratch_doubles(self, plan):
        return 2

    def sf_plan_energy(self, *args):
        return 0


def _solver(*status):
    """A solver behind a run that left 7 everywhere."""
    s = S.FDTDSolver.__new__(S.FDTDSolver)
    s.shape = SHAPE
    s._lib, s._torch, s._plan = _Lib(*status), torch, None
    s._grid = S.UniformGrid(SHAPE, 1e-3)
    s._dev = [[torch.full(SHAPE, 7.0) for _ in FIELDS] for _ in range(2)]
    s._host = {f: np.zeros(SHAPE, dtype=np.float32) for f in FIELDS}
    s._host_fresh = {f: False for f in FIELDS}
    s._host_exposed = {f: False for f in FIELDS}
    s._host_untouched = {f: True for f in FIELDS}
    s._vz_seen = False
    s._pending_traces, s._pending_mics = [], []
    s._probes, s._microphones = {}, {}
    s._boundaries, s._ade_debye, s._ade_lorentz = [], [], []
    s._snap_staged, s._snap_inflight, s._snapshots = [], [], []
    s._velocity_snapshots, s._energy_history = [], []
    return s


def test_a_read_that_failed_leaves_nothing_behind_a_reset():
    s = _solver(1)
    with pytest.raises(_native.NativeError):
        s.p
    s.reset()
    for f in FIELDS:
        assert not s._dev[0][FIELDS.index(f)].any()
        np.testing.assert_array_equal(getattr(s, f), np.zeros(SHAPE, np.float32), err_msg=f)


class _Recorder:
    """Stands for a microphone or a probe."""

    def __init__(self):
        self._data, self._times, self._samples = [], [], []

    def _append(self, rows, times):
        self._data.extend(rows[:, 0].tolist())


def test_microphones_alone_report_a_failed_run():
    s = _solver(1)
    s._microphones["m"] = _Recorder()
    s._pending_mics = [(torch.ones(3, 1), [("m", 1)], [0.0] * 3)]
    with pytest.raises(_native.NativeError):
        s._flush_traces()
    assert s._microphones["m"]._data == []


READS = {
    "probes": lambda s: s.get_probe_data(),
    "flush": lambda s: s._flush_traces(),
    "field": lambda s: s.vy,
    "device": lambda s: s.device_fields(),
    "snapshots": lambda s: s.get_snapshots(),
    "velocities": lambda s: s.get_velocity_snapshots(),
}


@pytest.mark.parametrize("first", READS)
@pytest.mark.parametrize("then", READS)
def test_every_read_raises_until_a_reset(first, then):
    """The library reports a failed run once; its traces are dropped, and whatever is
    read next raises too, until the state is a new one."""
    s = _solver(1)
    s._probes["a"] = _Recorder()
    s._pending_traces = [(torch.ones(3, 1), ["a"]), (torch.ones(2, 1), ["a"])]
    for read in (first, then, first):
        with pytest.raises(_native.NativeError):
            READS[read](s)
    assert s._probes["a"]._samples == [] and s._pending_traces == []
    s.reset()
    s._probes.clear()
    for read in (first, then):
        READS[read](s)


def test_fields_given_by_the_host_end_a_failed_run():
    s = _solver(1)
    with pytest.raises(_native.NativeError):
        s.p
    for f in FIELDS:
        with pytest.raises(_native.NativeError):
            s.device_fields()
        setattr(s, f, np.ones(SHAPE, np.float32))
    assert all(bool((t == 1).all()) for t in s.device_fields().values())


def test_a_trace_that_was_appended_leaves_the_list():
    """A failure between two traces: the first stays with its probe, once."""
    s = _solver(0, 1)  # (asked once behind each trace's copy)
    s._probes["a"] = _Recorder()
    s._pending_traces = [(torch.ones(3, 1), ["a"]), (torch.ones(2, 1), ["a"])]
    for _ in range(2):
        with pytest.raises(_native.NativeError):
            s._flush_traces()
        assert len(s._probes["a"]._samples) == 3


def test_a_failed_run_that_the_tuner_reports_is_not_forgotten(monkeypatch):
    """sf_plan_autotune synchronises and reports it; the fields are void all the same."""
    s = _solver()
    s._lib.sf_plan_autotune = lambda *a: 1
    s._sync_tables = lambda: None
    s._stream = lambda: None
    s._graph_epoch = 0
    monkeypatch.setattr(_native, "check", _failing_check)
    with pytest.raises(_native.NativeError):
        s.autotune()
    for f in FIELDS:
        with pytest.raises(_native.NativeError):
            getattr(s, f)


def _failing_check(rc, what=""):
    if rc:
        raise _native.NativeError(what + ": k_resident: a dependency wait expired (results ...)")
