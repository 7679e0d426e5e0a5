"""The dispatch rules on the host: which grids the state-on-chip kernel takes and
how it cuts them, and where pairs of steps run.  The rules are compiled into a
small program (dispatch_probe.cu) that answers for a device of 152 SMs; no GPU is
used."""
import os
import random
import subprocess

import pytest

from conftest import ROOT
from strata_fdtd_gb300 import _native

MAIL_MAX = 64 << 20  # bytes of mailboxes a launch may use


@pytest.fixture(scope="session")
def ask(tmp_path_factory):
    lib = _native.build()
    exe = str(tmp_path_factory.mktemp("dispatch") / "probe")
    csrc = os.path.join(_native.PKG, "csrc")
    subprocess.run([_native._nvcc(), _native.ARCH, "-O1", "-std=c++17", f"-I{csrc}",
                    f"-I{os.path.join(ROOT, 'include')}",
                    os.path.join(ROOT, "tests", "dispatch_probe.cu"), lib,
                    "-Xlinker", f"-rpath={os.path.dirname(lib)}", "-o", exe],
                   check=True, capture_output=True, text=True)

    def run(lines):
        out = subprocess.run([exe], input="\n".join(lines) + "\n", check=True,
                             capture_output=True, text=True).stdout.splitlines()
        assert len(out) == sum(not q.startswith("room") for q in lines)
        return [r.split() for r in out]

    return run


def _cuts(ask, shapes):
    """(kind, mailbox bytes) per (nx, ny, nz, probes, nu, planes)."""
    rows = ask(["cut %d %d %d %d %d %d" % s for s in shapes])
    out = []
    for r in rows:
        kind, bi, bj, bk, side_max, _ = map(int, r)
        out.append((kind, 2 * bi * bj * bk * 6 * side_max * 4 * 8))
    return out


def test_cuts_keep_their_mailboxes_within_the_limit(ask):
    """Thin grids (a side that no cut crosses used to size the mailboxes) and
    thick ones, uniform and stretched, with and without absorbing planes."""
    rng = random.Random(4)
    shapes = [(1000, 1, 1000), (1200, 1, 1200), (3000, 1, 400), (800, 2, 1000), (1, 1000, 1000),
              (1000, 1000, 1), (2, 2, 200000), (65535, 3, 4), (1, 1, 4), (65535, 1, 30)]
    for _ in range(150):
        thin = rng.choice((1, 1, 2, 3))
        a, b = (int(2 ** rng.uniform(2, 12)) for _ in range(2))
        shapes.append(tuple(rng.sample((thin, a, b), 3)))
    for _ in range(150):
        shapes.append(tuple(int(2 ** rng.uniform(2, 9.2)) for _ in range(3)))
    for extra in ((1, 0, 0), (1, 1, 0), (1, 0, 3)):
        cuts = _cuts(ask, [s + extra for s in shapes])
        assert sum(k >= 0 for k, _ in cuts) > 50
        for s, (kind, mail) in zip(shapes, cuts):
            assert kind < 0 or 0 < mail <= MAIL_MAX, (s, extra, mail)


def test_a_weighted_list_with_a_cell_twice_stays_off_the_chip(ask):
    """A block's list has room for each of its cells once; a sorted list without
    repeats, an unsorted one, and lists with a repeat in either."""
    lists = ([5, 6, 7, 300], [300, 7, 5, 6], [5, 6, 6, 300], [300, 6, 5, 6], [9] * 1000, [4])
    got = ask(["weighted 20 20 20 " + " ".join(map(str, c)) for c in lists])
    assert [int(g[0]) for g in got] == [1, 1, 0, 0, 0, 1]


@pytest.mark.parametrize("succeed", [3, 2, 1])
def test_launches_are_ordered_behind_one_that_was_queued_before_a_failure(ask, succeed):
    """The event that orders the launches of all streams, and that the mailboxes' release
    waits for, is recorded behind what was queued, also where a later launch fails."""
    (calls,) = ask(["steps 40 40 40 9000 %d" % succeed])
    assert calls.index("wait") < calls.index("launch")
    assert calls.count("launch") == min(3, succeed + 1)
    assert calls[-2] == "record" and int(calls[-1]) == (0 if succeed == 3 else 1)


def test_outgrown_mailboxes_are_queued_for_release(ask):
    """Mailboxes grow without cudaFree, which would wait for the device, and are
    allocated in the relaxed capture mode."""
    small, large, again = ask(["steps 20 20 20 9 1000", "steps 100 100 100 9 1000",
                               "steps 20 20 20 9 1000"])
    for calls in (small, large):
        assert calls == "mode malloc mode wait clear launch record 0".split()
    assert again == "wait launch record 0".split()


def test_launches_behind_a_fork_are_plain(ask):
    """On a branch (serial) the first launch of an ADE step has two predecessors and must
    not be a dependent one; the step kernel behind the density pass may be."""
    got = ask(["ade 1 1 1", "ade 0 2 1", "ade 2 0 1", "ade 1 1 0", "ade 0 2 0"])
    assert [" ".join(g) for g in got] == ["plain dependent 0", "plain 0", "plain dependent 0",
                                          "dependent dependent 0", "dependent 0"]


def test_no_memory_for_mailboxes_queues_nothing_and_keeps_the_old_ones(ask):
    """The caller then takes the single-step kernels; a smaller grid still has the
    mailboxes that were there."""
    small, large, again = ask(["steps 20 20 20 9 1000", "room 1000", "steps 100 100 100 9 1000",
                               "steps 20 20 20 9 1000"])
    assert large == "mode mode -1".split()
    assert again == "wait launch record 0".split()


def test_steps_beside_tuned_pairs_run_the_default_kernel(ask):
    """The steps that a tuned two-step configuration leaves over: with walls the kernel
    whose masks do not spill, as for a plan that was not tuned."""
    walls, free, plain = ask(["tuned 300 300 300 1 -1 tb2q_r16 7", "tuned 300 300 300 0 -1 tb2q_r20 5",
                              "tuned 300 300 300 1 -1 - 3"])
    assert walls == ["tb2q_r16"] * 2 + ["tile_r1_w4_m6_wb"] * 3 + ["0"]
    assert plain == ["tile_r1_w4_m6_wb"] * 3 + ["0"]
    assert free[:2] == ["tb2q_r20"] * 2 and free[2:] == ["tile_r1_w4"] + ["0"]


@pytest.mark.parametrize("axis", [-1, 0, 1, 2])
def test_windows_are_left_out_with_a_plane_source_across_their_planes(ask, axis):
    """By the automatic choice and by a tuned plan alike (-1: a point source)."""
    auto, tuned = ask(["pair 300 300 300 1 %d" % axis, "tuned 300 300 300 1 %d tb2q_r16 4" % axis])
    assert auto == (["tb2q_r16"] if axis < 1 else ["-"])
    assert tuned == (["tb2q_r16"] * 2 if axis < 1 else ["tile_r1_w4_m6_wb"] * 4) + ["0"]


# grids of test_gpu_pairs.py: pairs run on them (the padded twin of 223 is 224 wide)
@pytest.mark.parametrize("walls", [0, 1])
@pytest.mark.parametrize("shape,axis,pairs", [((210, 132, 224), 0, True), ((131, 204, 168), 0, True),
                                              ((131, 204, 168), 2, False), ((400, 400, 400), -1, True)])
def test_where_pairs_run(ask, shape, walls, axis, pairs):
    ((name,),) = ask(["pair %d %d %d %d %d" % (shape + (walls, axis))])
    assert name.startswith("tb2q") if pairs else name == "-"


def test_a_tuned_choice_decides_for_small_grids_too(ask):
    """A plan that the tuner has decided on, without having found the state-on-chip
    kernel faster, runs that choice; one that was not tuned stays on the chip."""
    tuned, plain = ask(["tuned 40 40 40 0 -1 tile_r1_w8 9", "tuned 40 40 40 0 -1 - 9"])
    assert tuned == ["tile_r1_w8"] * 9 + ["0"]
    assert plain.count("launch") == 1 and not any(c.startswith("tile") for c in plain)


def test_a_mask_that_fails_waits_before_its_scratch_is_lent_again(ask):
    """Copies and kernels queued before the failure still use it."""
    (calls,) = ask(["mask 40 40 40"])
    assert int(calls[-1]) != 0 and "lent" not in calls
    assert "sync" in calls[calls.index("copy"):]


def test_a_mask_takes_what_memory_there_is(ask):
    """12 MB of scratch for 400^3 cells: with less room the planes are done in slabs."""
    full, less, none = ask(["mask 400 400 400", "room 600000", "mask 500 500 500", "room 1000",
                            "mask 600 600 600"])
    for calls in (full, less):
        assert "malloc" in calls and "copy" in calls
    assert "copy" not in none and int(none[-1]) != 0
