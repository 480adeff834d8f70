"""Handles in pair-list mode whose lists are gone.  After a rejected edit that had
grown the buffers, steps, forces, energies, neighbour sets and RDF frames are
those of a handle that never saw the edit.  When the lists outgrow the device
memory, an AUTO handle goes on with the cell walk, and one that asked for lists
says so and can still be read and evaluated."""
import numpy as np
import pytest

from readdygpu_b200 import RdgpuError, _abi as A
from readdygpu_b200.system import System, ParticleType, PairPotential

from .test_gpu_pairlist import same
from .test_gpu_parity import Engine
from .test_gpu_run import plain

pytestmark = pytest.mark.gpu


def reject(e, n, born):
    """An edit that deletes one particle and appends `born`, the last of them off the chart."""
    rows = [[0, -1, 0, 0, 0, 7]] + [[1, k % 2, 1.0 + 0.1 * k, 2.0, 3.0, -1] for k in range(born)]
    rows[-1][3] = np.nan
    with pytest.raises(RdgpuError) as err:
        e.apply_edits(rows)
    assert err.value.code == -1 and e.n == n


def observe(e):
    cnt, h = e.neighbor_digest()
    F, en = e.forces()
    return [e.get_particles()[0], F, np.array([en, e.metrics()["energy"]]), cnt, h, e.rdf(40, 18.0, False)[0]]


@pytest.mark.parametrize("prec", ["f32c", "f64"])
@pytest.mark.parametrize("mode", ["cells", "list", "auto"])
@pytest.mark.parametrize("bonds", [False, True])
@pytest.mark.parametrize("born", [3, 300])
def test_rejected_edit_changes_nothing(prec, mode, bonds, born):
    """400 particles have room for 100 more: 3 appended ones fit, 300 grow the
    buffers before their coordinates are looked at."""
    sys_, xyz, types = plain(400)
    ij = np.array([[k, k + 1] for k in range(0, 60) if k % 6 != 5])
    chain = [PairPotential(A.P2_HARMONIC, [], 5.0, "spring", r0=3.0)]
    out = []
    for m, rejecting in (("cells", False), (mode, True)):
        with Engine(sys_, precision=prec, seed=9, neighbour_mode=m, skin=0.8 if m == "list" else 0.0) as e:
            e.set_particles(xyz, types)
            if m == "auto":
                e.autotune()
                assert e.metrics()["neighbour_mode"] == "list"
            if bonds:
                e.set_bonds(ij, np.zeros(len(ij), np.int32), chain)
            e.step(25)
            got = []
            if rejecting:
                reject(e, 400, born)
            got += observe(e)           # evaluated before the next step
            e.step(30)
            got += observe(e)
            if rejecting:
                reject(e, 400, 2 * born)
            e.step(30)                  # stepped before any evaluation
            got += observe(e)
            out.append(got)
    for a, b in zip(*out):
        if a.dtype.kind in "iu":
            assert np.array_equal(a, b)
        elif len(a) == 2:               # energies: FP32 or FP64 sums over the cells, FP64 over the lists
            assert np.abs(a - b).max() <= (1e-5 if prec == "f32c" else 1e-10) * np.abs(a).max()
        else:
            same(prec, a, b)


def clot(n=1_600_000, m=25_000):
    """m of n particles drawn into a cube of edge 1: lists that hold theirs would
    take 200 GB (16-bit entries) or more.  Next to no force, so that the clot stays."""
    sys_, xyz, types = plain(n)
    sys_.pair[0].k = 1e-3
    packed = xyz.copy()
    packed[:m] = 0.5 * sys_.hi[0] + np.random.default_rng(1).uniform(0, 1.0, (m, 3))
    return sys_, xyz, packed, types


def test_untuned_handle_whose_lists_do_not_fit_keeps_the_cell_walk():
    sys_, _, packed, types = clot()
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision="f32c", seed=2, neighbour_mode=mode) as e:
            e.set_particles(packed, types)
            e.step(40)
            e.step(3)
            m = e.metrics()
            out.append(e.get_particles()[0])
    assert m["neighbour_mode"] == "cells" and m["step"] == 43
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("tuned", [False, True])
def test_lists_longer_than_their_heads_can_count(tuned):
    """70,000 particles in a cube of edge 1: more partners than the 16-bit count
    of a list head takes.  AUTO handles keep the cell walk, a handle that asks
    for lists is refused its upload."""
    sys_, _, packed, types = clot(71_000, 70_000)
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision="f32c", seed=2, neighbour_mode=mode) as e:
            e.set_particles(packed, types)
            if tuned:
                e.autotune()
            e.step(40)
            m = e.metrics()
            out.append(e.get_particles()[0])
    assert m["neighbour_mode"] == "cells" and m["step"] == 40
    assert np.array_equal(out[0], out[1])
    with Engine(sys_, precision="f32c", neighbour_mode="list", skin=1.0) as e:
        with pytest.raises(RdgpuError) as err:
            e.set_particles(packed, types)
        assert err.value.code == -6 and "70" in str(err.value)


def test_tuner_passes_over_lists_that_do_not_fit():
    sys_, _, packed, types = clot()
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision="f32c", seed=2, neighbour_mode=mode) as e:
            e.set_particles(packed, types)
            e.autotune()
            e.step(5)
            m = e.metrics()
            out.append(e.get_particles()[0])
    assert m["neighbour_mode"] == "cells" and m["step"] == 5
    assert np.array_equal(out[0], out[1])


def gather(e, xyz, packed, types):
    """One step with the noise that takes every particle from xyz to packed."""
    b = np.sqrt(2.0 * np.array([t.D for t in e.system.types])[types] * e.system.dt)[:, None]
    e.step_with_noise((packed - xyz) / b)


def test_lists_that_outgrow_the_memory_in_a_step():
    """A handle that asks for lists: the step that draws the particles together
    stands and its lists are refused; the state can be read and evaluated, steps
    are refused as long as it lasts, and the next upload steps on."""
    sys_, xyz, packed, types = clot()
    with Engine(sys_, precision="f64", seed=2, neighbour_mode="list", skin=1.0) as e:
        e.set_particles(xyz, types)
        assert e.metrics()["neighbour_mode"] == "list"
        with pytest.raises(RdgpuError) as err:
            gather(e, xyz, packed, types)
        assert err.value.code == -6
        m = e.metrics()
        assert m["step"] == 1 and m["neighbour_mode"] == "list"
        x, t = e.get_particles()
        assert np.abs(x - packed).max() < 1e-3
        F, en = e.forces()
        cnt, h = e.neighbor_digest()
        with Engine(sys_, precision="f64", neighbour_mode="cells") as c:
            c.set_particles(x, t)
            Fc, enc = c.forces()
            cntc, hc = c.neighbor_digest()
            gc = c.rdf(20, 6.0, False)[0]
        assert np.array_equal(cnt, cntc) and np.array_equal(h, hc)
        assert np.linalg.norm(F - Fc) <= 1e-11 * np.linalg.norm(Fc)
        assert abs(en - enc) <= 1e-10 * abs(enc) and m["energy"] == pytest.approx(en, rel=1e-10)
        for _ in range(2):
            with pytest.raises(RdgpuError) as err:
                e.step(1)
            assert err.value.code == -6
        assert np.array_equal(e.rdf(20, 6.0, False)[0], gc)
        assert e.forces()[1] == pytest.approx(enc, rel=1e-10)
        e.set_particles(xyz, types)
        e.step(30)
        y, _ = e.get_particles()
    with Engine(sys_, precision="f64", seed=2, neighbour_mode="cells") as c:
        c.set_particles(xyz, types)
        c.step(30)
        same("f64", c.get_particles()[0], y)


@pytest.mark.parametrize("how", ["step", "upload", "edits"])
@pytest.mark.parametrize("tuned", [False, True])
def test_auto_handle_whose_lists_outgrow_the_memory(how, tuned):
    """An AUTO handle in pair-list mode goes on with the cell walk: through the
    step that draws the particles together, the upload of the clot (a bad
    coordinate is still refused) or the edits that add it."""
    sys_, xyz, packed, types = clot()
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision="f32c", seed=2, neighbour_mode=mode) as e:
            e.set_particles(xyz, types)
            if tuned:
                e.autotune()
            else:
                e.step(100)
                e.set_particles(xyz, types)
            first = e.metrics()["neighbour_mode"]
            if how == "step":
                gather(e, xyz, packed, types)
            elif how == "upload":
                bad = packed.copy()
                bad[3, 1] = np.nan
                with pytest.raises(RdgpuError) as err:
                    e.set_particles(bad, types)
                assert err.value.code == -1
                e.set_particles(packed, types)
            else:
                m = 25_000
                rows = np.zeros((m, 6), np.float32)
                rows[:, 2:5], rows[:, 5] = packed[:m], -1
                e.apply_edits(rows)
            e.step(10)
            last = e.metrics()
            F, en = e.forces()
            out.append((e.get_particles()[0], F))
    assert first == "list" and last["neighbour_mode"] == "cells"
    assert last["step"] == (11 if how == "step" else 10)
    for a, b in zip(*out):
        assert np.array_equal(a, b)


# Pairs a list radius of 9 nm apart on the z axis of a box of 7,000 nm whose
# upper particle is the first FP32 position of its cell.  Seen from the lower
# one, the distance to that cell rounds to more than 9 nm (1 + 5e-5).
LIST_EDGE = [(6765.7744140625, 6774.7744140625), (6585.59423828125, 6594.59423828125),
             (6864.87353515625, 6873.87353515625), (6405.4140625, 6414.4140625),
             (6684.693359375, 6693.693359375), (6225.23388671875, 6234.23388671875)]


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_lists_of_a_long_box_are_symmetric(prec):
    """The pairs meet within one list: the upper particles move far enough to be
    checked, the lower ones not, and the force must act on both."""
    sys_ = System([ParticleType("A", 1e6, 3.0)],
                  pair=[PairPotential(A.P2_HARMONIC, [(0, 0)], 1e4, "repulsive", r0=6.0)],
                  kT=2.437, dt=1e-9, lo=(0, 0, 0), hi=(40, 40, 7000), periodic=(1, 1, 1))
    xyz = np.array([(10.0 + k, 12.0, z) for k, p in enumerate(LIST_EDGE) for z in p])
    types = np.zeros(len(xyz), np.int32)
    move = np.zeros_like(xyz)
    move[0::2, 2], move[1::2, 2] = 0.9, -2.35
    out = []
    for mode in ("cells", "list"):
        with Engine(sys_, precision=prec, seed=2, neighbour_mode=mode, skin=3.0 if mode == "list" else 0.0) as e:
            e.set_particles(xyz, types)
            e.step_with_noise(move / np.sqrt(2.0 * 1e6 * 1e-9))
            F, en = e.forces()
            cnt, _ = e.neighbor_digest()
            e.step(1)
            m = e.metrics()
            out.append((F, cnt, e.get_particles()[0]))
    assert m["neighbour_mode"] == "list" and m["list_builds"] == 1      # the lists of the start
    assert np.array_equal(out[0][1], np.ones(len(xyz))) and np.array_equal(out[1][1], out[0][1])
    for a, b in ((out[0][0], out[1][0]), (out[0][2], out[1][2])):
        same(prec, a, b)


@pytest.mark.parametrize("change", ["upload", "edits", "few edits"])
@pytest.mark.parametrize("before", [40, 120])
def test_trial_of_an_untuned_handle_meets_another_system(change, before):
    """After 40 steps the trial is timing the list: another upload, or edits that
    add 40 % of the particles, send it back to the cell walk; 4 % do not, and
    after 120 steps it is over and its choice stays.  The trajectory is the cell
    walk's throughout."""
    sys_, xyz, types = plain(1000)
    x2 = np.random.default_rng(2).uniform(0, sys_.hi[0], (5000, 3))
    new = x2[:400 if change == "edits" else 40]
    born = np.zeros((len(new), 6), np.float32)
    born[:, 2:5], born[:, 5] = new, -1
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision="f32c", seed=4, neighbour_mode=mode) as e:
            e.set_particles(xyz, types)
            e.step(before)
            first = e.metrics()["neighbour_mode"]
            if change == "upload":
                e.set_particles(x2, np.zeros(len(x2), np.int32))
            else:
                e.apply_edits(born)
            e.step(8)
            second = e.metrics()["neighbour_mode"]
            e.step(90)
            out.append(e.get_particles()[0])
    if before == 40:
        assert first == "list"
    if first == "list":     # (the clock may have chosen the cell walk after 120 steps)
        assert second == ("cells" if before == 40 and change != "few edits" else "list")
    assert np.array_equal(out[0], out[1])
