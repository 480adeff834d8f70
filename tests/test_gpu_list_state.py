"""Handles in pair-list mode whose lists are gone.  After a rejected edit that had
grown the buffers, steps, forces, energies, neighbour sets and RDF frames are
those of a handle that never saw the edit.  When the lists outgrow the device
memory, the call that needs them says so and the rest goes on."""
import numpy as np
import pytest

from readdygpu_b200 import RdgpuError, _abi as A
from readdygpu_b200.system import PairPotential

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


@pytest.mark.parametrize("mode", ["list", "auto"])
def test_lists_that_outgrow_the_memory_in_a_step(mode):
    """The step that draws the particles together stands and its lists are
    refused; the state can be read and evaluated, steps are refused as long as
    it lasts, and the next upload steps on."""
    sys_, xyz, packed, types = clot()
    n = len(xyz)
    b = np.sqrt(2.0 * np.array([t.D for t in sys_.types])[types] * sys_.dt)[:, None]
    with Engine(sys_, precision="f64", seed=2, neighbour_mode=mode, skin=1.0 if mode == "list" else 0.0) as e:
        e.set_particles(xyz, types)
        if mode == "auto":
            e.autotune()
        assert e.metrics()["neighbour_mode"] == "list"
        with pytest.raises(RdgpuError) as err:
            e.step_with_noise((packed - xyz) / b)
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
