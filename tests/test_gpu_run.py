"""The pair-list steps of an AUTO handle run in one launch per rdgpu_step call
(list_run_kernel): the trajectory is the cell walk's, bit for bit in FP32C and
to rounding in FP64, at the sizes where its shape changes (one block per SM;
up to 8 and 13 tiles of 32 particles per SM a warp keeps its tile, beyond that
the warps draw tiles), for every potential path, across rebuilds and whatever
the split of the steps."""
import numpy as np
import pytest

from readdygpu_b200 import RdgpuError, _abi as A, configs
from readdygpu_b200.system import System, ParticleType, PairPotential, ExternalPotential

from .test_gpu_pairlist import cluster_system, same
from .test_gpu_parity import Engine, small_config2

pytestmark = pytest.mark.gpu


def plain(n, per=(1, 1, 1)):
    L = float(np.float32(max(40.0, 50.0 * (n / 1000.0) ** (1.0 / 3.0))))
    sys_ = System([ParticleType("A", 1e6, 1.5), ParticleType("B", 5e5, 2.0)],
                  pair=[PairPotential(A.P2_HARMONIC, [(0, 0), (0, 1), (1, 1)], 10.0, "repulsive")],
                  kT=2.437, dt=1e-9, lo=(0, 0, 0), hi=(L, L, L), periodic=per)
    xyz = np.random.default_rng(n).uniform(0.2 * L, 0.8 * L, (n, 3)) if 0 in per else \
        np.random.default_rng(n).uniform(0, L, (n, 3))
    return sys_, xyz, (np.arange(n) % 2).astype(np.int32)


def both(prec, sys_, xyz, types, split, boxes=None, offsets=None):
    """Final positions of the cell walk and of the run kernel, whose calls are one launch each."""
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision=prec, seed=3, boxes=boxes, neighbour_mode=mode) as e:
            e.set_particles(xyz, types, offsets=offsets)
            e.autotune()
            m0 = e.metrics()
            l0 = e.launch_count()
            for n in split:
                e.step(n)
            if mode == "auto":
                assert m0["neighbour_mode"] == "list"
                assert e.launch_count() - l0 == len(split)
            m = e.metrics()
            assert m["step"] == sum(split)
            out.append(e.get_particles()[0])
    return out[0], out[1], m["list_builds"] - m0["list_builds"]


# tiles of 32 particles on 148 SMs: warps that keep their tile up to 37,888 and
# 61,568 particles (two block sizes), a warp per tile up to 132,608 (FP64) and 151,552 (FP32C)
@pytest.mark.parametrize("prec", ["f32c", "f64"])
@pytest.mark.parametrize("n", [1, 33, 1000, 4737, 37_888, 37_889, 61_569, 132_609, 151_553])
def test_run_equals_cells_over_sizes(prec, n):
    sys_, xyz, types = plain(n)
    xc, xr, _ = both(prec, sys_, xyz, types, [1, 60, 39])
    same(prec, xc, xr)


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_equals_cells_over_rebuilds(prec):
    """1,500 steps in one call (two launches), with many rebuilds inside them."""
    sys_, xyz, types = plain(3000)
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision=prec, seed=3, neighbour_mode=mode) as e:
            e.set_particles(xyz, types)
            e.autotune()
            b0 = e.metrics()["list_builds"]
            e.step(1500)
            m = e.metrics()
            out.append(e.get_particles()[0])
    assert m["neighbour_mode"] == "list" and m["list_builds"] - b0 > 10
    same(prec, out[0], out[1])


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_general_potentials_and_open_axes(prec):
    """Weak attraction, a disk and an open z axis (the term-table variant)."""
    sys_, xyz, types = small_config2(1000)
    xc, xr, _ = both(prec, sys_, xyz, types, [130])
    same(prec, xc, xr)


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_open_axis_repulsion(prec):
    """Harmonic repulsion with an open axis (the per-axis variant)."""
    sys_, xyz, types = plain(2000, per=(1, 1, 0))
    xc, xr, _ = both(prec, sys_, xyz, types, [130])
    same(prec, xc, xr)


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_small_batch(prec):
    """Tiles that span systems, kept by their warps, across rebuilds."""
    w = configs.config4(n_systems=12, nmin=200, nmax=3000)
    xc, xr, nb = both(prec, w.system, w.xyz, w.types, [150, 1, 49], boxes=w.boxes, offsets=w.offsets)
    assert nb > 3
    same(prec, xc, xr)


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_batch_of_many_tiles(prec):
    """An uneven batch of several tiles per warp."""
    w = configs.config4(n_systems=140)
    xc, xr, nb = both(prec, w.system, w.xyz, w.types, [100], boxes=w.boxes, offsets=w.offsets)
    assert w.n > 4 * 32 * 148 * 32 and nb > 1
    same(prec, xc, xr)


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_overflow_regrows(prec):
    """A cluster drawn together by attraction overflows the lists inside a call."""
    sys_, xyz, types = cluster_system(n_gas=3000, n_cluster=60)
    sys_.pair.append(PairPotential(A.P2_WEAK_PIECEWISE, [(0, 0)], 60.0, r0=2.0, length=4.0, depth=40.0))
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision=prec, seed=5, neighbour_mode=mode) as e:
            e.set_particles(xyz, types)
            e.autotune()
            e.step(100)
            out.append(e.get_particles()[0])
    same(prec, out[0], out[1])


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_reports_a_failed_step(prec):
    """Two overlapping particles under an enormous force constant leave the box
    by more than an edge in one step: the step is reported and its input stays,
    as with the cell walk."""
    res = []
    for mode in ("cells", "auto"):
        sys_, xyz, types = plain(500)
        sys_.pair[0].k = 1e12
        xyz[1] = xyz[0] + 0.3
        with Engine(sys_, precision=prec, seed=5, neighbour_mode=mode) as e:
            e.set_particles(xyz, types)
            with pytest.raises(RdgpuError) as err:
                e.autotune()
                e.step(50)
            res.append((err.value.code, str(err.value).split("at step")[-1]))
            x, _ = e.get_particles()
            assert np.isfinite(x).all()
    assert res[0] == res[1]


def slab():
    """200,000 particles whose neighbour cells lie more than 32,767 sorted places apart (32-bit list entries)."""
    n = 200_000
    sys_ = System([ParticleType("A", 1e6, 1.0)], pair=[PairPotential(A.P2_HARMONIC, [(0, 0)], 10.0, "repulsive")],
                  kT=2.437, dt=1e-9, lo=(0, 0, 0), hi=(600, 600, 12), periodic=(1, 1, 1))
    return sys_, np.random.default_rng(4).uniform((0, 0, 0), (600, 600, 12), (n, 3)), np.zeros(n, np.int32), 4


@pytest.mark.parametrize("system", ["slab", "mixed", "lone"])
def test_diagnostics_over_the_list(system):
    """Forces, energy and neighbour sets evaluated over the list of a running
    handle equal those of a cell walk of the same positions: 32- and 16-bit
    entries, several terms per pair and an open axis, empty lists."""
    if system == "slab":
        sys_, xyz, types, width = slab()
    elif system == "mixed":
        sys_, xyz, types = small_config2(3000)
        width = 2
    else:
        sys_, xyz, types = plain(40)
        xyz, types, width = xyz[:1], types[:1], 2
    with Engine(sys_, precision="f64", seed=3, neighbour_mode="list", skin=1.0) as e:
        e.set_particles(xyz, types)
        e.step(37)
        x, t = e.get_particles()
        F, en = e.forces()
        cnt, h = e.neighbor_digest()
        m = e.metrics()
        assert m["list_entry_bytes"] == width and m["energy"] == en
        with Engine(sys_, precision="f64", neighbour_mode="cells") as c:
            c.set_particles(x, t)
            Fc, enc = c.forces()
            cntc, hc = c.neighbor_digest()
        assert np.array_equal(cnt, cntc) and np.array_equal(h, hc)
        assert np.linalg.norm(F - Fc) <= 1e-12 * np.linalg.norm(Fc)
        assert abs(en - enc) <= 1e-10 * abs(enc)
        # the evaluation leaves the run as it was
        e.step(20)
        y, _ = e.get_particles()
    with Engine(sys_, precision="f64", seed=3, neighbour_mode="list", skin=1.0) as e:
        e.set_particles(xyz, types)
        e.step(57)
        same("f64", e.get_particles()[0], y)


@pytest.mark.parametrize("prec", ["f32c", "f64"])
@pytest.mark.parametrize("system,split", [("plain", [100, 40]), ("plain", [7] * 18), ("plain", [1] * 110),
                                          ("mixed", [100]), ("small box", [100])])
def test_untuned_handle_tries_the_list(prec, system, split):
    """An AUTO handle that is never tuned and only gets short calls changes from
    the cell walk to the pair list (and maybe back) within its first 100 steps;
    the trajectory is the cell walk's.  A box too small for lists keeps the
    cell walk."""
    if system == "mixed":
        sys_, xyz, types = small_config2(3000)
    else:
        sys_, xyz, types = plain(3000)
        if system == "small box":
            sys_.hi = (10.0, 10.0, 10.0)
            xyz, types = xyz[:20] % 10.0, types[:20]
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision=prec, seed=4, neighbour_mode=mode) as e:
            e.set_particles(xyz, types)
            for n in split:
                e.step(n)
            m = e.metrics()
            out.append(e.get_particles()[0])
    assert m["step"] == sum(split)
    if system == "small box":
        assert m["neighbour_mode"] == "cells"
    same(prec, out[0], out[1])


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_tiles_in_the_order_of_their_cost(prec):
    """Several tiles per warp and several potentials (the ordered variant),
    across rebuilds and calls: the vesicle."""
    w = configs.config5(n=160_000)
    xc, xr, nb = both(prec, w.system, w.xyz, w.types, [40, 1, 19])
    assert nb > 1
    same(prec, xc, xr)


@pytest.mark.parametrize("prec", ["f32c", "f64"])
@pytest.mark.parametrize("out", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 1755, 1756, 3072, 3073])
def test_download_sizes(prec, out, n):
    """Downloads up to 48 KB (1,755 FP64 or 3,072 FP32 frames) and larger ones
    return the particles in their order, in either coordinate type."""
    sys_, xyz, types = plain(n)
    xyz = xyz.astype(np.float32)
    with Engine(sys_, precision=prec) as e:
        e.set_particles(xyz, types)
        x, t = e.get_particles(np.empty((n, 3), out), np.empty(n, np.int32))
    assert np.array_equal(x, xyz.astype(out)) and np.array_equal(t, types)


def test_run_wide_entries():
    """32-bit list entries in the run kernel."""
    sys_, xyz, types, width = slab()
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision="f32c", seed=3, neighbour_mode=mode) as e:
            e.set_particles(xyz, types)
            e.autotune()
            e.step(40)
            m = e.metrics()
            out.append(e.get_particles()[0])
    assert m["neighbour_mode"] == "list" and m["list_entry_bytes"] == width
    same("f32c", out[0], out[1])


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_with_bonds_edits_and_uploads(prec):
    """Bonded chains, reaction edits, a rejected upload and a new upload on a
    handle whose steps and list builds run in one launch: the cell walk's
    positions throughout."""
    sys_, xyz, types = plain(3000)
    chain = [PairPotential(A.P2_HARMONIC, [], 5.0, "spring", r0=3.0)]
    ij = np.array([[k, k + 1] for k in range(0, 600) if k % 6 != 5])
    gone = [[k, -1, 0, 0, 0, k] for k in (0, 17, 599, 2999)]
    born = [[0, 1, 5.0 + k, 6.0, 7.0, -1] for k in range(3)]
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision=prec, seed=6, neighbour_mode=mode) as e:
            e.set_particles(xyz, types)
            e.autotune()
            e.set_bonds(ij, np.zeros(len(ij), np.int32), chain)
            got = []
            e.step(60)
            got.append(e.get_particles()[0])
            e.apply_edits(gone + born)
            e.step(60)
            got.append(e.get_particles()[0])
            got.append(e.forces()[0])
            for bad_x, bad_t in ((np.nan, 0), (1e6, 0), (1.0, 7)):
                bx, bt = xyz.copy(), types.copy()
                bx[5, 1], bt[5] = bad_x, bad_t
                with pytest.raises(RdgpuError) as err:
                    e.set_particles(bx, bt)
                assert err.value.code == -1
            e.set_particles(xyz[::-1], types[::-1])
            e.step(30)
            got.append(e.get_particles()[0])
            assert e.metrics()["step"] == 30
        out.append(got)
    for a, b in zip(*out):
        same(prec, a, b)


def test_two_handles_in_two_threads():
    """Two handles too large to be resident together, stepped at the same time
    from two threads, go their own way unchanged."""
    import threading
    sys_, xyz, types = plain(160_000)
    alone, together = {}, {}

    def go(seed, out):
        with Engine(sys_, precision="f32c", seed=seed) as e:
            e.set_particles(xyz, types)
            e.autotune()
            for _ in range(6):
                e.step(50)
            out[seed] = e.get_particles()[0]

    for seed in (1, 2):
        go(seed, alone)
    ts = [threading.Thread(target=go, args=(seed, together)) for seed in (1, 2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for seed in (1, 2):
        assert np.array_equal(alone[seed], together[seed])


@pytest.mark.parametrize("prec", ["f32c", "f64"])
@pytest.mark.parametrize("m", [4, 41])
@pytest.mark.parametrize("gap", [-0.5, 0.3])
def test_run_kernel_reports_a_failed_step(prec, m, gap):
    """Particles on a grid (64: warps that keep their tile, 68,921: several
    tiles per warp), tuned to the list, then eight pairs of them next to each
    other: overlapping at once, or a few steps later.  Under an enormous force
    constant the first overlap is a jump.  Its step, the state before it and
    its forces are the cell walk's, and the next upload steps on."""
    L = 14.0 * m
    sys_ = System([ParticleType("A", 1e6, 1.5)],
                  pair=[PairPotential(A.P2_HARMONIC, [(0, 0)], 1e12, "repulsive", r0=3.5)],
                  kT=2.437, dt=1e-9, lo=(0, 0, 0), hi=(L, L, L), periodic=(1, 1, 1))
    g = 14.0 * np.arange(m) + 7.0
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    types = np.zeros(len(xyz), np.int32)
    near = xyz.copy()
    near[1:16:2] = near[0:16:2] + [3.5 + gap, 0, 0]
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision=prec, seed=5, neighbour_mode=mode) as e:
            e.set_particles(xyz, types)
            e.autotune()
            e.set_particles(near, types)
            assert mode == "cells" or e.metrics()["neighbour_mode"] == "list"
            l0 = e.launch_count()
            with pytest.raises(RdgpuError) as err:
                e.step(100)
            assert mode == "cells" or e.launch_count() == l0 + 1
            assert err.value.code == -7
            t = int(str(err.value).split("at step")[-1])
            assert t == 0 if gap < 0 else 1 < t < 100
            assert e.metrics()["step"] == t
            got = [e.get_particles()[0], e.forces()[0]]
            with pytest.raises(RdgpuError) as err:      # the same step again
                e.step(3)
            assert int(str(err.value).split("at step")[-1]) == t
            got.append(e.get_particles()[0])
            e.set_particles(xyz, types)
            e.step(20)
            got.append(e.get_particles()[0])
            out.append((t, got))
    assert out[0][0] == out[1][0]
    for k, (a, b) in enumerate(zip(out[0][1], out[1][1])):
        if prec == "f64" and k == 1:
            assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(a)
        else:
            same(prec, a, b)


@pytest.mark.parametrize("prec", ["f32c", "f64"])
def test_run_kernel_overflow_regrows(prec):
    """3,000 particles that a sphere's pull draws together within one call: lists
    made for the dispersed state overflow inside list_run_kernel and grow."""
    sys_ = System([ParticleType("A", 1e6, 1.0), ParticleType("B", 1e6, 1.0)],
                  pair=[PairPotential(A.P2_HARMONIC, [(0, 0), (0, 1), (1, 1)], 0.01, "repulsive", r0=3.0)],
                  external=[ExternalPotential(A.P1_SPHERE, [1], 100.0, "attractive", center=(40, 40, 40), radius=3.0)],
                  kT=2.437, dt=1e-9, lo=(0, 0, 0), hi=(80, 80, 80), periodic=(1, 1, 1))
    n = 3000
    xyz = np.random.default_rng(3).uniform(0, 80, (n, 3))
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision=prec, seed=5, neighbour_mode=mode) as e:
            e.set_particles(xyz, np.zeros(n, np.int32))     # type A is not drawn
            e.autotune()
            e.set_particles(xyz, np.ones(n, np.int32))
            m0 = e.metrics()
            e.step(100)
            m1 = e.metrics()
            e.step(30)
            out.append(e.get_particles()[0])
    assert m0["neighbour_mode"] == m1["neighbour_mode"] == "list"
    assert m1["list_capacity"] > m0["list_capacity"] and m1["step"] == 100
    same(prec, out[0], out[1])


@pytest.mark.parametrize("system", ["slab", "mixed", "batch"])
def test_fp32_diagnostics_over_the_list(oracle, system):
    """FP32C, a running AUTO handle: forces, energy and neighbour sets over its
    lists (32-bit entries, several terms per pair, a batch) are those of a cell
    walk that made the same steps: forces and sets to the bit, the energy, which
    the cells sum in FP32, to its rounding; and the oracle's."""
    boxes = offsets = None
    if system == "slab":
        sys_, xyz, types, width = slab()
    elif system == "mixed":
        sys_, xyz, types = small_config2(3000)
        width = 2
    else:
        w = configs.config4(n_systems=12, nmin=200, nmax=3000)
        sys_, xyz, types, boxes, offsets, width = w.system, w.xyz, w.types, w.boxes, w.offsets, 2
    out = []
    for mode in ("cells", "auto"):
        with Engine(sys_, precision="f32c", seed=3, boxes=boxes, neighbour_mode=mode) as e:
            e.set_particles(xyz, types, offsets=offsets)
            e.autotune()
            e.step(37)
            m = e.metrics()
            out.append((e.get_particles()[0], *e.forces(), *e.neighbor_digest(), m["energy"]))
    assert m["neighbour_mode"] == "list" and m["list_entry_bytes"] == width
    (x, F, en, cnt, h, en2), (xl, Fl, enl, cntl, hl, enl2) = out
    assert np.array_equal(x, xl) and np.array_equal(F, Fl) and np.array_equal(cnt, cntl) and np.array_equal(h, hl)
    assert enl == enl2 and abs(enl - en) <= 1e-5 * abs(en)
    if system == "mixed":
        hi, comp = oracle.to_rel_f32(sys_.to_desc(), xl)
        Fo, eo = oracle.forces_f64(sys_.to_desc(), hi.astype(np.float64).reshape(-1, 3), types)
        assert abs(enl - eo) <= 1e-5 * abs(eo)
        assert np.linalg.norm(Fl - Fo) <= 1e-5 * np.linalg.norm(Fo)
