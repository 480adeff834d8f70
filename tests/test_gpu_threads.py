"""Handles of different size that share a kernel, used at the same time from two
threads: each goes its own way, as alone."""
import threading

import numpy as np
import pytest

from readdygpu_b200 import configs

from .test_gpu_pairlist import same
from .test_gpu_parity import Engine, small_config2
from .test_gpu_run import plain

pytestmark = pytest.mark.gpu


def together(jobs):
    """The results of the jobs, run at the same time; the first error of any of them."""
    out, errors = [None] * len(jobs), []
    start = threading.Barrier(len(jobs))

    def go(k):
        try:
            start.wait()
            out[k] = jobs[k]()
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=go, args=(k,)) for k in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]
    return out


def vesicle(n):
    w = configs.config5(n=n)
    return w.system, w.xyz, w.types


@pytest.mark.parametrize("prec", ["f32c", "f64"])
@pytest.mark.parametrize("systems", [(lambda: plain(1000), lambda: plain(30_000)),
                                     (lambda: small_config2(1000), lambda: vesicle(20_000))],
                         ids=["sizes", "types"])
def test_single_steps_in_two_threads(prec, systems):
    """One step per call: 1,000 and 30,000 particles take blocks of 160 and 352
    threads of one variant, and 4 and 3 species tables of different size."""
    made = [s() for s in systems]
    engines = [Engine(m[0], precision=prec, seed=8) for m in made]
    alone = []
    for e, (_, xyz, types) in zip(engines, made):
        e.set_particles(xyz, types)
        e.autotune()
        assert e.metrics()["neighbour_mode"] == "list"
        for _ in range(300):
            e.step(1)
        alone.append(e.get_particles()[0])

    def job(e, xyz, types):
        e.set_particles(xyz, types)
        for _ in range(300):
            e.step(1)
        for _ in range(100):
            e.set_particles(xyz, types)     # a list build by itself
        for _ in range(300):
            e.step(1)
        return e.get_particles()[0]

    for a, b in zip(alone, together([lambda e=e, m=m: job(e, *m[1:]) for e, m in zip(engines, made)])):
        same(prec, a, b)
    for e in engines:
        e.close()


def test_rdf_frames_in_two_threads():
    """1,000 and 2,000 bins: histograms of different size in shared memory."""
    sys_, xyz, types = plain(3000)
    xyz = xyz[types == 0]
    types = types[types == 0]
    sys_.types = sys_.types[:1]
    sys_.pair[0].type_pairs = [(0, 0)]
    engines = [Engine(sys_, precision="f64") for _ in range(2)]
    for e in engines:
        e.set_particles(xyz, types)
    bins = (1000, 2000)
    alone = [e.rdf(b, 12.0, False)[0] for e, b in zip(engines, bins)]

    def job(e, b, want):
        for _ in range(500):
            assert np.array_equal(e.rdf(b, 12.0, False)[0], want)

    together([lambda e=e, b=b, w=w: job(e, b, w) for e, b, w in zip(engines, bins, alone)])
    for e in engines:
        e.close()
