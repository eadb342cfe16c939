"""GPU: both ways a batch advances a model, each in every tiling: the persistent
launch (handles told to stream, many small models) and runs on chip.  Whichever a run
takes, every model gets the bits of its own run."""
import numpy as np
import pytest

from helpers import make_solver
from seidart_gb300 import ELECTROMAG2, SEISMIC2
from seidart_gb300 import synthetic as sy
from seidart_gb300.batch import Batch, autotune
from seidart_gb300.solver import FIELDS, FLAG_LEGACY_QUIRKS, FLAG_STREAMING, FDTDSolver, MEMORY

pytestmark = pytest.mark.gpu


def cases(n, nstep, seed=300):
    return [sy.small_case(ELECTROMAG2 if q % 3 else SEISMIC2, seed=seed + q, nx=41 + 3 * (q % 7), nz=37 + 2 * (q % 5),
                          npml=5, nstep=nstep) for q in range(n)]


def results(s):
    return [s.traces()] + [s.field(f) for f in FIELDS[s.kind]] + [s.memory(m) for m in MEMORY[s.kind]]


def check(cs, solvers, flags=0):
    for c, s in zip(cs, solvers):
        with make_solver(c, flags=flags) as one:
            one.run(c.nstep)
            one.status()
            for a, b in zip(results(s), results(one)):
                assert np.array_equal(a, b)
        s.close()


@pytest.mark.parametrize("zb,bps", [(1, 3), (2, 3), (4, 2)])
def test_tilings_of_the_persistent_launch(gpu, zb, bps):
    cs = cases(6, 60)
    solvers = [make_solver(c, flags=FLAG_STREAMING) for c in cs]
    b = Batch(solvers)
    assert b.on_chip(60) == 0
    b.set_tiling(zb, bps)
    b.run(37)  # odd: the ping-pong parity differs between the two runs
    b.run(23)
    b.status()
    b.close()
    check(cs, solvers)


def test_shared_model(gpu):
    """Shots that read one model's coefficients take interleaved tiles."""
    base = sy.small_case(ELECTROMAG2, seed=70, nx=170, nz=44, npml=6, nstep=64)
    solvers, alone = [], []
    for q in range(5):
        for group in (solvers, alone):
            s = FDTDSolver(base.grid, base.nstep, len(base.rec_ijk), flags=FLAG_STREAMING)
            if group is solvers and group:
                s.share_model(group[0])
            else:
                s.set_model(base.planes)
            s.set_cpml(base.profiles)
            s.set_source((10 + 30 * q, 0, 12), base.srcfn)
            s.set_receivers(base.rec_ijk)
            group.append(s)
    b = Batch(solvers)
    b.run(base.nstep)
    b.status()
    b.close()
    for a, s in zip(alone, solvers):
        a.run(base.nstep)
        a.status()
        for x, y in zip(results(a), results(s)):
            assert np.array_equal(x, y)
        a.close()
        s.close()


@pytest.mark.parametrize("models,flags,expect", [
    (6, 0, {1: 0, 59: 6}),     # a step in the persistent launch, the rest on chip
    (40, 0, {1: 0, 59: 0}),    # too many to be faster one after another
])
def test_pieces_may_take_either(gpu, models, flags, expect):
    cs = cases(models, 60)
    solvers = [make_solver(c) for c in cs]
    b = Batch(solvers)
    for n, alone in expect.items():
        assert b.on_chip(n) == alone
        b.run(n)
    b.status()
    b.close()
    check(cs, solvers)


def test_legacy_quirks(gpu):
    cs = cases(3, 40)[:1] * 4
    solvers = [make_solver(c, flags=FLAG_LEGACY_QUIRKS) for c in cs]
    b = Batch(solvers)
    b.run(1)
    b.run(39)
    b.status()
    b.close()
    check(cs, solvers, FLAG_LEGACY_QUIRKS)


def test_a_trial_times_the_persistent_launch(gpu, tmp_path, monkeypatch):
    """A trial leaves the models that a whole run advances on chip where they are."""
    monkeypatch.setenv("SEIDART_GB300_TUNING", str(tmp_path / "tuning.json"))
    cs = cases(2, 60) + [sy.small_case(ELECTROMAG2, seed=1, nx=1040, nz=540, npml=9, nstep=60)]
    solvers = [make_solver(c, flags=FLAG_STREAMING if q < 2 else 0) for q, c in enumerate(cs)]
    b = Batch(solvers)
    assert b.on_chip(60) == 1
    b.trial(3)
    b.status()
    assert [s.status()[0] for s in solvers] == [3, 3, 0]
    autotune(b, steps=3)
    b.run(60)
    b.status()
    b.close()
    check(cs, solvers)
