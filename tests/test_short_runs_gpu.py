"""GPU: streaming runs take launches of several steps, single steps or both by their
length and the grid (csrc/sfd_api.cu): from random fields, runs of any lengths give the
same bits, and leave the state in the copy that one launch a step would."""
import numpy as np
import pytest

from helpers import make_solver
from seidart_gb300 import ELECTROMAG2, ELECTROMAG2C, SEISMIC2
from seidart_gb300 import synthetic as sy
from seidart_gb300.solver import FIELDS, FLAG_STREAMING, MEMORY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nx,nz,pieces", [
    (ELECTROMAG2, 300, 200, ((24,), (1,) * 24, (2, 3, 4, 5, 6, 4), (7, 8, 9), (11, 13))),
    (SEISMIC2, 150, 120, ((24,), (1,) * 24, (2, 3, 4, 5, 6, 4), (7, 8, 9), (11, 13))),
    (SEISMIC2, 700, 690, ((42,), (3,) * 14, (4, 33, 5))),   # two waves of tiles, worth it
    (SEISMIC2, 723, 549, ((42,), (3,) * 14, (4, 33, 5))),   # two waves, not worth it: single steps, by graph
    (ELECTROMAG2C, 150, 90, ((24,), (1,) * 24, (2, 3, 4, 5, 6, 4), (7, 8, 9))),
    (ELECTROMAG2C, 1000, 900, ((12,), (1, 2, 3, 2, 2, 2), (5, 7))),  # two steps in the step's two kernels
])
def test_any_lengths_give_the_same_bits(gpu, kind, nx, nz, pieces):
    n = sum(pieces[0])
    case = sy.small_case(kind, seed=nx, nx=nx, nz=nz, npml=12, nstep=n, nrec=30)
    rng = np.random.default_rng(nx)
    scale = {"E": 1.0, "H": 1.0 / 377.0, "v": 1.0, "s": 3e6}
    F = {f: (scale[f[0]] * rng.standard_normal((nz, nx))).astype(np.float32) for f in FIELDS[kind]}
    out = []
    for chunks in pieces:
        assert sum(chunks) == n
        with make_solver(case, flags=0 if kind == ELECTROMAG2C else FLAG_STREAMING) as s:
            assert s.on_chip() is None
            for f in F:
                s.set_field(f, F[f])
            start = s.field_tensor(FIELDS[kind][0]).data_ptr()
            for q, c in enumerate(chunks):
                s.run(c)
                same = s.field_tensor(FIELDS[kind][0]).data_ptr() == start
                assert same == (kind == ELECTROMAG2C or sum(chunks[:q + 1]) % 2 == 0)
            s.status()
            out.append({"traces": s.traces(), **{f: s.field(f) for f in F}, **{m: s.memory(m) for m in MEMORY[kind]}})
    for other in out[1:]:
        for name in out[0]:
            assert np.array_equal(out[0][name], other[name]), name


@pytest.mark.parametrize("nx,nz,npml", [
    (64, 48, 4), (65, 49, 7), (112, 80, 20), (113, 81, 6), (130, 131, 40), (12, 10, 2), (229, 73, 12),
])
@pytest.mark.parametrize("atten", [False, True])
def test_seismic2_tiles_as_single_steps(gpu, nx, nz, npml, atten):
    """Fewer steps than a graph of single steps holds take tiles on any grid: at the
    sizes where the tiles change (csrc/s2_stream.cu), two rows a warp among them, they
    give the single steps' bits."""
    case = sy.small_case(SEISMIC2, seed=nx + nz, nx=nx, nz=nz, npml=npml, nstep=30, nrec=30, atten=atten)
    case.rec_ijk[:4] = [(nx - 1, 0, nz // 2), (nx - 2, 0, nz - 2), (0, 0, 0), (nx // 2, 0, nz - 1)]
    rng = np.random.default_rng(nx)
    F = {f: ((1.0 if f[0] == "v" else 3e6) * rng.standard_normal((nz, nx))).astype(np.float32) for f in FIELDS[SEISMIC2]}
    out = []
    for chunks in ((30,), (4, 7, 19), (3,) * 10):
        with make_solver(case, flags=FLAG_STREAMING) as s:
            for f in F:
                s.set_field(f, F[f])
            for c in chunks:
                s.run(c)
            s.status()
            out.append({"traces": s.traces(), **{f: s.field(f) for f in F}, **{m: s.memory(m) for m in MEMORY[SEISMIC2]}})
    for other in out[:-1]:
        for name in other:
            assert np.array_equal(out[-1][name], other[name]), name


@pytest.mark.parametrize("kind,nx,nz,flags,nstep", [
    (ELECTROMAG2, 300, 200, FLAG_STREAMING, 13),
    (SEISMIC2, 723, 549, 0, 40),   # single steps, by graph outside a capture
    (SEISMIC2, 723, 549, 0, 7),
    (ELECTROMAG2C, 150, 90, 0, 7),
    (ELECTROMAG2C, 150, 90, 0, 1),
])
def test_runs_can_be_captured(gpu, kind, nx, nz, flags, nstep):
    import torch
    case = sy.small_case(kind, seed=nx, nx=nx, nz=nz, npml=12, nstep=nstep, nrec=30)
    rng = np.random.default_rng(nx)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream), make_solver(case, flags=flags) as s, make_solver(case, flags=flags) as t:
        for f in FIELDS[kind]:
            v = rng.standard_normal((nz, nx)).astype(np.float32)
            s.set_field(f, v)
            t.set_field(f, v)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            s.run(nstep)
        graph.replay()
        t.run(nstep)
        t.status()
        s.status()
        assert np.abs(t.traces()).max() > 0.1 and np.array_equal(s.traces(), t.traces())
        for f in FIELDS[kind]:
            assert np.array_equal(s.field(f), t.field(f)), f
