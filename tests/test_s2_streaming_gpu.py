"""GPU: streaming seismic2 runs (FLAG_STREAMING, corrected physics) at the sizes
where their tiles change, against the FP64 oracle: widths around one column of
tiles (64 cells) and two (112), depths around one band (48 rows) and around its
cuts (40 owned rows), strips so wide that frames have two rows a warp, and pieces
that are no multiple of the steps a launch advances.  Tolerances as in
test_parity_gpu.py."""
import numpy as np
import pytest

from helpers import make_solver, rel_l2, run_oracle
from seidart_gb300 import SEISMIC2
from seidart_gb300 import synthetic as sy
from seidart_gb300.solver import FIELDS, FLAG_STREAMING, MEMORY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,npml,chunks", [
    (64, 48, 4, (1, 2, 3, 4, 60)),
    (65, 49, 7, (5, 6, 7, 61)),
    (112, 80, 20, (60, 47)),
    (113, 81, 6, (8, 90)),
    (130, 131, 40, (64, 59)),
    (12, 10, 2, (3, 14)),
    (229, 73, 12, (100, 3)),
])
@pytest.mark.parametrize("atten", [False, True])
def test_tile_edges(gpu, nx, nz, npml, chunks, atten):
    case = sy.small_case(SEISMIC2, seed=nx + nz, nx=nx, nz=nz, npml=npml, nstep=sum(chunks), nrec=40, atten=atten)
    case.rec_ijk[:4] = [(nx - 1, 0, nz // 2), (nx - 2, 0, nz - 2), (0, 0, 0), (nx // 2, 0, nz - 1)]
    st, ref, _, blew = run_oracle(case)
    assert not blew
    with make_solver(case, flags=FLAG_STREAMING) as s:
        assert s.on_chip() is None
        for n in chunks:
            s.run(n)
        s.status()
        assert rel_l2(s.traces(), ref) <= 1e-5
        for q, name in enumerate(FIELDS[SEISMIC2]):
            assert rel_l2(s.field(name), st.fields[q]) <= 1e-5, name
        for q, name in enumerate(MEMORY[SEISMIC2]):
            if np.abs(st.memory[q]).max() > 1e-37:  # below, FP32 has no normal number
                assert rel_l2(s.memory(name), st.memory[q]) <= 1e-4, name


def test_streams_as_on_chip(gpu):
    """Bit for bit the on-chip run's states, in pieces of any length."""
    case = sy.small_case(SEISMIC2, seed=2, nx=150, nz=120, npml=10, nstep=45, nrec=300)
    out = []
    for flags, chunks in ((0, (45,)), (FLAG_STREAMING, (45,)), (FLAG_STREAMING, (1, 6, 3, 4, 31))):
        with make_solver(case, flags=flags) as s:
            assert (s.on_chip() is None) == bool(flags)
            for n in chunks:
                s.run(n)
            s.status()
            out.append([s.traces()] + [s.field(f) for f in FIELDS[SEISMIC2]] + [s.memory(m) for m in MEMORY[SEISMIC2]])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
