"""GPU: the on-chip seismic2 tiles at the sizes where their edges move, against
the FP64 oracle: one tile column and two (64, 65 columns), odd widths, rows a
warp from one to three, strips wider than a tile, attenuation, stress sources,
and runs that end on, before and after a hand-over between tiles (every two
steps), split into pieces.  Tolerances as in test_parity_gpu.py."""
import numpy as np
import pytest

from golden.make_golden import stress_source
from helpers import make_solver, rel_l2, run_oracle
from seidart_gb300 import SEISMIC2
from seidart_gb300 import synthetic as sy
from seidart_gb300.solver import FIELDS, MEMORY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,npml,chunks,atten,stress", [
    (64, 30, 4, (1, 2, 1, 60), True, False),      # one column of tiles, exactly as wide as a warp's rows
    (65, 75, 7, (3, 4, 5, 90), False, True),      # two columns, the last cell alone in its lane
    (67, 47, 15, (2, 2, 8, 100), True, True),     # strips wider than the bands of rows
    (121, 200, 9, (9, 150), True, False),         # two columns whose halos reach the strips
    (125, 61, 1, (120,), False, False),           # three columns, one-cell strips
    (30, 700, 6, (7, 131), True, True),           # many bands of a narrow grid
    (900, 40, 5, (6, 100), True, False),          # many columns of a flat one
    (333, 401, 11, (4, 3, 120), True, True),      # three rows a warp
])
def test_tile_edges(gpu, nx, nz, npml, chunks, atten, stress):
    case = sy.small_case(SEISMIC2, seed=nx + nz, nx=nx, nz=nz, npml=npml, nstep=sum(chunks), nrec=40, atten=atten)
    if stress:
        case.stress_srcfn = stress_source(SEISMIC2, 1e6 * case.srcfn[0])
    # receivers on the last planes too
    case.rec_ijk[:4] = [(nx - 1, 0, nz // 2), (nx - 2, 0, nz - 2), (0, 0, 0), (nx // 2, 0, nz - 1)]
    with make_solver(case) as s:
        assert s.on_chip() is not None
        for n in chunks:
            s.run(n)
        s.status()
        st, ref, _, blew = run_oracle(case)
        assert not blew
        assert rel_l2(s.traces(), ref) <= 1e-5
        for q, name in enumerate(FIELDS[SEISMIC2]):
            assert rel_l2(s.field(name), st.fields[q]) <= 1e-5, name
        for q, name in enumerate(MEMORY[SEISMIC2]):
            # below, FP32 has no normal number at the fields' scale
            if np.abs(st.memory[q]).max() > 1e-37:
                assert rel_l2(s.memory(name), st.memory[q]) <= 1e-4, name


def test_pieces_give_the_same_bits(gpu):
    """A run in pieces of any length gives the plain run's states bit for bit,
    whichever tile computed a halo cell."""
    case = sy.seismic2_firn_ice(nstep=45)
    out = []
    for chunks in ((45,), (1, 6, 3, 4, 31), (5,) * 9, (2, 1) * 15):
        with make_solver(case) as s:
            for n in chunks:
                s.run(n)
            s.status()
            out.append([s.traces()] + [s.field(f) for f in FIELDS[SEISMIC2]] + [s.memory(m) for m in MEMORY[SEISMIC2]])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
