"""GPU: the on-chip electromag2 tiles at the sizes where their edges move,
against the FP64 oracle: one tile column and two (128, 129 columns), widths
that are no multiple of four, rows a warp from one to four, strips wider than a
tile, and runs that end on, before and after a hand-over between tiles (every
four steps), split into pieces.  Tolerances as in test_parity_gpu.py."""
import numpy as np
import pytest

from helpers import make_solver, rel_l2, run_oracle
from seidart_gb300 import ELECTROMAG2
from seidart_gb300 import synthetic as sy
from seidart_gb300.solver import FIELDS, MEMORY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,npml,chunks", [
    (128, 30, 4, (1, 2, 1, 40)),      # one column of tiles, exactly as wide as a warp's rows
    (129, 75, 7, (3, 4, 5, 37)),      # two columns, the last cell alone in its lane
    (131, 47, 20, (4, 4, 8, 30)),     # strips wider than the bands of rows
    (249, 200, 9, (9, 50)),           # two columns whose halos reach the strips
    (253, 61, 1, (60,)),              # three columns, one-cell strips
    (46, 700, 6, (7, 41)),            # many bands of a narrow grid
    (900, 40, 5, (6, 50)),            # many columns of a flat one
    (131, 47, 20, (61, 79, 80)),      # long enough for the waves to cross every strip
    (150, 96, 8, (101, 99)),
    (90, 260, 13, (111, 109)),
])
def test_tile_edges(gpu, nx, nz, npml, chunks):
    case = sy.small_case(ELECTROMAG2, seed=nx + nz, nx=nx, nz=nz, npml=npml, nstep=sum(chunks), nrec=40)
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
        for q, name in enumerate(FIELDS[ELECTROMAG2]):
            assert rel_l2(s.field(name), st.fields[q]) <= 1e-5, name
        for q, name in enumerate(MEMORY[ELECTROMAG2]):
            if np.abs(st.memory[q]).max() > 1e-37:  # below, FP32 has no normal number
                assert rel_l2(s.memory(name), st.memory[q]) <= 1e-4, name


def test_pieces_give_the_same_bits(gpu):
    """A run in pieces of any length gives the plain run's states bit for bit,
    whichever tile computed a halo cell."""
    case = sy.electromag2_layers(nstep=45)
    out = []
    for chunks in ((45,), (1, 6, 3, 4, 31), (5,) * 9):
        with make_solver(case) as s:
            for n in chunks:
                s.run(n)
            s.status()
            out.append([s.traces()] + [s.field(f) for f in FIELDS[ELECTROMAG2]] + [s.memory(m) for m in MEMORY[ELECTROMAG2]])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
