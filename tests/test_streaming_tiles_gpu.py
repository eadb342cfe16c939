"""GPU: streaming runs (FLAG_STREAMING) at the sizes where their tiles change,
against the FP64 oracle: widths around one column of tiles (128 cells) and two
(240), depths around one band (32 rows) and around its cuts (24 owned rows),
strips deeper than a tile, and pieces that are no multiple of the steps a
launch advances.  Tolerances as in test_parity_gpu.py."""
import numpy as np
import pytest

from helpers import make_solver, rel_l2, run_oracle
from seidart_gb300 import ELECTROMAG2
from seidart_gb300 import synthetic as sy
from seidart_gb300.solver import FIELDS, FLAG_STREAMING, MEMORY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nx,nz,npml,chunks", [
    (ELECTROMAG2, 128, 32, 4, (1, 2, 3, 4, 60)),
    (ELECTROMAG2, 129, 33, 7, (5, 6, 7, 61)),
    (ELECTROMAG2, 121, 56, 20, (90, 77)),
    (ELECTROMAG2, 240, 48, 6, (8, 90)),
    (ELECTROMAG2, 241, 49, 1, (99, 1)),
    (ELECTROMAG2, 90, 131, 33, (64, 99)),
    (ELECTROMAG2, 7, 6, 1, (3, 14)),
    (ELECTROMAG2, 395, 73, 12, (150, 3)),
])
def test_tile_edges(gpu, kind, nx, nz, npml, chunks):
    case = sy.small_case(kind, seed=nx + nz, nx=nx, nz=nz, npml=npml, nstep=sum(chunks), nrec=40)
    case.rec_ijk[:4] = [(nx - 1, 0, nz // 2), (nx - 2, 0, nz - 2), (0, 0, 0), (nx // 2, 0, nz - 1)]
    with make_solver(case, flags=FLAG_STREAMING) as s:
        assert s.on_chip() is None
        for n in chunks:
            s.run(n)
        s.status()
        st, ref, _, blew = run_oracle(case)
        assert not blew
        assert rel_l2(s.traces(), ref) <= 1e-5
        for q, name in enumerate(FIELDS[kind]):
            assert rel_l2(s.field(name), st.fields[q]) <= 1e-5, name
        for q, name in enumerate(MEMORY[kind]):
            if np.abs(st.memory[q]).max() > 1e-37:  # below, FP32 has no normal number
                assert rel_l2(s.memory(name), st.memory[q]) <= 1e-4, name


def test_pieces_give_the_same_bits(gpu):
    """A streaming run in pieces of any length gives the plain run's states bit
    for bit, wherever a launch's steps begin."""
    case = sy.electromag2_layers(nstep=45)
    out = []
    for chunks in ((45,), (1, 6, 3, 4, 31), (5,) * 9):
        with make_solver(case, flags=FLAG_STREAMING) as s:
            for n in chunks:
                s.run(n)
            s.status()
            out.append([s.traces()] + [s.field(f) for f in FIELDS[ELECTROMAG2]] + [s.memory(m) for m in MEMORY[ELECTROMAG2]])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
