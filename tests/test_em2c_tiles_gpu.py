"""GPU: electromag2c runs at the sizes where the streaming tiles change, against
the FP64 oracle: widths around one column of tiles (64 cells) and two (112),
strips deeper than a tile, pieces that are no multiple of the steps a launch
advances, grids whose tiles have one to five rows a warp, and strips that leave
a tile's coefficients no room on chip.  Tolerances as in test_complex_em_gpu.py."""
import numpy as np
import pytest

from helpers import make_solver, rel_l2, run_oracle
from seidart_gb300 import ELECTROMAG2C
from seidart_gb300 import synthetic as sy
from seidart_gb300.solver import FIELDS, FLAG_TWO_PASS, MEMORY

pytestmark = pytest.mark.gpu


def check(s, st, ref):
    assert rel_l2(s.traces(), ref) <= 1e-5
    for q, name in enumerate(FIELDS[ELECTROMAG2C]):
        assert rel_l2(s.field(name), st.fields[q]) <= 1e-5, name
    for q, name in enumerate(MEMORY[ELECTROMAG2C]):
        assert rel_l2(s.memory(name), st.memory[q], floor=1e-30) <= 1e-4, name


@pytest.mark.parametrize("nx,nz,npml,chunks", [
    (64, 40, 4, (1, 2, 3, 4, 60)),
    (65, 41, 7, (5, 6, 7, 61)),
    (112, 64, 20, (90, 77)),
    (113, 65, 6, (8, 90)),
    (90, 131, 33, (64, 99)),
    (7, 6, 1, (3, 14)),
    (230, 73, 12, (150, 3)),
    (400, 170, 10, (9, 30)),    # two rows a warp
    (601, 400, 20, (17, 20)),   # three
    (900, 440, 15, (20, 5)),    # four
    (1040, 540, 20, (9, 20)),   # five
    (1039, 539, 60, (10, 19)),  # five, coefficients read from L2 in the corners
])
def test_tile_edges(gpu, nx, nz, npml, chunks):
    case = sy.small_case(ELECTROMAG2C, seed=nx + nz, nx=nx, nz=nz, npml=npml, nstep=sum(chunks), nrec=40)
    case.rec_ijk[:4] = [(nx - 1, 0, nz // 2), (nx - 2, 0, nz - 2), (0, 0, 0), (nx // 2, 0, nz - 1)]
    if nx > 300:  # a few steps: from a corner, so that the strips see the wave
        case.src_ijk = (nx - npml - 5, 0, nz - npml - 4)
        case.rec_ijk[4:] = [(nx - npml - 30 + q, 0, nz - npml - 10 + q % 7) for q in range(36)]
    st, ref, _, blew = run_oracle(case)
    assert not blew
    with make_solver(case) as s:
        for n in chunks:
            s.run(n)
        s.status()
        check(s, st, ref)


def test_two_pass_form(gpu):
    """The two-kernel step (FLAG_TWO_PASS), which no default run takes."""
    case = sy.small_case(ELECTROMAG2C, seed=8, nx=61, nz=47, npml=6, nstep=120)
    st, ref, _, blew = run_oracle(case)
    assert not blew
    with make_solver(case, flags=FLAG_TWO_PASS) as s:
        s.run(50)
        s.run(70)
        s.status()
        check(s, st, ref)


def test_pieces_give_the_same_bits(gpu):
    """A run in pieces of any length gives the plain run's states bit for bit,
    and more receivers than a tile lists are all recorded."""
    case = sy.small_case(ELECTROMAG2C, seed=3, nx=150, nz=90, npml=8, nstep=45, nrec=400)
    case.rec_ijk = np.concatenate([case.rec_ijk[:1].repeat(300, 0), case.rec_ijk])
    case.rec_ijk[:300, 0] = np.arange(300) % 20 + 70
    case.rec_ijk[:300, 2] = np.arange(300) // 20 + 40
    out = []
    for chunks in ((45,), (1, 6, 3, 4, 31), (5,) * 9):
        with make_solver(case) as s:
            for n in chunks:
                s.run(n)
            s.status()
            out.append([s.traces()] + [s.field(f) for f in FIELDS[ELECTROMAG2C]] +
                       [s.memory(m) for m in MEMORY[ELECTROMAG2C]])
    st, ref, _, blew = run_oracle(case)
    assert not blew and rel_l2(out[0][0], ref) <= 1e-5
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
