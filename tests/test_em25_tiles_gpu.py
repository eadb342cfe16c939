"""GPU: electromag25 at the sizes where its blocks change, against the FP64
oracle: blocks of 4, 8 and 16 rows, widths and depths around their edges (32
columns, four a thread), strips one cell and a third of the grid wide, a
thread with cells of both x strips, one plane a segment.  Tolerances as in
test_parity_gpu.py."""
import numpy as np
import pytest

from helpers import make_solver, rel_l2, run_oracle
from seidart_gb300 import ELECTROMAG25
from seidart_gb300 import synthetic as sy
from seidart_gb300.solver import FIELDS, MEMORY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,npml,nstep", [
    (12, 12, 12, 5, 40),     # columns 4 and 7 of a thread in different x strips
    (8, 8, 8, 1, 12),
    (33, 14, 17, 3, 60),
    (31, 24, 33, 8, 60),
    (64, 13, 65, 1, 60),
    (130, 14, 130, 5, 50),   # blocks of 8 rows
    (200, 14, 201, 6, 50),   # of 16
    (97, 40, 95, 9, 40),
])
def test_block_edges(gpu, nx, ny, nz, npml, nstep):
    case = sy.small_case(ELECTROMAG25, seed=nx + nz, nx=nx, ny=ny, nz=nz, npml=npml, nstep=nstep, nrec=20)
    case.rec_ijk[:3] = [(nx - 1, ny // 2, nz // 2), (0, 0, 0), (nx // 2, ny - 1, nz - 1)]
    st, ref, _, blew = run_oracle(case)
    assert not blew
    with make_solver(case) as s:
        s.run(nstep // 3)
        s.run(nstep - nstep // 3)
        s.status()
        assert rel_l2(s.traces(), ref) <= 1e-5
        for q, name in enumerate(FIELDS[ELECTROMAG25]):
            assert rel_l2(s.field(name), st.fields[q]) <= 1e-5, name
        for q, name in enumerate(MEMORY[ELECTROMAG25]):
            if np.abs(st.memory[q]).max() > 1e-37:  # below, FP32 has no normal number
                assert rel_l2(s.memory(name), st.memory[q]) <= 1e-4, name
