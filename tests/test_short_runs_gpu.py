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
