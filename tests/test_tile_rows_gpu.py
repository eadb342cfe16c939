"""GPU: on-chip tiles of every number of rows a warp (electromag2 one to four,
seismic2 one to three) against the kernels that advance one step a launch (handles
told to stream, a step or two a run), from random fields, bit for bit: fields, memory
variables, traces, and checkpoints written from chip."""
import ctypes as C

import numpy as np
import pytest

from helpers import make_solver
from seidart_gb300 import ELECTROMAG2, SEISMIC2, _lib
from seidart_gb300 import synthetic as sy
from seidart_gb300.solver import FIELDS, FLAG_STREAMING, MEMORY

pytestmark = pytest.mark.gpu


def results(s):
    return {"traces": s.traces(), **{f: s.field(f) for f in FIELDS[s.kind]}, **{m: s.memory(m) for m in MEMORY[s.kind]}}


def checkpoints(s, nstep, every, device):
    """The state before every `every`-th step of a run of nstep steps written from chip."""
    import torch
    from seidart_gb300.adjoint import _declare
    _declare(s._L)
    n = C.c_size_t()
    assert s._L.sfd_checkpoint_bytes(s._h, C.byref(n)) == 0
    rows = torch.zeros((nstep // every, n.value), dtype=torch.uint8, device=device)
    assert s._L.sfd_run_checkpointed(s._h, nstep, C.c_void_p(rows.data_ptr()), C.c_size_t(n.value), every) == 0, \
        _lib.lib().sfd_last_error()
    return rows


@pytest.mark.parametrize("kind,nx,nz,npml", [
    (ELECTROMAG2, 120, 90, 10),     # one row a warp
    (ELECTROMAG2, 491, 434, 20),    # two
    (ELECTROMAG2, 1040, 540, 20),   # three
    (ELECTROMAG2, 900, 800, 20),    # four
    (ELECTROMAG2, 1088, 742, 1),    # four, one-cell strips
    (SEISMIC2, 120, 90, 10),        # one row a warp
    (SEISMIC2, 333, 401, 11),       # two
    (SEISMIC2, 480, 440, 20),       # three
    (SEISMIC2, 600, 450, 1),        # three, one-cell strips
])
def test_as_single_steps(gpu, kind, nx, nz, npml):
    import torch
    nstep, every = 14, 7
    case = sy.small_case(kind, seed=nx + nz, nx=nx, nz=nz, npml=npml, nstep=nstep, nrec=60)
    case.rec_ijk[:4] = [(nx - 1, 0, nz // 2), (nx - 2, 0, nz - 2), (0, 0, 0), (nx // 2, 0, nz - 1)]
    rng = np.random.default_rng(nx)
    scale = {"E": 1.0, "H": 1.0 / 377.0, "v": 1.0, "s": 3e6}
    F = {f: (scale[f[0]] * rng.standard_normal((nz, nx))).astype(np.float32) for f in FIELDS[kind]}
    out = []
    for flags, pieces in ((0, (nstep,)), (FLAG_STREAMING, (2, 2, 2, 1) * 2)):
        with make_solver(case, flags=flags) as s:
            assert (s.on_chip() is None) == bool(flags)
            for f in F:
                s.set_field(f, F[f])
            for n in pieces:
                s.run(n)
            s.status()
            out.append(results(s))
    for name in out[0]:
        assert np.array_equal(out[0][name], out[1][name]), name
    if kind == ELECTROMAG2:
        with make_solver(case) as s, make_solver(case) as t:
            for q in (s, t):
                for f in F:
                    q.set_field(f, F[f])
            rows = checkpoints(s, nstep, every, gpu)
            s.status()
            for name, v in results(s).items():
                assert np.array_equal(v, out[0][name]), name
            one = torch.zeros_like(rows[0])
            for r in rows:
                assert t._L.sfd_checkpoint_save(t._h, C.c_void_p(one.data_ptr())) == 0
                t.run(every)
                t.status()
                assert torch.equal(one, r)
