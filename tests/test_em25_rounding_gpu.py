"""GPU: electromag25 steps round as their source says, in every cell: two steps
from random fields give, bit for bit, what NumPy gives with the same roundings in
FP32.  The grids take blocks of 4, 8 and 16 rows: a cell's bits depend neither on
the block's rows nor on whether its block holds strip cells."""
import numpy as np
import pytest

from f32 import ahead, behind, f32, fma, strip, tables
from helpers import make_solver
from seidart_gb300 import ELECTROMAG25
from seidart_gb300 import synthetic as sy
from seidart_gb300.solver import FIELDS, MEMORY

pytestmark = pytest.mark.gpu
EPS0, MU0 = 8.85418782e-12, 4.0e-7 * np.pi
Z, Y, X = 0, 1, 2  # axes of a field


def step(case, F, M):
    """One step of the fields F and memory variables M (dicts), no source."""
    g, W, dt = case.grid, case.grid.npml, case.grid.dt
    NX, NY, NZ = g.nx, g.ny, g.nz
    k, j, i = np.ogrid[:NZ, :NY, :NX]
    shape = {X: (1, 1, NX), Y: (1, NY, 1), Z: (NZ, 1, 1)}
    T = {a: [t.reshape(shape[a]) for t in tables(p, d)] for a, p, d in zip((X, Y, Z), case.profiles, (g.dx, g.dy, g.dz))}
    S = {a: strip(n, W).reshape(shape[a]) for a, n in ((X, NX), (Y, NY), (Z, NZ))}
    i0, k0 = i // 32 * 32, k // 4 * 4  # the groups of 32 x 4 columns off strips and faces
    plain = ((i0 >= max(W, 1)) & (i0 + 31 <= min(NX - W - 1, NX - 3)) & (k0 >= max(W, 1)) &
             (k0 + 3 <= min(NZ - W - 1, NZ - 3)))
    F, M = {n: v.copy() for n, v in F.items()}, {n: v.copy() for n, v in M.items()}

    def derivative(name, d, axis, half, act):
        """The scaled derivative with its memory variable, and whether it may be fused (it has none)."""
        ik, ad, b = T[axis][3 * half:3 * half + 3]
        m = fma(ad, d, b * M[name])
        at = S[axis] & act
        M[name] = np.where(at, m, M[name])
        return np.where(at, d * ik + m, d * ik)

    loop = (i <= NX - 2) & (j <= NY - 2) & (k <= NZ - 2)
    hface = {"Hx": (i == 0) | (k == 0) | (k == NZ - 2) | (j == 0) | (j == NY - 2),
             "Hy": (i == 0) | (i == NX - 2) | (k == 0) | (k == NZ - 2) | (j == 0),
             "Hz": (i == 0) | (i == NX - 2) | (k == 0) | (j == 0) | (j == NY - 2)}
    Ex, Ey, Ez = F["Ex"], F["Ey"], F["Ez"]
    # each curl: the derivative that leads (rounded), the other (fused where plain) with its raw difference
    curls = {"Hx": (("dEz_dy", Ez - ahead(Ez, Y), Y, 1), ("dEy_dz", ahead(Ey, Z) - Ey, Z, 1)),
             "Hy": (("dEz_dx", ahead(Ez, X) - Ez, X, 0), ("dEx_dz", Ex - ahead(Ex, Z), Z, 0)),
             "Hz": (("dEx_dy", ahead(Ex, Y) - Ex, Y, 0), ("dEy_dx", Ey - ahead(Ey, X), X, 0))}

    def curl(lead, other, act):
        v, w = derivative(*lead, act), derivative(*other, act)
        ik = T[other[2]][3 * other[3]]
        return np.where(plain, fma(other[1], ik, v), v + w)

    for n, (lead, other) in curls.items():
        act = loop & (k >= 1) if n == "Hz" else loop
        old = np.where(hface[n], f32(0), F[n])
        F[n] = np.where(act, fma(f32(dt / MU0), curl(lead, other, act), old), F[n])
    e11, e12, e13, e22, e23, e33, s11, s12, s13, s22, s23, s33 = case.planes
    c = []
    for e, s in ((e11 + e12 + e13, s11 + s12 + s13), (e12 + e22 + e23, s12 + s22 + s23), (e13 + e23 + e33, s13 + s23 + s33)):
        q = s * dt / (2.0 * (e * EPS0))
        c += [((1.0 - q) / (1.0 + q)).astype(f32), ((dt / (e * EPS0)) / (1.0 + q)).astype(f32)]
    six = lambda a, dz: (f32(4) * a + np.roll(a, 1, 1) + np.roll(a, dz, 0)) / f32(6)  # noqa: E731
    c = [a[:, None, :] for a in (c[0], c[1], six(c[2], 1), six(c[3], 1), six(c[4], -1), six(c[5], -1))]
    Hx, Hy, Hz = F["Hx"], F["Hy"], F["Hz"]
    curls = {"Ex": (("dHz_dy", Hz - behind(Hz, Y), Y, 1), ("dHy_dz", behind(Hy, Z) - Hy, Z, 0)),
             "Ey": (("dHx_dz", Hx - behind(Hx, Z), Z, 1), ("dHz_dx", behind(Hz, X) - Hz, X, 1)),
             "Ez": (("dHx_dy", behind(Hx, Y) - Hx, Y, 1), ("dHy_dx", Hy - behind(Hy, X), X, 1))}
    inner = {a: (x >= 1) & (x <= n - 2) for a, x, n in ((X, i, NX), (Y, j, NY), (Z, k, NZ))}
    acts = {"Ex": inner[Z] & inner[Y] & (i <= NX - 2), "Ey": inner[Z] & inner[X] & (j <= NY - 2),
            "Ez": inner[X] & inner[Y] & (k <= NZ - 2)}
    last = {"Ex": (2, 1, 1), "Ey": (1, 2, 1), "Ez": (1, 1, 2)}
    for q, (n, (lead, other)) in enumerate(curls.items()):
        new = fma(c[2 * q], F[n], c[2 * q + 1] * curl(lead, other, acts[n]))
        a, b, d = last[n]
        face = (i == 0) | (i == NX - a) | (j == 0) | (j == NY - b) | (k == 0) | (k == NZ - d)
        F[n] = np.where(face, f32(0), np.where(acts[n], new, F[n]))
    end = {"Hx": (1, 2, 2), "Hy": (2, 1, 2), "Hz": (2, 2, 1)}  # the stored H keeps its faces at zero
    for n, (a, b, d) in end.items():
        face = (i == 0) | (i == NX - a) | (j == 0) | (j == NY - b) | (k == 0) | (k == NZ - d)
        F[n] = np.where(face, f32(0), F[n])
    return F, M


@pytest.mark.parametrize("nx,ny,nz,npml", [
    (61, 15, 50, 5),     # blocks of 4 rows
    (130, 16, 131, 6),   # of 8
    (200, 16, 201, 7),   # of 16
])
def test_steps_round_as_written(gpu, nx, ny, nz, npml):
    case = sy.small_case(ELECTROMAG25, seed=nx, nx=nx, ny=ny, nz=nz, npml=npml, nstep=2, nrec=1)
    case.srcfn[:] = 0.0
    rng = np.random.default_rng(nx)
    scale = {"E": 1.0, "H": 1.0 / 377.0}
    F = {n: (scale[n[0]] * rng.standard_normal((nz, ny, nx))).astype(f32) for n in FIELDS[ELECTROMAG25]}
    M = {n: np.zeros((nz, ny, nx), f32) for n in MEMORY[ELECTROMAG25]}
    with make_solver(case) as s:
        for n in F:
            s.set_field(n, F[n])
        for t in range(2):
            F, M = step(case, F, M)
            s.run(1)
            s.status()
            for n in F:
                assert np.array_equal(s.field(n), F[n]), (t, n, int((s.field(n) != F[n]).sum()))
            for n in M:
                assert np.array_equal(s.memory(n), M[n]), (t, n)
