"""GPU: electromag2 steps round as their source says, in every cell and form: on
chip, streamed, one step a launch (runs of one step) and batched in the persistent
launch, steps from random fields give, bit for bit, what NumPy gives with the same
roundings in FP32."""
import numpy as np
import pytest

from f32 import ahead, behind, f32, fma, strip, tables
from helpers import make_solver
from seidart_gb300 import ELECTROMAG2
from seidart_gb300 import synthetic as sy
from seidart_gb300.batch import Batch
from seidart_gb300.solver import FIELDS, FLAG_STREAMING, MEMORY

pytestmark = pytest.mark.gpu
EPS0, MU0 = 8.85418782e-12, 4.0e-7 * np.pi


def coefficients(case):
    dt = case.grid.dt
    e11, e13, e33, s11, s13, s33 = case.planes
    out = []
    for (e, s), axis in (((e11 + e13, s11 + s13), 0), ((e13 + e33, s13 + s33), 1)):
        e = e * EPS0
        q = s * dt / (2.0 * e)
        for c in ((1.0 - q) / (1.0 + q), (dt / e) / (1.0 + q)):
            out.append(((c + behind(c, axis)) / 2).astype(f32))
    return out


def step(case, F, M, c):
    """One step of the fields F and memory variables M (dicts), no source."""
    g, W = case.grid, case.grid.npml
    NX, NZ = g.nx, g.nz
    k, i = np.ogrid[:NZ, :NX]
    ikx, adx, bx, ikxh, adxh, bxh = (t[None, :] for t in tables(case.profiles[0], g.dx))
    ikz, adz, bz, ikzh, adzh, bzh = (t[:, None] for t in tables(case.profiles[1], g.dz))
    xs, zs = strip(NX, W)[None, :], strip(NZ, W)[:, None]
    Ex, Ez, Hy = (F[n] for n in FIELDS[ELECTROMAG2])
    M = dict(M)

    def derivative(name, d, ik, ad, b, at):
        m = fma(b, M[name], ad * d) if name.endswith("dx") else fma(ad, d, b * M[name])
        M[name] = np.where(at, m, M[name])
        return np.where(at, d * ik + m, d * ik)

    loop = (i <= NX - 2) & (k <= NZ - 2)
    dEx, dEz = ahead(Ex, 0) - Ex, ahead(Ez, 1) - Ez
    vz = derivative("dEx_dz", dEx, ikz, adz, bz, zs & loop)
    vx = derivative("dEz_dx", dEz, ikx, adx, bx, xs & loop)
    i0, lo, hi = i // 4 * 4, max(W, 1), max(W, 2)
    rounded = (i0 < lo) | (i0 + 3 >= NX - hi) | (k < lo) | (k >= NZ - hi)
    h = fma(f32(g.dt / MU0), np.where(rounded, vx + vz, fma(dEz, ikx, vz)), Hy)
    Hy = np.where(loop, h, Hy)
    px, pz = loop & (k >= 1), loop & (i >= 1)
    dx = derivative("dHy_dz", Hy - behind(Hy, 0), ikzh, adzh, bzh, zs & px)
    dz = derivative("dHy_dx", Hy - behind(Hy, 1), ikxh, adxh, bxh, xs & pz)
    Ex = np.where(px, fma(c[0], Ex, c[1] * dx), Ex)
    Ez = np.where(pz, fma(c[2], Ez, c[3] * dz), Ez)
    zero = f32(0)
    Ex = np.where((i == 0) | (i == NX - 2) | (k == 0) | (k == NZ - 1), zero, Ex)
    Ez = np.where((i == 0) | (i == NX - 1) | (k == 0) | (k == NZ - 2), zero, Ez)
    Hy = np.where(loop & ((i == 0) | (i == NX - 2) | (k == 0) | (k == NZ - 2)), zero, Hy)
    return dict(zip(FIELDS[ELECTROMAG2], (Ex, Ez, Hy))), M


@pytest.mark.parametrize("form", ["on chip", "streaming", "batch 1", "batch 2", "batch 4"])
@pytest.mark.parametrize("nx,nz,npml", [
    (61, 50, 5),
    (301, 99, 9),    # tiles of 128 x 8 to 128 x 32 inside the strips, strips that end within four columns
    (262, 140, 1),   # planes off the strips
])
def test_steps_round_as_written(gpu, nx, nz, npml, form):
    chunks = (1, 5, 2)
    case = sy.small_case(ELECTROMAG2, seed=nx, nx=nx, nz=nz, npml=npml, nstep=sum(chunks), nrec=1)
    case.srcfn[:] = 0.0
    rng = np.random.default_rng(nx)
    F = {n: ((1.0 if n[0] == "E" else 1.0 / 377.0) * rng.standard_normal((nz, nx))).astype(f32)
         for n in FIELDS[ELECTROMAG2]}
    M = {n: np.zeros((nz, nx), f32) for n in MEMORY[ELECTROMAG2]}
    c = coefficients(case)
    s = make_solver(case, flags=0 if form == "on chip" else FLAG_STREAMING)
    b = Batch([s]) if form.startswith("batch") else None
    if b:
        b.set_tiling(int(form[-1]), 2)
    for n in F:
        s.set_field(n, F[n])
    for chunk in chunks:
        (b or s).run(chunk)
        (b or s).status()
        for _ in range(chunk):
            F, M = step(case, F, M, c)
        for n in F:
            assert np.array_equal(s.field(n), F[n]), (chunk, n, int((s.field(n) != F[n]).sum()))
        for n in M:
            assert np.array_equal(s.memory(n), M[n]), (chunk, n)
    if b:
        b.close()
    s.close()
