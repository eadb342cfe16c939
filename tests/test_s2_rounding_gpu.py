"""GPU: seismic2 steps (corrected physics) round as their source says, in every cell
and form: on chip, streamed, one step a launch (runs of one step) and batched in the
persistent launch, steps from random fields give, bit for bit, what NumPy gives with
the same roundings in FP32."""
import dataclasses

import numpy as np
import pytest

from f32 import ahead, behind, f32, fma, strip, tables
from helpers import make_solver
from seidart_gb300 import SEISMIC2
from seidart_gb300 import synthetic as sy
from seidart_gb300.batch import Batch
from seidart_gb300.solver import FIELDS, FLAG_STREAMING, MEMORY

pytestmark = pytest.mark.gpu
Z, X = 0, 1  # axes of a field


def coefficients(case):
    dt = case.grid.dt
    c11, c13, c15, c33, c35, c55, rho, gx, gz = case.planes
    k, i = np.ogrid[:rho.shape[0], :rho.shape[1]]
    nz, nx = rho.shape
    A = [np.where((k >= 1) & (i <= nx - 2), (ahead(c, X) + 2 * c + behind(c, Z)) / 4 * dt, 0).astype(f32)
         for c in (c11, c13, c15, c33, c35)]
    B = [np.where((k <= nz - 2) & (i >= 1), (ahead(c, Z) + 2 * c + behind(c, X)) / 4 * dt, 0).astype(f32)
         for c in (c15, c35, c55)]
    rx = dt / ((2 * rho + behind(rho, X) + behind(rho, Z)) / 4)
    rz = dt / ((2 * rho + ahead(rho, X) + ahead(rho, Z)) / 4)
    return A, B, rx.astype(f32), rz.astype(f32), (1.0 - gx).astype(f32), (1.0 - gz).astype(f32)


def step(case, F, M, c):
    """One step of the fields F and memory variables M (dicts), no source."""
    g, W = case.grid, case.grid.npml
    NX, NZ = g.nx, g.nz
    k, i = np.ogrid[:NZ, :NX]
    T = {X: [t[None, :] for t in tables(case.profiles[0], g.dx)], Z: [t[:, None] for t in tables(case.profiles[1], g.dz)]}
    S = {X: strip(NX, W)[None, :], Z: strip(NZ, W)[:, None]}
    A, B, rx, rz, gx, gz = c
    vx, vz, sxx, szz, sxz = (F[n] for n in FIELDS[SEISMIC2])
    M = dict(M)

    def memory(name, d, axis, half, loop):
        """The memory variable's next value, zero off the strip, and 1/K."""
        ik, ad, b = T[axis][3 * half:3 * half + 3]
        at = S[axis] & loop
        M[name] = np.where(at, fma(b, M[name], ad * d), M[name])
        return np.where(at, M[name], f32(0)), ik

    def gradient(name, d, axis, half, loop):
        m, ik = memory(name, d, axis, half, loop)
        return fma(d, ik, m)

    def rounded(name, d, axis, half, loop):
        m, ik = memory(name, d, axis, half, loop)
        return d * ik + m

    def stress(s, a, dx, b, dz, c, shear, loop):
        return np.where(loop, s + fma(c, shear, fma(a, dx, b * dz)), s)

    l1, l2 = (k >= 1) & (i <= NX - 2), (k <= NZ - 2) & (i >= 1)
    dx = gradient("dvx_dx", ahead(vx, X) - vx, X, 1, l1)
    dz = gradient("dvz_dz", vz - behind(vz, Z), Z, 0, l1)
    shear = gradient("dvz_dx", ahead(vz, X) - vz, X, 0, l1) + gradient("dvx_dz", vx - behind(vx, Z), Z, 1, l1)
    sxx = stress(sxx, A[0], dx, A[1], dz, A[2], shear, l1)
    szz = stress(szz, A[1], dx, A[3], dz, A[4], shear, l1)
    dx = gradient("dvx_dx_sxz", vx - behind(vx, X), X, 1, l2)
    dz = gradient("dvz_dz_sxz", ahead(vz, Z) - vz, Z, 0, l2)
    shear = gradient("dvz_dx_sxz", vz - behind(vz, X), X, 0, l2) + gradient("dvx_dz_sxz", ahead(vx, Z) - vx, Z, 1, l2)
    sxz = stress(sxz, B[0], dx, B[1], dz, B[2], shear, l2)
    lx, lz = (k >= 1) & (i >= 1), (k <= NZ - 2) & (i <= NX - 2)
    ax = rounded("dsigmaxx_dx", sxx - behind(sxx, X), X, 0, lx) + rounded("dsigmaxz_dz", sxz - behind(sxz, Z), Z, 0, lx)
    az = rounded("dsigmaxz_dx", ahead(sxz, X) - sxz, X, 1, lz) + rounded("dsigmazz_dz", ahead(szz, Z) - szz, Z, 1, lz)
    inner = (i >= 1) & (i <= NX - 2) & (k >= 1) & (k <= NZ - 2)
    vx = np.where(inner, fma(ax, rx, vx * gx), f32(0))
    vz = np.where(inner, fma(az, rz, vz * gz), f32(0))
    return dict(zip(FIELDS[SEISMIC2], (vx, vz, sxx, szz, sxz))), M


@pytest.mark.parametrize("form", ["on chip", "streaming", "batch 1", "batch 2", "batch 4"])
@pytest.mark.parametrize("nx,nz,npml,atten", [
    (61, 50, 5, True),
    (230, 99, 9, False),   # tiles of 32 x 8 to 32 x 32 inside the strips
    (131, 140, 1, True),
])
def test_steps_round_as_written(gpu, nx, nz, npml, atten, form):
    chunks = (1, 5, 2)
    case = sy.small_case(SEISMIC2, seed=nx, nx=nx, nz=nz, npml=npml, nstep=sum(chunks), nrec=1, atten=atten)
    case.grid = dataclasses.replace(case.grid, dx=0.7, dz=0.6)  # spacings whose inverses are rounded
    case.srcfn[:] = 0.0
    rng = np.random.default_rng(nx)
    F = {n: ((1.0 if n[0] == "v" else 3e6) * rng.standard_normal((nz, nx))).astype(f32) for n in FIELDS[SEISMIC2]}
    M = {n: np.zeros((nz, nx), f32) for n in MEMORY[SEISMIC2]}
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
