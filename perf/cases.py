"""The work a user has this framework do, one case per kind of call.

A case is a shot (or a survey, or a gradient) through the public entry points:
``FDTDSolver`` for single shots, ``ShotPipeline`` for shots from and to host
arrays, ``Batch`` for surveys in one launch, ``TraceMisfit`` and
``SeismicTraceMisfit`` for gradients.  Grid sizes are full grids, CPML
included, of the repository's own workloads (1040 x 540 electromagnetic,
440 x 240 and 2040 x 1540 elastic, 630 x 70 x 330 for the 2.5-D kinds) and
generic smaller and larger ones; a run lasts while its waves cross the model.
"""
import math

import numpy as np
import torch

EPS0 = 8.85418782e-12
MU0 = 4.0e-7 * math.pi
CLIGHT = 299792458.0
EM2, EM2C, EM25, SEIS2, SEIS25 = "electromag2", "electromag2c", "electromag25", "seismic2", "seismic25"
NFIELDS = {EM2: 3, EM2C: 6, EM25: 6, SEIS2: 5, SEIS25: 9}
NCOEF = {EM2: 4, EM2C: 8, EM25: 6, SEIS2: 12, SEIS25: 39}
NCHAN = {EM2: 2, EM2C: 4, EM25: 3, SEIS2: 2, SEIS25: 3}
FLOPS = {EM2: 17, EM2C: 52, EM25: 45, SEIS2: 50, SEIS25: 189}  # a cell update off the CPML strips
VOIGT21 = [(a, b) for a in range(6) for b in range(a, 6)]


# ---------------------------------------------------------------------------
# The cases

def listed():
    return [
        # a small survey line or a test of a setting: latency and launches count
        dict(name="em2_small", path="run", kind=EM2, nx=120, ny=1, nz=90, npml=10, nstep=120, nrec=12, cpml="axes",
             model="planes"),
        # a ground-penetrating-radar shot of the repository's headline size
        dict(name="em2_shot", path="run", kind=EM2, nx=1040, ny=1, nz=540, npml=20, nstep=1000, nrec=100, cpml="axes",
             model="planes"),
        # a long, finely gridded radar section, given as a material image: far too large for the chip
        dict(name="em2_large", path="run", kind=EM2, nx=4040, ny=1, nz=3040, npml=20, nstep=96, nrec=200, cpml="axes",
             model="ids"),
        # complex permittivities (dispersive ground)
        dict(name="em2c_shot", path="run", kind=EM2C, nx=1040, ny=1, nz=540, npml=20, nstep=256, nrec=100, cpml="axes",
             model="planes"),
        # an elastic shot: firn over ice
        dict(name="seis2_shot", path="run", kind=SEIS2, nx=440, ny=1, nz=240, npml=20, nstep=400, nrec=40, cpml="axes",
             model="planes", atten=False, density="arithmetic", stress=False),
        # a large elastic section with attenuation and an explosive source
        dict(name="seis2_large", path="run", kind=SEIS2, nx=2040, ny=1, nz=1540, npml=20, nstep=128, nrec=100,
             cpml="axes", model="planes", atten=True, density="arithmetic", stress=True),
        # 2.5-D elastic, full stiffness per (x, z) column
        dict(name="seis25_shot", path="run", kind=SEIS25, nx=630, ny=70, nz=330, npml=15, nstep=48, nrec=100,
             cpml="axes", model="planes", atten=True, density="arithmetic", stress=True),
        # 2.5-D electromagnetic
        dict(name="em25_shot", path="run", kind=EM25, nx=630, ny=70, nz=330, npml=15, nstep=64, nrec=100, cpml="axes",
             model="planes"),
        # one gradient of a waveform inversion, radar and elastic: forward and backward
        dict(name="em2_gradient", path="gradient", kind=EM2, nx=1040, ny=1, nz=540, npml=20, nstep=800, nrec=100,
             cpml="axes", model="planes", every=200),
        dict(name="seis2_gradient", path="gradient", kind=SEIS2, nx=440, ny=1, nz=240, npml=20, nstep=400, nrec=40,
             cpml="axes", model="planes", atten=False, density="arithmetic", stress=False, every=200),
        # a survey in one launch: radar shots of one model and elastic models of uneven sizes
        dict(name="survey_batch", path="batch", kind=EM2, nx=1040, ny=1, nz=540, npml=20, nstep=256, nrec=40,
             cpml="axes", model="planes", shots=8, elastic=4),
        # shots from host arrays to host traces, one after another
        dict(name="shot_pipeline", path="pipeline", kind=EM2, nx=1040, ny=1, nz=540, npml=20, nstep=1000, nrec=100,
             cpml="axes", model="planes", shots=4),
    ]


def draw(rng):
    """One more case: a listed one's path and kind at another size, with other options."""
    base = dict(rng.choice(listed()))
    name = base.pop("name")
    span = {"em2_small": (7e3, 1.2e5), "em2_shot": (1e5, 9e5), "em2_large": (1e6, 1.2e7), "em2c_shot": (3e4, 1.5e6),
            "seis2_shot": (1e4, 2.8e5), "seis2_large": (2.5e5, 3.1e6), "seis25_shot": (1e5, 1.4e7),
            "em25_shot": (1e5, 1.4e7), "em2_gradient": (5e4, 5.6e5), "seis2_gradient": (2e4, 1.05e5),
            "survey_batch": (5e4, 5.6e5), "shot_pipeline": (5e4, 5.6e5)}[name]
    cells = math.exp(rng.uniform(math.log(span[0]), math.log(span[1])))
    base["npml"] = c = rng.choice([8, 10, 15, 20])
    least = 2 * c + 12
    if base["ny"] > 1:
        base["ny"] = max(least, min(rng.randint(least, 90), int(cells / (2 * least * least))))
        cells /= base["ny"]
    aspect = math.exp(rng.uniform(math.log(0.4), math.log(3.5)))  # nx / nz
    base["nx"] = max(least, int(math.sqrt(cells * aspect)))
    base["nz"] = max(least, int(math.sqrt(cells / aspect)))
    most = min(base["nstep"], int(max(base["nx"], base["nz"])))  # while the waves are in the model
    base["nstep"] = max(16, int(most * rng.uniform(0.4, 1.0)))
    base["nrec"] = rng.randint(1, base["nrec"])
    if base["path"] == "gradient":
        base["every"] = rng.choice([50, 100, 200])
    if base["path"] == "batch":
        base["shots"], base["elastic"] = rng.randint(1, 8), rng.randint(1, 4)
    if base["path"] == "pipeline":
        base["shots"] = rng.randint(1, 4)
    if "density" in base and base["path"] == "run":
        base["density"] = rng.choice(["arithmetic", "arithmetic", "harmonic", "geometric"])
        base["atten"] = rng.random() < 0.5
        base["stress"] = rng.random() < 0.4
    if base["path"] == "run" and base["kind"] in (EM2, SEIS2) and rng.random() < 0.2:
        base["cpml"] = "fields"  # the driver's 2-D CPML fields in place of the per-axis profiles
    return base


# ---------------------------------------------------------------------------
# Inputs, from the seed alone

def _extend(interior, c):
    return np.pad(interior, [(0, 0)] * (interior.ndim - 2) + [(c, c), (c, c)], mode="edge")


def _layers(rng, nx, nz, count):
    """Layer index (nz, nx): `count` layers with polygonal interfaces."""
    out = np.zeros((nz, nx), dtype=np.int32)
    xs = np.linspace(0, nx - 1, 8)
    for q in range(1, count):
        lo, hi = 0.15 + 0.7 * (q - 1) / (count - 1), 0.15 + 0.7 * q / (count - 1)
        line = np.interp(np.arange(nx), xs, rng.uniform(lo * nz, hi * nz, 8))
        out += np.arange(nz)[:, None] >= line[None, :]
    return out


def _profile(n, c, delta, sig, alp, scale, half):
    """K, a, b of one axis: quadratic CPML profiles over the c outer cells of both ends."""
    d = (delta * c - (np.arange(c) + (0.5 if half else 0.0)) * delta) / (delta * c)
    d = d / d.max()
    d = np.concatenate([d, np.zeros(n - 2 * c), d[::-1]])
    inside = np.r_[np.ones(c), np.zeros(n - 2 * c), np.ones(c)] > 0
    s, K = sig * d ** 2, 1.0 + 4.0 * d ** 2
    al = np.where(inside, alp * (1.0 - d) ** 2, 0.0)
    b = np.exp(-(s / K + al) * scale)
    a = np.where(s > 1e-6, s * (b - 1.0) / np.where(s > 1e-6, K * s + K * al, 1.0), 0.0)
    return K, a, b


def _hexagonal(rng, n):
    """(n, 6, 6) stiffness of ice crystals, c axis tilted up to 30 degrees from z."""
    C = np.zeros((6, 6))
    C[0, 0] = C[1, 1] = 13.9e9
    C[2, 2], C[0, 1], C[1, 0], C[5, 5] = 15.0e9, 7.1e9, 7.1e9, 3.4e9
    C[0, 2] = C[2, 0] = C[1, 2] = C[2, 1] = 5.8e9
    C[3, 3] = C[4, 4] = 3.0e9
    v = np.array([[0, 5, 4], [5, 1, 3], [4, 3, 2]])
    T = C[v[:, :, None, None], v[None, None]]
    t, p = np.deg2rad(rng.uniform(0, 30, n)), np.deg2rad(rng.uniform(0, 360, n))
    ct, st, cp, sp, z, one = np.cos(t), np.sin(t), np.cos(p), np.sin(p), np.zeros(n), np.ones(n)
    Ry = np.stack([ct, z, st, z, one, z, -st, z, ct], -1).reshape(n, 3, 3)
    Rz = np.stack([cp, -sp, z, sp, cp, z, z, z, one], -1).reshape(n, 3, 3)
    R = Rz @ Ry
    T = np.einsum("nai,nbj,nck,ndl,ijkl->nabcd", R, R, R, R, T, optimize=True)
    pairs = [(0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1)]
    return np.stack([np.stack([T[:, i, j, k, l] for k, l in pairs], -1) for i, j in pairs], -2)


def _ricker(nstep, dt, f0):
    a = np.pi * f0 * (np.arange(nstep) * dt - 1.0 / f0)
    return (1.0 - 2.0 * a * a) * np.exp(-a * a)


def _model(kind, case, rng):
    """(planes (n, nz, nx), largest speed, material image or None, its table)."""
    c = case["npml"]
    nx, nz = case["nx"] - 2 * c, case["nz"] - 2 * c
    if kind in (EM2, EM2C, EM25):
        ids = _extend(_layers(rng, nx, nz, 3), c)
        e = {k: rng.uniform(1.5, 3.2, 3) for k in ("11", "22", "33")}
        o = {k: rng.uniform(0.0, 0.05, 3) for k in ("12", "13", "23")}
        s = 10.0 ** rng.uniform(-6, -3, 3)
        zero = np.zeros(3)
        if kind == EM25:
            table = [e["11"], o["12"], o["13"], e["22"], o["23"], e["33"], s, zero, zero, s, zero, s]
        elif kind == EM2C:
            loss = [-rng.uniform(0.005, 0.02, 3) for _ in range(3)]
            table = [e["11"], e["11"] * loss[0], o["13"], o["13"] * loss[1], e["33"], e["33"] * loss[2], s, zero, s]
        else:
            table = [e["11"], o["13"], e["33"], s, zero, s]
        table = np.stack(table, 1)
        vmax = CLIGHT / math.sqrt(min(v.min() for v in e.values()))
        planes = None if case["model"] == "ids" else np.ascontiguousarray(table.T[:, ids])
        return planes, vmax, ids, table
    gamma = [rng.uniform(0.0, 0.02, (nz, nx)) if case["atten"] else np.zeros((nz, nx)) for _ in range(3)]
    if kind == SEIS25:
        C = _hexagonal(rng, 512)
        table = np.stack([C[:, a, b] for a, b in VOIGT21] + [np.full(512, 917.0)])
        planes = np.concatenate([table[:, rng.integers(0, 512, (nz, nx))], np.stack(gamma)])
        return _extend(planes, c), 4100.0, None, None
    lay = _layers(rng, nx, nz, 2)
    mats = np.array([[5e9, 2e9, 0.0, 5e9, 0.0, 1.5e9, 500.0], [13.9e9, 5.8e9, 0.3e9, 15.0e9, -0.2e9, 3.0e9, 917.0]]).T
    planes = mats[:, lay] * (1.0 + 0.02 * rng.uniform(-1, 1, (1, nz, nx)))
    return _extend(np.concatenate([planes, np.stack([gamma[0], gamma[2]])]), c), 4100.0, None, None


def _inputs(case, seed, kind=None, salt=0):
    """Everything a shot takes, as plain host arrays."""
    kind = kind or case["kind"]
    rng = np.random.default_rng([int(seed), salt, 77])
    case = {"atten": False, "density": "arithmetic", "stress": False, **case}
    c, nx, ny, nz, nstep = case["npml"], case["nx"], case["ny"], case["nz"], case["nstep"]
    three = kind in (SEIS25, EM25)
    seismic = kind in (SEIS2, SEIS25)
    d = 1.0 if kind == SEIS25 else 0.5 if kind == SEIS2 else 0.05
    planes, vmax, ids, table = _model(kind, case, rng)
    dt = (0.5 if kind == SEIS2 else 0.57 if three else 0.7) / (vmax * math.sqrt((3 if three else 2) / d ** 2))
    f0 = vmax / (24.0 * d) * rng.uniform(0.8, 1.1)
    if seismic:
        sig, alp, scale = -math.log(1e-3) * 3.0 * 0.7 * vmax / (2.0 * c), math.pi * f0, dt
    else:
        sig, alp, scale = -3.0 * math.log(1e-3) * EPS0 * CLIGHT / (2.0 * c * d), math.pi * EPS0 * f0, dt / EPS0
    axes = [_profile(n, c, d, sig, alp, scale, h) for n in ((nx, ny, nz) if three else (nx, nz)) for h in (False, True)]
    axes = [axes[2 * q] + axes[2 * q + 1] for q in range(len(axes) // 2)]
    fields2d = None
    if case["cpml"] == "fields":  # the x strips' coefficients, overwritten by the z strips'
        zin = (np.arange(nz) < c) | (np.arange(nz) >= nz - c)
        fields2d = np.stack([np.where(zin[:, None], axes[1][q][:, None], axes[0][q][None, :]) for q in range(6)])
    pos = lambda n: int(rng.integers(c + 2, n - c - 2))  # noqa: E731
    src = (pos(nx), pos(ny) if three else 0, pos(nz))
    reach = max(4, nstep // 4)  # cells a wave crosses in half the run: receivers lie where it arrives, up to the surface
    rec = np.stack([np.clip(src[0] + rng.integers(-reach, reach + 1, case["nrec"]), 1, nx - 3),
                    np.full(case["nrec"], src[1]),
                    np.maximum(c, src[2] - rng.integers(0, reach, case["nrec"]))], 1).astype(np.int32)
    w = _ricker(nstep, dt, f0)
    ncomp = 3 if three else 2
    srcfn = np.outer(np.zeros(ncomp) if case["stress"] else rng.uniform(0.4, 1.0, ncomp), w)
    stress = None
    if case["stress"]:
        stress = np.outer([1, 1, 1, 0, 0, 0] if three else [1, 1, 0], 1e4 * w)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, npml=c, nstep=nstep, d=d, dt=dt, f0=f0, planes=planes, ids=ids,
                table=table, axes=axes, fields2d=fields2d, src=src, rec=rec, srcfn=srcfn, stress=stress,
                density=case["density"], use_ids=case["model"] == "ids")


def _survey_shots(case, seed):
    """The radar shots of a survey: one model, the source and its receivers moved along the section."""
    out = [_inputs(case, seed)]
    nx, edge = out[0]["nx"], out[0]["npml"] + 3
    for q in range(1, case["shots"]):
        i = edge + (q * 61) % (nx - 2 * edge)
        rec = out[0]["rec"].copy()
        rec[:, 0] = np.clip(rec[:, 0] + i - out[0]["src"][0], 1, nx - 3)
        out.append(dict(out[0], src=(i, 0, out[0]["src"][2]), rec=rec))
    return out


def _elastic_cases(case):
    """Elastic models of uneven sizes beside the radar shots of a survey."""
    out = []
    for q in range(case["elastic"]):
        f = 0.25 + 0.7 * ((q * 5) % 7) / 7.0
        least = 2 * case["npml"] + 12
        out.append(dict(case, nx=max(least, int(case["nx"] * f)), nz=max(least, int(case["nz"] * (1.15 - f)))))
    return out


def _observed(x, seed):
    """Recorded traces to fit: two arrivals per receiver and channel."""
    rng = np.random.default_rng([int(seed), 5])
    t = np.arange(x["nstep"]) * x["dt"]
    out = np.zeros((x["nstep"], 2, len(x["rec"])))
    for r in range(len(x["rec"])):
        for ch in range(2):
            for amp in (1.0, 0.4):
                a = np.pi * x["f0"] * (t - rng.uniform(0.1, 0.9) * t[-1])
                out[:, ch, r] += amp * rng.uniform(-1, 1) * (1 - 2 * a * a) * np.exp(-a * a)
    return out * x["dt"] / (5.0 if x["kind"] == EM2 else 5000.0)


# ---------------------------------------------------------------------------
# Through the framework

def _grid(x):
    import seidart_gb300 as sg
    from seidart_gb300.solver import GridSpec
    kinds = {EM2: sg.ELECTROMAG2, EM25: sg.ELECTROMAG25, SEIS2: sg.SEISMIC2, SEIS25: sg.SEISMIC25}
    if x["kind"] == EM2C:
        from seidart_gb300._lib import ELECTROMAG2C
        kinds[EM2C] = ELECTROMAG2C
    return GridSpec(kinds[x["kind"]], x["nx"], x["nz"], x["d"], x["d"], x["dt"], x["npml"], ny=x["ny"], dy=x["d"])


def _packed(x):
    return np.concatenate([np.stack(a).ravel() for a in x["axes"]])


def _solver(x, like=None):
    from seidart_gb300.solver import FLAG_CPML_2D, FDTDSolver
    opts = {"density": x["density"]} if x["kind"] in (SEIS2, SEIS25) else {}
    s = FDTDSolver(_grid(x), x["nstep"], len(x["rec"]), flags=FLAG_CPML_2D if x["fields2d"] is not None else 0, **opts)
    if like is not None:
        s.share_model(like)
    elif x["use_ids"]:
        s.set_model_ids(x["ids"], x["table"])
    else:
        s.set_model(x["planes"])
    if x["fields2d"] is not None:
        s.set_cpml2d(x["fields2d"])
    else:
        s.set_cpml(_packed(x))
    s.set_source(x["src"], x["srcfn"])
    if x["stress"] is not None:
        s.set_stress_source(x["src"], x["stress"])
    s.set_receivers(x["rec"])
    return s


def prepare(case, seed):
    path = case["path"]
    if path == "batch":
        from seidart_gb300.batch import Batch
        shots = _survey_shots(case, seed)
        solvers = [_solver(shots[0])]
        solvers += [_solver(x, like=solvers[0]) for x in shots[1:]]
        solvers += [_solver(_inputs(k, seed, SEIS2, 1 + q)) for q, k in enumerate(_elastic_cases(case))]
        b = Batch(solvers)
        b.set_tiling(4, 3)
        return dict(path=path, batch=b, nstep=case["nstep"])
    if path == "pipeline":
        from seidart_gb300.solver import ShotPipeline
        xs = [_inputs(case, seed, salt=q) for q in range(case["shots"])]
        shots = [(_grid(x), x["planes"], _packed(x), x["src"], x["srcfn"], x["rec"]) for x in xs]
        return dict(path=path, pipeline=ShotPipeline(), shots=shots)
    x = _inputs(case, seed)
    if path == "run":
        return dict(path=path, solver=_solver(x), nstep=case["nstep"])
    from seidart_gb300 import adjoint
    obs = torch.tensor(_observed(x, seed), dtype=torch.float32, device="cuda")
    args = (_grid(x), x["planes"], _packed(x), x["src"], x["srcfn"], x["rec"])
    if x["kind"] == EM2:
        model = adjoint.TraceModel(*args, ckpt_every=case["every"])
        params = [x["planes"][0], x["planes"][2], x["planes"][3]]
    else:
        model = adjoint.SeismicTraceModel(*args, ckpt_every=case["every"])
        params = [x["planes"]]
    params = [torch.tensor(p, dtype=torch.float32, device="cuda", requires_grad=True) for p in params]
    return dict(path=path, model=model, params=params, obs=obs)


def _solver_outputs(s):
    from seidart_gb300.solver import FIELDS
    return {"traces": s.traces_tensor(), **{f: s.field_tensor(f) for f in FIELDS[s.kind]}}


def run(state):
    path = state["path"]
    if path == "run":  # one shot from rest, everything on the device
        s = state["solver"]
        s.reset()
        s.run(state["nstep"])
        return _solver_outputs(s)
    if path == "batch":
        b = state["batch"]
        b.reset()
        b.run(state["nstep"])
        return [_solver_outputs(s) for s in b.solvers]
    if path == "pipeline":
        return list(state["pipeline"].run(state["shots"]))
    from seidart_gb300 import adjoint
    fn = adjoint.TraceMisfit if len(state["params"]) == 3 else adjoint.SeismicTraceMisfit
    traces = fn.apply(*state["params"], state["model"])
    resid = traces.detach() - state["obs"]  # of half the squared misfit
    grads = torch.autograd.grad(traces, state["params"], resid)
    return {"traces": traces.detach(), "gradients": list(grads)}


def work(case):
    """Model and final state across memory once, and the arithmetic of every step."""
    def one(kind, k, n=1):
        cells = k["nx"] * k["ny"] * k["nz"]
        plane = k["nx"] * k["nz"] if kind in (SEIS25, EM25) else cells
        traces = k["nstep"] * NCHAN[kind] * k["nrec"]
        return (4.0 * (NCOEF[kind] * plane + n * (NFIELDS[kind] * cells + traces)),
                1.0 * n * FLOPS[kind] * cells * k["nstep"])
    path = case["path"]
    b, f = one(case["kind"], case, case.get("shots", 1))
    if path == "batch":
        for k in _elastic_cases(case):
            b2, f2 = one(SEIS2, k)
            b, f = b + b2, f + f2
    if path == "pipeline":  # every shot brings its own FP64 planes
        cells = case["nx"] * case["nz"]
        b = case["shots"] * (8.0 * 6 * cells + 4.0 * case["nstep"] * 2 * case["nrec"])
    if path == "gradient":  # a transposed step costs two forward ones
        b, f = 2 * b, 3 * f
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# In 64 bits, with plain torch

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    a = np.asarray(a)
    return torch.tensor(a, dtype=torch.complex128 if np.iscomplexobj(a) else torch.float64, device=_dev())


class _Space:
    """Differences and CPML recursions on full arrays (z, [y,] x), masked to the loops' ranges."""

    def __init__(self, x):
        self.three = x["kind"] in (SEIS25, EM25)
        self.dims = {"z": 0, "y": 1, "x": 2} if self.three else {"z": 0, "x": 1}
        self.shape = (x["nz"], x["ny"], x["nx"]) if self.three else (x["nz"], x["nx"])
        self.d = x["d"]
        self.tab = {}
        for ax, prof in zip("xyz" if self.three else "xz", x["axes"]):
            view = [1] * len(self.shape)
            view[self.dims[ax]] = -1
            vals = [_t(v).view(view) for v in prof] if x["fields2d"] is None else [_t(v) for v in x["fields2d"]]
            for h in (0, 1):
                K, a, b = vals[3 * h:3 * h + 3]
                self.tab[ax, h] = (1.0 / (K * self.d), a / self.d, b)

    def at(self, f, ax, by):
        """f at the cell `by` further along ax (wraps: masked where it would matter)."""
        return torch.roll(f, -by, self.dims[ax])

    def diff(self, f, ax, side):
        return self.at(f, ax, 1) - f if side > 0 else f - self.at(f, ax, -1)

    def mask(self, **ranges):
        """1.0 in the cells with lo <= index <= n - 1 - hi along each named axis."""
        m = torch.ones(self.shape, dtype=torch.float64, device=_dev())
        for ax, (lo, hi) in ranges.items():
            q, n = self.dims[ax], self.shape[self.dims[ax]]
            if lo:
                m.narrow(q, 0, lo).zero_()
            if hi:
                m.narrow(q, n - hi, hi).zero_()
        return m

    def without(self, *planes):
        """1.0 off the planes (axis, index)."""
        m = torch.ones(self.shape, dtype=torch.float64, device=_dev())
        for ax, i in planes:
            m.select(self.dims[ax], i).zero_()
        return m

    def memory(self, dtype=torch.float64):
        return torch.zeros(self.shape, dtype=dtype, device=_dev())

    def cpml(self, psi, d, ax, half, where):
        """(psi, derivative) after the recursion in the cells of `where`."""
        ik, a, b = self.tab[ax, half]
        psi = psi + where * ((b - 1.0) * psi + a * d)
        return psi, d * ik + psi


def _spot(sp, x):
    m = torch.zeros(sp.shape, dtype=torch.float64, device=_dev())
    i, j, k = x["src"]
    m[(k, j, i) if sp.three else (k, i)] = 1.0
    return m


def _em2_steps(x, planes, start=None):
    """A function advancing (state, t) by one step, for real and complex permittivities."""
    sp = _Space(x)
    dt = x["dt"]
    if x["kind"] == EM2C:
        e11, e13, e33 = (torch.complex(planes[2 * q], planes[2 * q + 1]) for q in range(3))
        s11, s13, s33 = planes[6], planes[7], planes[8]
    else:
        e11, e13, e33, s11, s13, s33 = planes
    ca, cb = [], []
    for e, s in (((e11 + e13) * EPS0, s11 + s13), ((e13 + e33) * EPS0, s13 + s33)):
        ca.append((1 - s * dt / (2 * e)) / (1 + s * dt / (2 * e)))
        cb.append((dt / e) / (1 + s * dt / (2 * e)))
    inh, inx, inz = sp.mask(x=(0, 1), z=(0, 1)), sp.mask(x=(0, 1), z=(1, 1)), sp.mask(x=(1, 1), z=(0, 1))
    nx, nz = x["nx"], x["nz"]
    zx = sp.without(("x", 0), ("x", nx - 2), ("z", 0), ("z", nz - 1))
    zz = sp.without(("x", 0), ("x", nx - 1), ("z", 0), ("z", nz - 2))
    zh = sp.without(("x", 0), ("x", nx - 2), ("z", 0), ("z", nz - 2))
    av = lambda c, ax: (c + sp.at(c, ax, -1)) / 2  # noqa: E731
    cax, cbx = zx * (1 + inx * (av(ca[0], "z") - 1)), zx * inx * av(cb[0], "z")
    caz, cbz = zz * (1 + inz * (av(ca[1], "x") - 1)), zz * inz * av(cb[1], "x")
    spot = _spot(sp, x)
    i, _, k = x["src"]
    amp = [x["srcfn"][0] * dt, x["srcfn"][1] * dt]
    spotx, spotz = spot / e11[k, i], spot / e33[k, i]
    dbh = inh * (dt / MU0)

    def step(st, t):
        ex, ez, hy, p1, p2, p3, p4 = st
        p1, vz = sp.cpml(p1, sp.diff(ex, "z", 1), "z", 0, inh)
        p2, vx = sp.cpml(p2, sp.diff(ez, "x", 1), "x", 0, inh)
        hy = hy + dbh * (vx + vz)
        p3, d = sp.cpml(p3, sp.diff(hy, "z", -1), "z", 1, inx)
        ex = cax * ex + cbx * d + spotx * amp[0][t]
        p4, d = sp.cpml(p4, sp.diff(hy, "x", -1), "x", 1, inz)
        ez = caz * ez + cbz * d + spotz * amp[1][t]
        return ex, ez, hy * zh, p1, p2, p3, p4

    dtype = torch.complex128 if x["kind"] == EM2C else torch.float64
    return step, tuple(sp.memory(dtype) for _ in range(7)), 2, 3


def _rho_avg(method, w, r, a, b):
    if method == "geometric":
        return (r ** w * a * b) ** (1.0 / (w + 2))
    if method == "harmonic":
        return (w + 2.0) / (w / r + 1.0 / a + 1.0 / b)
    return (w * r + a + b) / (w + 2.0)


def _seis2_steps(x, planes):
    sp = _Space(x)
    dt = x["dt"]
    c11, c13, c15, c33, c35, c55, rho, gx, gz = planes
    la, lb = sp.mask(x=(0, 1), z=(1, 0)), sp.mask(x=(1, 0), z=(0, 1))
    inn = sp.mask(x=(1, 1), z=(1, 1))
    A = [la * (sp.at(c, "x", 1) + 2 * c + sp.at(c, "z", -1)) / 4 * dt for c in (c11, c13, c15, c33, c35)]
    B = [lb * (sp.at(c, "z", 1) + 2 * c + sp.at(c, "x", -1)) / 4 * dt for c in (c15, c35, c55)]
    rx = inn * dt / _rho_avg(x["density"], 2, rho, sp.at(rho, "x", -1), sp.at(rho, "z", -1))
    rz = inn * dt / _rho_avg(x["density"], 2, rho, sp.at(rho, "x", 1), sp.at(rho, "z", 1))
    gx, gz = inn * (1 - gx), inn * (1 - gz)
    i, _, k = x["src"]
    spot = _spot(sp, x)
    force = spot * (dt / rho[k, i])
    f, s = x["srcfn"], x["stress"]

    def step(st, t):
        vx, vz, sxx, szz, sxz, *m = st
        m = list(m)
        m[0], xx = sp.cpml(m[0], sp.diff(vx, "x", 1), "x", 1, la)
        m[1], zz = sp.cpml(m[1], sp.diff(vz, "z", -1), "z", 0, la)
        m[2], xz = sp.cpml(m[2], sp.diff(vx, "z", -1), "z", 1, la)
        m[3], zx = sp.cpml(m[3], sp.diff(vz, "x", 1), "x", 0, la)
        sxx = sxx + A[0] * xx + A[1] * zz + A[2] * (zx + xz)
        szz = szz + A[1] * xx + A[3] * zz + A[4] * (zx + xz)
        m[4], xx = sp.cpml(m[4], sp.diff(vx, "x", -1), "x", 1, lb)
        m[5], zz = sp.cpml(m[5], sp.diff(vz, "z", 1), "z", 0, lb)
        m[6], xz = sp.cpml(m[6], sp.diff(vx, "z", 1), "z", 1, lb)
        m[7], zx = sp.cpml(m[7], sp.diff(vz, "x", -1), "x", 0, lb)
        sxz = sxz + B[0] * xx + B[1] * zz + B[2] * (zx + xz)
        if s is not None:
            sxx, szz, sxz = sxx + spot * (s[0][t] * dt), szz + spot * (s[1][t] * dt), sxz + spot * (s[2][t] * dt)
        m[8], d1 = sp.cpml(m[8], sp.diff(sxx, "x", -1), "x", 0, sp_vx)
        m[9], d2 = sp.cpml(m[9], sp.diff(sxz, "z", -1), "z", 0, sp_vx)
        vx = gx * vx + rx * (d1 + d2) + force * f[0][t]
        m[10], d1 = sp.cpml(m[10], sp.diff(sxz, "x", 1), "x", 1, sp_vz)
        m[11], d2 = sp.cpml(m[11], sp.diff(szz, "z", 1), "z", 1, sp_vz)
        vz = gz * vz + rz * (d1 + d2) + force * f[1][t]
        return (vx, vz, sxx, szz, sxz, *m)

    sp_vx, sp_vz = sp.mask(x=(1, 0), z=(1, 0)), sp.mask(x=(0, 1), z=(0, 1))
    return step, tuple(sp.memory() for _ in range(17)), 2, 5


def _seis25_steps(x, planes):
    sp = _Space(x)
    dt = x["dt"]
    col = [p[:, None, :] for p in planes]
    C = {ab: col[q] for q, ab in enumerate(VOIGT21)}
    C.update({(b, a): v for (a, b), v in C.items()})
    rho, g = col[21], col[22:25]

    def quad(c, dx, dz):
        return (c + torch.roll(c, -dx, 2) + torch.roll(c, -dz, 0) + torch.roll(c, (-dz, -dx), (0, 2))) / 4 * dt

    # per stress loop: sides and offsets of the x, y, z differences, the stresses it advances
    loops = [((1, 1), (-1, 0), (-1, 0), (0, 1, 2)), ((-1, 0), (1, 1), (-1, 1), (5,)),
             ((-1, 0), (-1, 0), (1, 1), (4,)), ((1, 1), (1, 1), (1, 1), (3,))]
    span = lambda side: (0, 1) if side > 0 else (1, 0)  # noqa: E731
    where, K = [], []
    for sx, sy, sz, rows in loops:
        where.append(sp.mask(x=span(sx[0]), y=span(sy[0]), z=span(sz[0])))
        K.append({(r, q): quad(C[r, q], sx[0], sz[0]) * (1.0 if q < 3 else 0.5) for r in rows for q in range(6)})
    vel = [((-1, 0), (-1, 0), (-1, 0), (0, 5, 4), (-1, -1)), ((1, 1), (1, 1), (-1, 0), (5, 1, 3), (1, -1)),
           ((1, 1), (-1, 0), (1, 1), (4, 3, 2), (1, 1))]
    vwhere = [sp.mask(x=span(v[0][0]), y=span(v[1][0]), z=span(v[2][0])) for v in vel]
    inn = sp.mask(x=(1, 1), y=(1, 1), z=(1, 1))
    r = [dt / _rho_avg(x["density"], 4, rho, torch.roll(rho, -v[4][0], 2), torch.roll(rho, -v[4][1], 0)) for v in vel]
    i, j, k = x["src"]
    spot = _spot(sp, x)
    f, s = x["srcfn"], x["stress"]
    force = dt / planes[21][k, i]

    def step(st, t):
        v, sig, m, n = list(st[:3]), [st[q] for q in (3, 4, 5, 8, 7, 6)], list(st[9:18]), list(st[18:27])
        for q, (sx, sy, sz, rows) in enumerate(loops):
            D = [[None] * 3 for _ in range(3)]  # D[a][b]: derivative of v[a] along axis b
            for b, (ax, (side, half)) in enumerate(zip("xyz", (sx, sy, sz))):
                for a in range(3):
                    raw = sp.diff(v[a], ax, side)
                    m[3 * a + b], D[a][b] = sp.cpml(m[3 * a + b], raw, ax, half, where[q])
                    if q == 1 and (a, b) in ((2, 0), (0, 2)):  # the two the sigma_xy loop leaves unscaled
                        D[a][b] = raw / sp.d
            e = [D[0][0], D[1][1], D[2][2], D[1][2] + D[2][1], D[0][2] + D[2][0], D[0][1] + D[1][0]]
            for row in rows:
                sig[row] = sig[row] + where[q] * sum(K[q][row, p] * e[p] for p in range(6))
        if s is not None:
            for row, comp in zip((0, 1, 2, 5, 4, 3), range(6)):
                sig[row] = sig[row] + spot * (s[comp][t] * dt)
        for a, (sx, sy, sz, parts, _) in enumerate(vel):
            total = 0.0
            for b, (ax, (side, half)) in enumerate(zip("xyz", (sx, sy, sz))):
                n[3 * a + b], d = sp.cpml(n[3 * a + b], sp.diff(sig[parts[b]], ax, side), ax, half, vwhere[a])
                total = total + d
            v[a] = inn * (v[a] * (1 - g[a]) + total * r[a]) + spot * (force * f[a][t])
        return (*v, sig[0], sig[1], sig[2], sig[5], sig[4], sig[3], *m, *n)

    return step, tuple(sp.memory() for _ in range(27)), 3, 9


def _em25_steps(x, planes):
    sp = _Space(x)
    dt, nx, ny, nz = x["dt"], x["nx"], x["ny"], x["nz"]
    e11, e12, e13, e22, e23, e33, s11, s12, s13, s22, s23, s33 = (p[:, None, :] for p in planes)
    ca, cb = [], []
    for e, s in ((e11 + e12 + e13, s11 + s12 + s13), (e12 + e22 + e23, s12 + s22 + s23),
                 (e13 + e23 + e33, s13 + s23 + s33)):
        q = s * dt / (2 * e * EPS0)
        ca.append((1 - q) / (1 + q))
        cb.append((dt / (e * EPS0)) / (1 + q))
    six = lambda c, dz: (4 * c + torch.roll(c, 1, 2) + torch.roll(c, -dz, 0)) / 6  # noqa: E731
    ca, cb = [ca[0], six(ca[1], -1), six(ca[2], 1)], [cb[0], six(cb[1], -1), six(cb[2], 1)]
    lo, up = (0, 1), (1, 1)
    hin = [sp.mask(x=lo, y=lo, z=lo), sp.mask(x=lo, y=lo, z=lo), sp.mask(x=lo, y=lo, z=up)]
    ein = [sp.mask(x=lo, y=up, z=up), sp.mask(x=up, y=lo, z=up), sp.mask(x=up, y=up, z=lo)]
    face = lambda a, b, c: sp.without(("x", 0), ("x", nx - a), ("y", 0), ("y", ny - b), ("z", 0), ("z", nz - c))  # noqa: E731
    ez0 = [face(2, 1, 1), face(1, 2, 1), face(1, 1, 2)]
    hz0 = [face(1, 2, 2), face(2, 1, 2), face(2, 2, 1)]
    # (field, axis, half offset, sign): the two derivatives of each H, then of each E
    hd = [((2, "y", 1, -1), (1, "z", 1, 1)), ((0, "z", 0, -1), (2, "x", 0, 1)), ((0, "y", 0, 1), (1, "x", 0, -1))]
    ed = [((2, "y", 1, 1), (1, "z", 0, -1)), ((2, "x", 1, -1), (0, "z", 1, 1)), ((0, "y", 1, -1), (1, "x", 1, 1))]
    spot = _spot(sp, x)
    i, j, k = x["src"]
    amp = [x["srcfn"][q] * dt / float(planes[p][k, i]) for q, p in enumerate((0, 3, 5))]

    def step(st, t):
        E, H, m, n = list(st[:3]), list(st[3:6]), list(st[6:12]), list(st[12:18])
        for a in range(3):
            total = 0.0
            for q, (b, ax, half, sign) in enumerate(hd[a]):
                m[2 * a + q], d = sp.cpml(m[2 * a + q], sign * sp.diff(E[b], ax, 1), ax, half, hin[a])
                total = total + d
            H[a] = H[a] + hin[a] * (dt / MU0) * total
        for a in range(3):
            total = 0.0
            for q, (b, ax, half, sign) in enumerate(ed[a]):
                n[2 * a + q], d = sp.cpml(n[2 * a + q], sign * sp.diff(H[b], ax, -1), ax, half, ein[a])
                total = total + d
            E[a] = ez0[a] * (E[a] + ein[a] * ((ca[a] - 1) * E[a] + cb[a] * total) + spot * amp[a][t])
        return (*E, *(h * z for h, z in zip(H, hz0)), *m, *n)

    return step, tuple(sp.memory() for _ in range(18)), 3, 6


STEPS = {EM2: _em2_steps, EM2C: _em2_steps, EM25: _em25_steps, SEIS2: _seis2_steps, SEIS25: _seis25_steps}
NAMES = {EM2: ["Ex", "Ez", "Hy"], EM2C: ["Ex_re", "Ex_im", "Ez_re", "Ez_im", "Hy_re", "Hy_im"],
         EM25: ["Ex", "Ey", "Ez", "Hx", "Hy", "Hz"], SEIS2: ["vx", "vz", "sigmaxx", "sigmazz", "sigmaxz"],
         SEIS25: ["vx", "vy", "vz", "sigmaxx", "sigmayy", "sigmazz", "sigmaxy", "sigmaxz", "sigmayz"]}


def _planes64(x):
    if x["planes"] is not None:
        return [_t(p) for p in x["planes"]]
    ids = torch.tensor(x["ids"], device=_dev(), dtype=torch.int64)
    return [_t(col)[ids] for col in x["table"].T]


def _sampler(x):
    rec = torch.tensor(x["rec"].astype(np.int64), device=_dev())
    if x["kind"] in (SEIS25, EM25):
        return lambda f: f[rec[:, 2], rec[:, 1], rec[:, 0]]
    return lambda f: f[rec[:, 2], rec[:, 0]]


def _parts(values):
    """Complex arrays as real and imaginary ones, in turn."""
    out = []
    for v in values:
        out += [v.real, v.imag] if v.is_complex() else [v]
    return out


@torch.no_grad()
def _shot64(x):
    step, st, nch, nf = STEPS[x["kind"]](x, _planes64(x))
    take = _sampler(x)
    traces = []
    for t in range(x["nstep"]):
        st = step(st, t)
        traces.append(torch.stack(_parts([take(f) for f in st[:nch]])))
    return {"traces": torch.stack(traces), **dict(zip(NAMES[x["kind"]], _parts(st[:nf])))}


def _gradient64(x, seed, every=50):
    """Traces and gradient by automatic differentiation, the states kept every few steps and the rest rerun."""
    obs = torch.tensor(_observed(x, seed), dtype=torch.float32, device=_dev()).double()
    planes = [torch.tensor(p, dtype=torch.float32, device=_dev()).double() for p in x["planes"]]
    if x["kind"] == EM2:  # eps13 and sig13 stay as given; sig11 = sig33
        fixed = _planes64(x)
        leaves = [planes[0], planes[2], planes[3]]
        build = lambda v: [v[0], fixed[1], v[1], v[2], fixed[4], v[2]]  # noqa: E731
    else:
        leaves = [torch.stack(planes)]
        build = lambda v: list(v[0])  # noqa: E731
    leaves = [v.requires_grad_() for v in leaves]
    take = _sampler(x)
    nstep = x["nstep"]
    with torch.no_grad():
        step, st, nch, _ = STEPS[x["kind"]](x, build(leaves))
        kept, traces = [], []
        for t in range(nstep):
            if t % every == 0:
                kept.append(st)
            st = step(st, t)
            traces.append(torch.stack([take(f) for f in st[:nch]]))
        traces = torch.stack(traces)
        resid = traces - obs
    grads = [torch.zeros_like(v) for v in leaves]
    lam = [torch.zeros_like(v) for v in st]
    for q in reversed(range(len(kept))):
        first = tuple(v.detach().requires_grad_() for v in kept[q])
        with torch.enable_grad():
            step, _, nch, _ = STEPS[x["kind"]](x, build(leaves))
            cur, misfit = first, 0.0
            for t in range(q * every, min(nstep, (q + 1) * every)):
                cur = step(cur, t)
                misfit = misfit + (torch.stack([take(f) for f in cur[:nch]]) * resid[t]).sum()
            total = misfit + sum((a * b).sum() for a, b in zip(cur, lam))
            got = torch.autograd.grad(total, [*leaves, *first], allow_unused=True)
        for g, v in zip(grads, got):
            if v is not None:
                g += v
        lam = [torch.zeros_like(a) if v is None else v for a, v in zip(first, got[len(leaves):])]
    return {"traces": traces, "gradients": grads}


def exact(case, seed):
    path = case["path"]
    if path == "batch":
        out = [_shot64(x) for x in _survey_shots(case, seed)]
        return out + [_shot64(_inputs(k, seed, SEIS2, 1 + q)) for q, k in enumerate(_elastic_cases(case))]
    if path == "pipeline":
        return [_shot64(_inputs(case, seed, salt=q))["traces"] for q in range(case["shots"])]
    x = _inputs(case, seed)
    return _shot64(x) if path == "run" else _gradient64(x, seed)
