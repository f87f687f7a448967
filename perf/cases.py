"""Performance cases of the propagation path, through the entry points a user's program calls.

Kinds of case (``case["kind"]``):

  forward, adjoint   one shot's nonlinear propagation or its time-reversed adjoint with device
                     signals (``Propagator.nl_propagate_device``)
  batch              several shots of one medium in one launch sequence
                     (``Propagator.nl_forward_batch_device``)
  born_forward,      one shot's linearised modelling and its adjoint on host arrays, as the
  born_adjoint       reference's drivers are called (``Propagator.born_forward`` / ``born_adjoint``)
  operator           the drop-in nonlinear operator over its shots on host arrays
                     (``nonlinearPropElasticShotsGpu_3D.forward``)
  misfit             misfit and gradient over (rho, lambda, mu) through autograd
                     (``ElasticFwiMisfit``)
  gradient           one shot of such an evaluation on a grid whose wavefields are checkpointed and
                     recomputed (``FwiProblem.shot_misfit_and_gradient``)

Grids run from the 64-cell grids of the tests to the full modelling grid of 392 x 488 x 488 cells.
Records are cut short, so that a pass stays below a second; the time loop does the same work per
fine step whatever the record's length.  ``exact`` restates the scheme in plain torch in FP64.
"""
from __future__ import annotations

import functools

import numpy as np
import torch

from elasticisolib_3d_b200 import fwi as F
from elasticisolib_3d_b200 import hostprep as H
from elasticisolib_3d_b200 import operators as OP
from elasticisolib_3d_b200.engine import COMP_GRID, Propagator

FAT = 4
D = 10.0            # cell size, metres
DTW = 0.0005        # fine time step, seconds (Courant number 0.28 at 2750 m/s)
VX, VY, VZ, SXX, SYY, SZZ, SXZ, SXY, SYZ = range(9)


# ----------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------
def listed():
    return [
        # a test-sized grid: a long record of short fine steps, where launches and latency count
        dict(name="forward-small", kind="forward", nz=72, nx=72, ny=60, pad=8, nts=100, sub=4, nrec=8, surface=False),
        # plain forward modelling: 120^3 interior, 30-cell sponge, free surface, 40 x 40 receivers
        dict(name="forward-plain", kind="forward", nz=168, nx=200, ny=188, pad=30, nts=50, sub=4, nrec=40,
             surface=True),
        # the full modelling grid, 400 x 400 x 300 interior and 40-cell sponge, 200 x 200 receivers
        dict(name="forward-large", kind="forward", nz=392, nx=488, ny=488, pad=40, nts=10, sub=4, nrec=200,
             surface=False),
        # a grid that no block size divides: odd on every axis, odd number of fine steps per sample
        dict(name="forward-odd", kind="forward", nz=101, nx=91, ny=117, pad=12, nts=60, sub=3, nrec=20,
             surface=False),
        # the time-reversed adjoint with every receiver component injected, odd number of planes
        dict(name="adjoint-plain", kind="adjoint", nz=168, nx=152, ny=171, pad=20, nts=50, sub=4, nrec=40,
             surface=False),
        # several shots of one medium advanced together
        dict(name="batch-six-shots", kind="batch", nz=136, nx=136, ny=124, pad=16, nts=40, sub=4, nrec=24, shots=6),
        # linearised modelling and its adjoint, host arrays in and out
        dict(name="born-forward", kind="born_forward", nz=168, nx=168, ny=152, pad=24, nts=30, sub=4, nrec=32),
        dict(name="born-adjoint", kind="born_adjoint", nz=168, nx=168, ny=152, pad=24, nts=30, sub=4, nrec=32),
        # the drop-in operator: two shots, host arrays, spreading and interpolation included
        dict(name="operator-two-shots", kind="operator", nz=104, nx=104, ny=96, pad=12, nts=100, sub=4, nrec=16,
             shots=2),
        # a small inversion's objective: misfit and gradient of one shot through autograd
        dict(name="misfit-small", kind="misfit", nz=72, nx=72, ny=64, pad=8, nts=60, sub=4, nrec=16),
        # one shot of a gradient on 200^3 interior + 40, wavefields checkpointed in FP32
        dict(name="gradient-medium", kind="gradient", nz=296, nx=296, ny=288, pad=40, nts=20, sub=4, nrec=100,
             segment=6, store="fp32"),
        # one shot of a gradient on 300^3 interior + 40 with FP16 checkpoints and velocity slots, most
        # of the source wavefield recomputed, 150 x 150 receivers
        dict(name="gradient-large", kind="gradient", nz=392, nx=392, ny=388, pad=40, nts=15, sub=4, nrec=150,
             segment=3, store="fp16"),
    ]


def _cells(c):
    return (c["nz"] - 2 * FAT) * (c["nx"] - 2 * FAT) * (c["ny"] - 2 * FAT)


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    """A case of the listed ranges: grids of 64 to about 400 cells an axis, records of 10 to 100 samples."""
    kind = rng.choice(["forward", "forward", "adjoint", "batch", "born_forward", "born_adjoint", "operator", "misfit",
                       "gradient", "gradient"])
    top = {"forward": 400, "adjoint": 400, "batch": 200, "born_forward": 200, "born_adjoint": 200, "operator": 140,
           "misfit": 140, "gradient": 300}[kind]
    bottom = 160 if kind == "gradient" else 64
    size = _log_uniform(rng, bottom, top)
    ax = [max(56, min(top + 40, int(size * (0.8 + 0.4 * rng.random())))) for _ in range(3)]
    # grids of the shot operators and of FwiProblem are blocks of 16 and the ring along z and x; a
    # Propagator takes any size
    block = kind in ("operator", "misfit", "gradient") or rng.random() < 0.6
    nz, nx = ((n - 8) // 16 * 16 + 8 if block else n for n in ax[:2])
    sub = 2 * rng.randint(1, 3) if kind in ("operator", "misfit", "gradient") else rng.randint(2, 6)
    c = dict(kind=kind, nz=nz, nx=nx, ny=ax[2], pad=rng.randint(8, 20), sub=sub)
    if kind == "batch":
        c["nz"] = (c["nz"] - 8) // 4 * 4 + 8  # the batched launch takes rows of a multiple of four cells
    room = max(8, min(c["nz"], c["nx"], c["ny"]) - 2 * FAT - 2 * c["pad"] - 4)
    c["nrec"] = rng.randint(4, room // 2)
    shots = rng.randint(2, 6) if kind == "batch" else rng.randint(1, 3) if kind == "operator" else 1
    if kind in ("batch", "operator"):
        c["shots"] = shots
    # the record: about 20 to 2000 million cell updates, 10 to 100 samples
    updates = _log_uniform(rng, 2e7, 2e9)
    c["nts"] = max(10, min(100, int(updates / (_cells(c) * sub * shots))))
    if kind == "forward":
        c["surface"] = rng.random() < 0.3
    if kind == "gradient":
        c["segment"] = rng.randint(2, 6)
        c["store"] = rng.choice(["fp32", "fp16"])
    return c


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _smooth(c, seed, salt):
    """A smooth random field in [-1, 1], drawn on a grid eight times coarser."""
    shape = (c["ny"], c["nx"], c["nz"])
    coarse = torch.randn((1, 1) + tuple(n // 8 + 2 for n in shape), device="cuda", generator=_gen(seed, salt))
    f = torch.nn.functional.interpolate(coarse, size=shape, mode="trilinear", align_corners=True)[0, 0]
    return f / f.abs().max()


def _model(c, seed):
    """(rho, lambda, mu): 2500 m/s and 2000 kg/m^3 with smooth perturbations of up to 10 %."""
    vp = 2500.0 * (1 + 0.10 * _smooth(c, seed, 1))
    vs = vp / 1.732 * (1 + 0.03 * _smooth(c, seed, 2))
    rho = 2000.0 * (1 + 0.10 * _smooth(c, seed, 3))
    mu = rho * vs * vs
    return rho.contiguous(), (rho * vp * vp - 2 * mu).contiguous(), mu.contiguous()


def _avg(f, dim):
    """The staggering average of the medium along one axis, first and last cells as the scheme has them."""
    n = f.shape[dim]
    a, b = f.narrow(dim, 1, n - 2), f.narrow(dim, 0, n - 2)
    last = f.narrow(dim, n - 1, 1) + 0.5 * f.narrow(dim, n - 2, 1)
    return torch.cat([0.5 * f.narrow(dim, 0, 1), 0.5 * (a + b), last], dim)


def _planes64(rho, lam, mu):
    """The eight scaled medium planes in FP64."""
    rho, lam, mu = rho.double(), lam.double(), mu.double()
    two = 2.0 * float(np.float32(DTW))
    mx = _avg(mu, 1)
    return [two / _avg(rho, 1), two / _avg(rho, 0), two / _avg(rho, 2), two * (lam + 2 * mu), two * lam,
            two * _avg(mx, 2), two * _avg(mx, 0), two * _avg(_avg(mu, 0), 2)]


def _planes(c, seed):
    return torch.stack([p.float() for p in _planes64(*_model(c, seed))])


def _ricker(c, f=15.0):
    t = np.arange(c["nts"]) * DTW * c["sub"]
    a = (np.pi * f * (t - min(1.0 / f, 0.35 * t[-1]))) ** 2
    return ((1 - 2 * a) * np.exp(-a)).astype(np.float32)


def _dts(c):
    return float(np.float32(DTW) * np.float32(c["sub"]))


def _pads(c):
    """The sponge: free-surface grids have none on top."""
    top = FAT if c.get("surface") else c["pad"]
    return top, c["pad"]


def _stations(c, seed):
    """Cell indices (z, x, y) of the receivers' lower corners, on a square near the top, and those of
    the shots' sources, drawn from the seed."""
    zp, p = _pads(c)
    lo, nx, ny = FAT + p, c["nx"] - 2 * FAT - 2 * p - 3, c["ny"] - 2 * FAT - 2 * p - 3
    n = c["nrec"]
    x, y = (lo + np.linspace(0, m, n).astype(np.int64) for m in (nx, ny))
    X, Y = np.meshgrid(x, y, indexing="ij")
    rec = np.stack([np.full(X.size, FAT + zp + 1), X.ravel(), Y.ravel()])
    rng = np.random.default_rng(1000 + seed)
    ns = c.get("shots", 1)
    src = np.stack([np.full(ns, FAT + zp + 3), lo + (nx * (0.2 + 0.6 * rng.random(ns))).astype(np.int64),
                    lo + (ny * (0.2 + 0.6 * rng.random(ns))).astype(np.int64)])
    return rec, src


def _corner_table(c, st):
    """Regular points of the devices at cells st (3, n): the eight corners of each, in first-seen order."""
    base = (st[2] * c["nx"] + st[1]) * c["nz"] + st[0]
    off = [k + c["nz"] * (i + c["nx"] * j) for j in (0, 1) for i in (0, 1) for k in (0, 1)]
    pts = (base[:, None] + np.asarray(off)[None, :]).ravel()
    _, first = np.unique(pts, return_index=True)
    return pts[np.sort(first)]


def _regular(c, seed):
    """Regular-grid acquisition: the explosive sources' tables and signals (already scaled by the
    medium) per shot, the receivers' table, and for the adjoints random data at every receiver point."""
    rec, src = _stations(c, seed)
    w = 1.0e3 * _ricker(c)
    tabs = [_corner_table(c, src[:, i:i + 1]) for i in range(src.shape[1])]
    sig = [np.outer(w, 0.125 * (1 + 0.1 * np.arange(len(t)))).astype(np.float32) for t in tabs]
    return tabs, sig, _corner_table(c, rec)


def _data(c, seed, npts):
    """Adjoint data (nts, 9, npts): smooth in time, random over the points."""
    a = torch.randn((2, 9, npts), device="cuda", generator=_gen(seed, 11))
    t = torch.arange(c["nts"], device="cuda", dtype=torch.float32) * (DTW * c["sub"])
    ph = torch.stack([torch.sin(2 * np.pi * 15.0 * t), torch.cos(2 * np.pi * 15.0 * t)])
    d = torch.einsum("pt,pkn->tkn", ph, a)
    d[:, :3] *= 1e-7  # velocities beside stresses, in SI units
    return d.contiguous()


def _device_sets(tab, rtab):
    """Component-concatenated tables: an explosive source has the three normal stresses, the receivers
    all nine components on one table."""
    so = [len(tab) * min(max(k - 3, 0), 3) for k in range(10)]
    ro = [len(rtab) * k for k in range(10)]
    return (torch.from_numpy(np.tile(tab, 3)).cuda(), so, torch.from_numpy(np.tile(rtab, 9)).cuda(), ro)


def _propagator(c, seed, **kw):
    p = Propagator(c["nz"], c["nx"], c["ny"], c["nts"], c["sub"], c["pad"], D, D, D, _dts(c), **kw)
    planes = _planes(c, seed)
    torch.cuda.synchronize()  # the propagator reads the planes on a stream of its own
    p.set_medium(planes)
    return p


@functools.lru_cache(maxsize=None)
def _stream():
    """The stream that a modelling program queues its shots on."""
    return torch.cuda.Stream()


def _survey_axes(c):
    axes = tuple(H.Axis(n, -(FAT + c["pad"]) * D, D) for n in (c["nz"], c["nx"], c["ny"]))
    par = H.ParamObj(nts=c["nts"], dts=_dts(c), sub=c["sub"] // 2, nz=c["nz"], nx=c["nx"], ny=c["ny"], dz=D, dx=D,
                     dy=D, zPadMinus=c["pad"], zPadPlus=c["pad"], xPadMinus=c["pad"], xPadPlus=c["pad"],
                     yPad=c["pad"], fMax=25.0, blockSize=16, fat=FAT, alphaCos=0.99, mod_par=0, freeSurface=0)
    return axes, par


def _coords(c, st, seed):
    """Coordinates (z, x, y) of devices in the cells st, a quarter or a half cell off the grid points."""
    rng = np.random.default_rng(2000 + seed)
    q = 0.25 * rng.integers(0, 3, size=st.shape) * D
    return [(st[k] - FAT - c["pad"]) * D + q[k] for k in range(3)]


@functools.lru_cache(maxsize=1)
def _parameters(key):
    """The survey's parameters, which a program builds once for its grid (FdParam of the background)."""
    c = dict(key)
    axes, par = _survey_axes(c)
    return H.FdParam(torch.stack(_model(c, 0)).cpu().numpy(), axes, par)


def _grid_key(c):
    return tuple((k, c[k]) for k in ("nz", "nx", "ny", "pad", "nts", "sub"))


def _acquisition(c, seed):
    axes, par = _survey_axes(c)
    ax7 = H.grid_axes(*(a.n for a in axes), *(a.o for a in axes), *(a.d for a in axes))
    rec, src = _stations(c, seed)
    rc = _coords(c, rec, seed)
    srcs = [H.build_devices(*_coords(c, src[:, i:i + 1], seed + i), ax7, c["nts"], par) for i in range(src.shape[1])]
    return srcs, H.build_devices(*rc, ax7, c["nts"], par), rc


def _explosive(c):
    irr = np.zeros((9, 1, c["nts"]), np.float32)
    irr[3:6, 0] = _ricker(c)
    return irr


def _observed(c, seed):
    """Observed traces (9, nRec, nts) on the GPU: arrivals with the moveout of the direct wave."""
    rec, src = _stations(c, seed)
    r = torch.from_numpy(np.sqrt(((rec - src[:, :1]) ** 2).sum(0)) * D).cuda().float()
    t = torch.arange(c["nts"], device="cuda", dtype=torch.float32) * (DTW * c["sub"])
    delay = min(1.0 / 15.0, 0.35 * float(t[-1]))
    a = (np.pi * 15.0 * (t[None, :] - r[:, None] / 2400.0 - delay)) ** 2
    tr = (1 - 2 * a) * torch.exp(-a) / (1 + r[:, None] / D)
    amp = torch.tensor([1e-6] * 3 + [5.0] * 6, device="cuda")
    return amp[:, None, None] * tr[None]


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(case=c)
    if kind in ("forward", "adjoint", "batch"):
        # the batched launch takes each receiver component on its own table
        p = s["prop"] = _propagator(c, seed, **({"q2compat": 0} if kind == "batch" else {}),
                                    **({"free_surface": 1} if c.get("surface") else {}))
        p.set_stream(_stream())
        tabs, sig, rtab = _regular(c, seed)
        if kind == "batch":
            models = [[0 * g.T] * 3 + [g.T] * 3 + [0 * g.T] * 3 for g in sig]
            s["tables"] = p.batch_tables(models, [[t] * 7 for t in tabs], [rtab] * 7)
        else:
            sp, so, rp, ro = _device_sets(tabs[0], rtab)
            s["sets"] = (sp, so, rp, ro)
            if kind == "forward":
                s["src"] = torch.from_numpy(np.tile(sig[0], 3)).cuda()
                s["rec"] = torch.empty((c["nts"], ro[9]), device="cuda")
            else:
                s["src"] = torch.empty((c["nts"], so[9]), device="cuda")
                s["rec"] = _data(c, seed, len(rtab)).reshape(c["nts"], -1)
        torch.cuda.synchronize()
    elif kind in ("born_forward", "born_adjoint"):
        p = s["prop"] = _propagator(c, seed)
        tabs, sig, rtab = _regular(c, seed)
        empty = np.zeros((0, c["nts"]), np.float32)
        s["src9"] = [empty] * 3 + [np.ascontiguousarray(sig[0].T)] * 3 + [empty] * 3
        s["pos"] = ([tabs[0]] + [np.zeros(0, np.int64)] * 6, [rtab] * 7)
        if kind == "born_forward":
            s["pert"] = list(_perturbation(c, seed).cpu().numpy())
        else:
            s["data"] = [np.ascontiguousarray(x) for x in _data(c, seed, len(rtab)).permute(1, 2, 0).cpu().numpy()]
    elif kind == "operator":
        axes, par = _survey_axes(c)
        elastic = torch.stack(_model(c, seed)).cpu().numpy()
        srcs, rec, _ = _acquisition(c, seed)
        s["model"] = np.stack([_explosive(c)])
        s["data"] = np.zeros((c["shots"], 9, c["nrec"] ** 2, c["nts"]), np.float32)
        s["op"] = OP.nonlinearPropElasticShotsGpu_3D(s["model"], s["data"], elastic, par,
                                                     *[[d[g] for d in srcs] for g in range(7)],
                                                     *[[rec[g]] for g in range(7)])
    else:
        fd = _parameters(_grid_key(c))
        kw = {} if kind == "misfit" else dict(ckpt=c["store"], velocity=c["store"], segment=c["segment"])
        s["prob"] = F.FwiProblem(fd, device="cuda:0", **kw)
        srcs, rec, _ = _acquisition(c, seed)
        s["shot"] = F.make_shot(srcs[0], rec, list(_explosive(c)), None, "cuda:0")
        s["shot"].d_obs = F.time_major(_observed(c, seed))
        model = _model(c, seed)
        if kind == "misfit":
            s["prob"].shots.append(s["shot"])
            s["model"] = [m.requires_grad_(True) for m in model]
        else:
            s["planes"] = s["prob"].set_model(*model)
    return s


def _perturbation(c, seed):
    """Sparse reflectivity: eight perturbation planes, scaled as the medium planes are."""
    m = _planes(c, seed)
    keep = torch.rand(m.shape[1:], device="cuda", generator=_gen(seed, 21)) < 0.01
    f = (torch.rand((8,) + tuple(m.shape[1:]), device="cuda", generator=_gen(seed, 22)) - 0.5) * 0.1 * keep
    # the velocity terms take the density relative to the scaled buoyancy plane
    out = torch.empty_like(m)
    out[:3] = 2000.0 * f[:3] * m[:3]
    out[3] = f[3] * m[4]
    out[4] = f[4] * m[5]
    out[5:] = f[5:] * m[5:]
    return out


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind in ("forward", "adjoint"):
        state["prop"].nl_propagate_device(kind == "adjoint", *state["sets"], state["src"], state["rec"])
        return state["rec"] if kind == "forward" else state["src"]
    if kind == "batch":
        state["prop"].nl_forward_batch_device(state["tables"])
        return state["tables"].rec_sig
    if kind == "born_forward":
        return state["prop"].born_forward(state["src9"], state["pert"], *state["pos"])
    if kind == "born_adjoint":
        return state["prop"].born_adjoint(state["src9"], state["data"], *state["pos"])
    if kind == "operator":
        state["op"].forward(False, state["model"], state["data"])
        return state["data"]
    if kind == "misfit":
        m = state["model"]
        for x in m:
            x.grad = None
        loss = F.ElasticFwiMisfit.apply(*m, state["prob"])
        loss.backward()
        return [loss.detach()] + [x.grad for x in m]
    loss, grad8 = state["prob"].shot_misfit_and_gradient(state["shot"], state["planes"])
    return [loss, grad8]


# ----------------------------------------------------------------------------
# the work and the tolerance
# ----------------------------------------------------------------------------
def work(case):
    """Bytes and operations of one pass.  A fine step of a propagation reads its two levels and the
    medium and writes the new level (35 values a cell; 18 stencil derivatives, 234 operations); a
    coarse sample of Born scattering or imaging reads or writes nine fields, eight planes and the
    velocities of three samples."""
    c, kind = case, case["kind"]
    cells, n = _cells(c), c["nz"] * c["nx"] * c["ny"]
    steps = (c["nts"] - 1) * c["sub"]
    shots = c.get("shots", 1)
    traces = 4 * c["nts"] * 9 * c["nrec"] ** 2 * shots
    coarse = c["nts"] * cells * 4 * (9 + 16 + 9)
    if kind in ("forward", "adjoint", "operator"):
        passes, extra = shots, 0
    elif kind == "batch":
        # the medium is read once for all shots
        passes, extra = shots, -(shots - 1) * steps * cells * 32
    elif kind in ("born_forward", "born_adjoint"):
        passes, extra = 2, coarse + 32 * n
    elif kind == "misfit":
        passes, extra = 2, coarse + 24 * n
    else:
        # the source wavefield of all but the last segment is propagated twice
        blocks, seg = c["nts"] - 1, c["segment"]
        passes = 2 + max(0, blocks - seg) / blocks
        extra = coarse + 64 * n
    return {"bytes": passes * steps * cells * 140 + extra + traces, "flops": passes * steps * cells * 234}


def tolerance(case):
    """FP32 sums over a few hundred steps (up to 4e-7 off FP64 in the traces and images); some gradients
    store states and velocities in FP16 (1e-4 to 3e-4 off)."""
    if case["kind"] == "gradient" and case["store"] == "fp16":
        return {"rel": 1e-3, "max": 0.1}
    return {"rel": 1e-5, "max": 1e-3}


# ----------------------------------------------------------------------------
# the scheme in FP64, in plain torch
# ----------------------------------------------------------------------------
_COEF = [1.196289062541883, -0.079752604188901, 0.009570312506634, -6.975446437140719e-04]
_COEF = [float(np.float32(k / D)) for k in _COEF]  # the scheme's coefficients are FP32 numbers


def _der(f, dim, plus):
    """Eighth-order staggered derivative of f over the interior, forward (plus) or backward."""
    v = f
    for d in range(3):
        if d != dim:
            v = v.narrow(d, FAT, v.shape[d] - 2 * FAT)
    n = f.shape[dim] - 2 * FAT
    o = FAT + (1 if plus else 0)
    out = None
    for k in range(4):
        t = v.narrow(dim, o + k, n) - v.narrow(dim, o - k - 1, n)
        out = t.mul_(_COEF[0]) if k == 0 else out.add_(t, alpha=_COEF[k])
    return out


_Y, _X, _Z = 0, 1, 2


def _velocity_forces(s):
    """Stress divergence; s: the six stresses sxx, syy, szz, sxz, sxy, syz."""
    return (_der(s[0], _X, False).add_(_der(s[4], _Y, True)).add_(_der(s[3], _Z, True)),
            _der(s[4], _X, True).add_(_der(s[1], _Y, False)).add_(_der(s[5], _Z, True)),
            _der(s[3], _X, True).add_(_der(s[5], _Y, True)).add_(_der(s[2], _Z, False)))


def _strains(v):
    """dvx/dx, dvy/dy, dvz/dz and the xz, xy, yz pairs of the velocities."""
    return (_der(v[0], _X, True), _der(v[1], _Y, True), _der(v[2], _Z, True),
            _der(v[0], _Z, False).add_(_der(v[2], _X, False)), _der(v[0], _Y, False).add_(_der(v[1], _X, False)),
            _der(v[2], _Y, False).add_(_der(v[1], _Z, False)))


def _inner(f):
    return f[FAT:-FAT, FAT:-FAT, FAT:-FAT]


class _Scheme:
    def __init__(self, c, planes):
        self.c, self.m = c, [p.double() for p in planes]
        self.mi = [_inner(p) for p in self.m]
        self.surface = bool(c.get("surface"))
        self.shape = (c["ny"], c["nx"], c["nz"])
        pad, big = c["pad"], 1 << 30
        taper = np.ones(pad + 1)
        for i in range(pad):
            taper[i] = np.float32(np.float32(0.99) + (1.0 - np.float32(0.99)) * np.cos(
                float(np.float32(np.pi / (1.0 * pad) * (pad - i)))))
        dist = []
        for n, top in zip(self.shape, (False, False, self.surface)):
            i = torch.arange(n - 2 * FAT, device="cuda")
            low = torch.full_like(i, big) if top else i
            dist.append(torch.minimum(low, (n - 2 * FAT - 1) - i))
        d = torch.minimum(torch.minimum(dist[0][:, None, None], dist[1][None, :, None]), dist[2][None, None, :])
        self.G = torch.from_numpy(taper).cuda()[d.clamp(max=pad)]
        self.Gfull = torch.ones(self.shape, device="cuda", dtype=torch.float64)
        _inner(self.Gfull).copy_(self.G)
        # time interpolation between a coarse sample and the next
        ntw = (c["nts"] - 1) * c["sub"] + 1
        sc = 1.0 / np.sqrt(float(np.float32(ntw) / np.float32(c["nts"])))
        left = [float(np.float32(1.0 - 1.0 * i / c["sub"])) for i in range(c["sub"] + 1)]
        self.wl = [float(np.float32(a * sc)) for a in left]
        self.wr = [float(np.float32(float(np.float32(1.0 - a)) * sc)) for a in left]

    def zeros(self, k=9):
        return [torch.zeros(self.shape, device="cuda", dtype=torch.float64) for _ in range(k)]

    def update(self, old, cur, sign=1.0, transpose=False, extra=None):
        """Advance the old level in place by one fine step of the current one; transpose: the exact
        adjoint of the forward step; extra: a secondary source added before the sponge."""
        m, mi = self.m, self.mi
        if transpose:
            q = [cur[k] * m[k] for k in range(3)]
            t = cur[3] + cur[4] + cur[5]
            q += [m[3] * cur[k] + m[4] * (t - cur[k]) for k in (3, 4, 5)]
            del t
            q += [cur[6] * m[5], cur[7] * m[6], cur[8] * m[7]]
            cur, sign = q, -1.0
        f, e = _velocity_forces(cur[3:]), _strains(cur[:3])
        if transpose:
            up = list(f) + list(e)
        else:
            tr = e[0] + e[1] + e[2]
            up = [mi[k] * f[k] for k in range(3)]
            up += [mi[3] * e[k] + mi[4] * (tr - e[k]) for k in range(3)]
            up += [mi[5] * e[3], mi[6] * e[4], mi[7] * e[5]]
            del tr
        del f, e
        for k in range(9):
            o = _inner(old[k])
            v = o * self.G
            v.add_(up[k], alpha=sign)
            if extra is not None:
                v.add_(extra[k])
            o.copy_(v.mul_(self.G))

    def inject(self, lev, tabs, sig, its, k):
        for i, pos in tabs.items():
            add = sig[i][its] * self.wl[k] + sig[i][its + 1] * self.wr[k]
            lev[i].view(-1).index_add_(0, pos, add * self.Gfull.view(-1)[pos])

    def record(self, lev, tabs, out, its, k):
        for i, pos in tabs.items():
            v = lev[i].view(-1)[pos]
            out[i][its] += v * self.wl[k]
            out[i][its + 1] += v * self.wr[k]

    def free_surface(self, new, cur, sign=1.0):
        if not self.surface:
            return
        zs = FAT
        sl = lambda a: a[FAT:-FAT, FAT:-FAT]  # noqa: E731
        e = [t[:, :, 0] for t in _strains(cur[:3])[:3]]
        lam, l2m = sl(self.m[4])[:, :, zs], sl(self.m[3])[:, :, zs]
        corr = sign * self.G[:, :, 0] * (-lam * e[2] - lam * lam / l2m * (e[0] + e[1]))
        sl(new[SXX])[:, :, zs] += corr
        sl(new[SYY])[:, :, zs] += corr
        zz = sl(new[SZZ])
        zz[:, :, zs] = 0
        for k in range(1, FAT + 1):
            zz[:, :, zs - k] = -zz[:, :, zs + k]
        for r in range(FAT + 1):
            for f in (SXZ, SYZ):
                sl(new[f])[:, :, r] = -sl(new[f])[:, :, 2 * FAT + 1 - r]
            sl(new[VZ])[:, :, r] = 0

    def traces(self, tabs):
        return {i: torch.zeros((self.c["nts"], len(p)), device="cuda", dtype=torch.float64) for i, p in tabs.items()}

    def forward(self, stabs, sig, rtabs, velocity=None):
        """Recorded traces of the nonlinear forward; velocity: the decimated source velocities per
        coarse sample, accumulated when given."""
        a, b, out = self.zeros(), self.zeros(), self.traces(rtabs)
        for its in range(self.c["nts"] - 1):
            for it2 in range(1, self.c["sub"] + 1):
                self.update(a, b)
                self.inject(a, stabs, sig, its, it2 - 1)
                self.free_surface(a, b)
                self.record(a, rtabs, out, its, it2)
                if velocity is not None:
                    for k in range(3):
                        velocity[its][k].add_(a[k], alpha=self.wl[it2])
                        velocity[its + 1][k].add_(a[k], alpha=self.wr[it2])
                a, b = b, a
        return out

    def reversed_adjoint(self, rtabs, data, stabs):
        a, b, out = self.zeros(), self.zeros(), self.traces(stabs)
        for its in reversed(range(self.c["nts"] - 1)):
            for it2 in reversed(range(self.c["sub"])):
                self.update(a, b, -1.0)
                self.inject(a, rtabs, data, its, it2 + 1)
                self.record(a, stabs, out, its, it2)
                a, b = b, a
        return out

    def _velocity_terms(self, V, t):
        e = _strains(V[t])
        inv = float(np.float32(1.0 / (2.0 * float(np.float32(_dts(self.c))))))
        # the sample before the first and the one after the last are zero
        td = [torch.zeros_like(e[0]) for _ in range(3)]
        for k in range(3):
            if t > 0:
                td[k].add_(_inner(V[t - 1][k]), alpha=inv)
            if t + 1 < len(V):
                td[k].sub_(_inner(V[t + 1][k]), alpha=inv)
        return e, td

    def secondary(self, V, t, pert):
        """Secondary source of coarse sample t (interior); the yz term takes the xz pair."""
        e, td = self._velocity_terms(V, t)
        p = [_inner(x) for x in pert]
        div = e[0] + e[1] + e[2]
        return [p[0] * td[0], p[1] * td[1], p[2] * td[2]] + [p[3] * div + 2 * p[4] * e[k] for k in range(3)] + \
            [p[5] * e[3], p[6] * e[4], p[7] * e[3]]

    def born_forward(self, stabs, sig, pert, rtabs):
        V = [self.zeros(3) for _ in range(self.c["nts"])]
        self.forward(stabs, sig, {}, V)
        a, b, out = self.zeros(), self.zeros(), self.traces(rtabs)
        nxt = self.secondary(V, 0, pert)
        for its in range(self.c["nts"] - 1):
            prv, nxt = nxt, self.secondary(V, its + 1, pert)
            for it2 in range(1, self.c["sub"] + 1):
                ss = [p * self.wl[it2 - 1] + q * self.wr[it2 - 1] for p, q in zip(prv, nxt)]
                self.update(a, b, extra=ss)
                self.record(a, rtabs, out, its, it2)
                a, b = b, a
        return out

    def _image(self, V, t, A, pert):
        e, td = self._velocity_terms(V, t)
        A = [_inner(x) for x in A]
        p = [_inner(x) for x in pert]
        for k in range(3):
            p[k].addcmul_(A[k], td[k])
        p[3].addcmul_(A[3] + A[4] + A[5], e[0] + e[1] + e[2])
        for k in range(3):
            p[4].addcmul_(A[3 + k], e[k], value=2.0)
        p[5].addcmul_(A[6], e[3])
        p[6].addcmul_(A[7], e[4])
        p[7].addcmul_(A[8], e[3])

    def born_adjoint(self, V, rtabs, data):
        """The eight image planes of the data, V the decimated source velocities."""
        a, b, pert = self.zeros(), self.zeros(), self.zeros(8)
        right = self.zeros()
        for its in reversed(range(self.c["nts"] - 1)):
            left = self.zeros()
            for it2 in reversed(range(self.c["sub"])):
                self.update(a, b, transpose=True)
                self.inject(a, rtabs, data, its, it2 + 1)
                for k in range(9):
                    left[k].add_(a[k], alpha=self.wl[it2])
                    right[k].add_(a[k], alpha=self.wr[it2])
                a, b = b, a
            self._image(V, its + 1, right, pert)
            right = left
        self._image(V, 0, right, pert)
        return pert


# staggering of the seven grids (z, x, y half cells) in the order centre, x, y, z, xz, xy, yz
_STAGGER = [(0, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 0), (1, 1, 0), (0, 1, 1), (1, 0, 1)]


def _trilinear(c, coords, receivers):
    """Per component: regular points, and per device its eight slots into them and weights.  The sxz
    receivers are read at the points of the z grid, as the reference does."""
    o = -(FAT + c["pad"]) * D
    per = []
    for st in _STAGGER:
        w, base = [], []
        for k in range(3):
            u = (np.asarray(coords[k], dtype=np.float64) - (o - 0.5 * D * st[k])) / D
            base.append(np.floor(u).astype(np.int64))
            w.append(u - base[k])
        idx, wt = [], []
        for j in (0, 1):
            for i in (0, 1):
                for k in (0, 1):
                    idx.append(((base[2] + j) * c["nx"] + base[1] + i) * c["nz"] + base[0] + k)
                    wt.append((w[0] if k else 1 - w[0]) * (w[1] if i else 1 - w[1]) * (w[2] if j else 1 - w[2]))
        idx, wt = np.stack(idx, 1), np.stack(wt, 1)
        u, first, inv = np.unique(idx.ravel(), return_index=True, return_inverse=True)
        order = np.argsort(first)
        rank = np.empty(len(u), np.int64)
        rank[order] = np.arange(len(u))
        per.append((u[order], rank[inv.reshape(-1)].reshape(idx.shape), wt))
    tabs, slots, wts = {}, {}, {}
    for k in range(9):
        u, s, w = per[COMP_GRID[k]]
        if receivers and k == SXZ:
            u = per[3][0][:len(u)]
        tabs[k], slots[k], wts[k] = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (u, s, w))
    return tabs, slots, wts


def _to_devices(reg, slots, wts):
    """Regular traces (nts, points) to devices (devices, nts), per component."""
    return {k: (reg[k][:, slots[k]] * wts[k]).sum(2).t() for k in reg}


def _to_points(dev, tabs, slots, wts):
    out = {}
    for k in tabs:
        nts = dev[k].shape[1]
        r = torch.zeros((nts, len(tabs[k])), device="cuda", dtype=torch.float64)
        up = dev[k].t()[:, :, None] * wts[k]
        out[k] = r.index_add_(1, slots[k].reshape(-1), up.reshape(nts, -1))
    return out


def _scaled_explosive(c, sch, tabs, slots, wts):
    """The explosive source's regular signals scaled by the medium, per normal stress."""
    w = torch.from_numpy(_ricker(c)).cuda().double()[None, :]
    reg = _to_points({k: w for k in (3, 4, 5)}, {k: tabs[k] for k in (3, 4, 5)}, slots, wts)
    f = (sch.m[3] + 2 * sch.m[4]).view(-1)[tabs[3]] * float(np.float32(1.0 / D ** 3))
    return {k: reg[k] * f for k in reg}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("forward", "adjoint", "batch", "born_forward", "born_adjoint"):
        sch = _Scheme(c, _planes(c, seed))
        tabs, sig, rtab = _regular(c, seed)
        R = torch.from_numpy(rtab).cuda()
        rt = {k: R for k in range(9)}
        st = [{k: torch.from_numpy(t).cuda() for k in (3, 4, 5)} for t in tabs]
        sg = [{k: torch.from_numpy(g).cuda().double() for k in (3, 4, 5)} for g in sig]
        if kind == "forward":
            d = sch.forward(st[0], sg[0], rt)
            return torch.cat([d[k] for k in range(9)], 1)
        if kind == "batch":
            d = [sch.forward(a, b, rt) for a, b in zip(st, sg)]
            return torch.cat([x[k] for k in range(9) for x in d], 1)
        if kind == "born_forward":
            d = sch.born_forward(st[0], sg[0], list(_perturbation(c, seed).double()), rt)
            return [d[k].t().contiguous() for k in range(9)]
        data = _data(c, seed, len(rtab)).double()
        dd = {k: data[:, k] for k in range(9)}
        if kind == "adjoint":
            d = sch.reversed_adjoint(rt, dd, st[0])
            return torch.cat([d[k] for k in (3, 4, 5)], 1)
        V = [sch.zeros(3) for _ in range(c["nts"])]
        sch.forward(st[0], sg[0], {}, V)
        return sch.born_adjoint(V, rt, dd)
    rho, lam, mu = _model(c, seed)
    sch = _Scheme(c, _planes64(rho, lam, mu) if kind != "gradient" else _planes(c, seed))
    rec, src = _stations(c, seed)
    rtab, rslot, rw = _trilinear(c, _coords(c, rec, seed), True)
    shots = []
    for i in range(src.shape[1]):
        t = _trilinear(c, _coords(c, src[:, i:i + 1], seed + i), False)
        shots.append(({k: t[0][k] for k in (3, 4, 5)}, _scaled_explosive(c, sch, *t)))
    if kind == "operator":
        out = []
        for st, sg in shots:
            d = _to_devices(sch.forward(st, sg, rtab), rslot, rw)
            out.append(torch.stack([d[k] for k in range(9)]))
        return torch.stack(out)
    V = [sch.zeros(3) for _ in range(c["nts"])]
    d = _to_devices(sch.forward(*shots[0], rtab, V), rslot, rw)
    obs = _observed(c, seed).double()
    res = {k: d[k] - obs[k] for k in range(9)}
    loss = 0.5 * sum(float((r * r).sum()) for r in res.values())
    g8 = sch.born_adjoint(V, rtab, _to_points(res, rtab, rslot, rw))
    if kind == "gradient":
        return [torch.tensor(loss, dtype=torch.float64), torch.stack(g8)]

    def spread(f, dim):
        """The transpose of the perturbation's staggering: the mean of a cell and the next."""
        n = f.shape[dim]
        return torch.cat([0.5 * (f.narrow(dim, 0, n - 1) + f.narrow(dim, 1, n - 1)), f.narrow(dim, n - 1, 1)], dim)

    two = 2.0 * float(np.float32(DTW))
    g = [g8[k] * sch.m[k] for k in range(3)] + [x * two for x in g8[3:]]
    drho = spread(g[0], 1) + spread(g[1], 0) + spread(g[2], 2)
    dmu = g[4] + spread(spread(g[5], 2), 1) + spread(spread(g[6], 0), 1) + spread(spread(g[7], 2), 0)
    return [torch.tensor(loss, dtype=torch.float64), drho, g[3], dmu]
