"""What a user of this framework has it do, as measurable cases.

A case is one pass of a user's program over a model, an ensemble or a
differentiable rollout that is set up and running: ``steps`` iterations of the
run loop, then the updated state read back (FP64 fields as float64, the FP32
form's as the float32 that the history stores), or a rollout with its
gradient. Sizes are those of the framework's own configurations and defaults
(``Param``'s 40 x 40, eulerpsi 256^2, rsw 512^2, qg 1024^2 and 4096^2, the
256-member ensemble, the 512^2 adjoint), and generic odd and ragged ones.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch
import torch.utils.checkpoint

import fluids2d_gb300 as f2d
from fluids2d_gb300._lib import check, lib
from fluids2d_gb300.adjoint import rollout

HALO = 3

# the fields that are read back: the prognostic variables and what the
# elliptic solve of the diagnostics gives
FIELDS = {
    "eulerpsi": ("omega", "psi"),
    "qg": ("pv", "psi"),
    "rsw": ("h", "u.x", "u.y"),
    "euler": ("u.x", "u.y", "p"),
    "boussinesq": ("b", "u.x", "u.y", "p"),
}


def listed():
    return [
        # the default model at the default size of Param: an interactive
        # script that plots every few iterations; launches and latency count
        _case("euler_40_fp64", "euler", 40, 40, steps=5),
        # the vortex experiment of the configurations, in the reference's
        # own precision
        _case("eulerpsi_256_fp64", "eulerpsi", 256, 256, steps=5),
        # a basin of odd size with islands, no-slip walls and a passive tracer
        _case("eulerpsi_501x387_fp32_tracer", "eulerpsi", 501, 387, precision="fp32", steps=5,
              islands=3, noslip=True, tracer=True),
        # shallow water in an x-periodic channel with islands
        _case("rsw_512_fp64", "rsw", 512, 512, steps=5, islands=3, xperiodic=True),
        # shallow water in a large closed basin, FP32
        _case("rsw_1500x1030_fp32", "rsw", 1500, 1030, precision="fp32", steps=5, islands=3),
        # QG turbulence on a beta-plane with islands: the FP64 Helmholtz solve
        _case("qg_1024_fp64", "qg", 1024, 1024, steps=2, islands=20),
        # the largest single model
        _case("qg_4096_fp32", "qg", 4096, 4096, precision="fp32", steps=5, islands=20),
        # the momentum-pressure form: the Neumann pressure solve
        _case("euler_512_fp64", "euler", 512, 512, steps=3, islands=3),
        # stratified flow in a wide x-periodic channel, FP32
        _case("boussinesq_640x352_fp32", "boussinesq", 640, 352, precision="fp32", steps=3,
              islands=2, xperiodic=True),
        # a twin-experiment-sized ensemble of uneven members, FP64
        _case("ensemble_24_fp64", "eulerpsi", 160, 160, kind="ensemble", members=24, steps=2,
              islands=2),
        # the 256-member ensemble of 64^2 to 512^2 basins
        _case("ensemble_256_fp32", "eulerpsi", 512, 512, kind="ensemble", members=256,
              precision="fp32", steps=4, islands=4),
        # gradient of a rollout with respect to its initial vorticity
        _case("adjoint_512_fp64", "eulerpsi", 512, 512, kind="adjoint", steps=20),
    ]


def _case(name, model, nx, ny, kind="model", precision="fp64", steps=5, islands=0,
          xperiodic=False, noslip=False, tracer=False, members=0):
    return dict(name=name, kind=kind, model=model, nx=nx, ny=ny, precision=precision,
                steps=steps, islands=islands, xperiodic=xperiodic, noslip=noslip,
                tracer=tracer, members=members)


def _spread(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["model"] * 8 + ["ensemble"] * 2 + ["adjoint"])
    if kind == "ensemble":
        n = _spread(rng, 64, 512)
        c = _case("", "eulerpsi", n, n, kind=kind, members=_spread(rng, 4, 64),
                  precision=rng.choice(["fp64", "fp32"]), steps=2, islands=rng.randint(0, 4))
    elif kind == "adjoint":
        nx = _spread(rng, 64, 512)
        c = _case("", "eulerpsi", nx, min(512, int(nx * rng.uniform(0.6, 1.6))), kind=kind,
                  steps=rng.randint(8, 20))
    else:
        model = rng.choice(["eulerpsi", "qg", "rsw", "euler", "boussinesq"])
        precision = rng.choice(["fp64", "fp32"])
        small = model in ("euler", "boussinesq")
        lo, hi = (40, 640) if small else (64, 1536)
        nx = _spread(rng, lo, hi)
        ny = min(hi, max(lo, int(nx * rng.uniform(0.6, 1.6))))
        c = _case("", model, nx, ny, precision=precision, steps=rng.randint(2, 4),
                  islands=rng.randint(0, 3 if small else 6), noslip=rng.random() < 0.25,
                  xperiodic=model in ("rsw", "euler", "boussinesq") and rng.random() < 0.5,
                  tracer=model in ("eulerpsi", "qg") and rng.random() < 0.3)
    del c["name"]
    return c


# ---- inputs, from the seed alone --------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _sizes(case, rng):
    """Grid sizes of the members of an ensemble: from an eighth of the
    largest to the largest, odd ones among them."""
    top = case["nx"]
    return [(int(rng.integers(max(24, top // 8), top + 1)),) * 2 for _ in range(case["members"])]


def _coords(nx, ny, which="c"):
    sx = 0.5 if which in ("c", "y") else 0.0
    sy = 0.5 if which in ("c", "x") else 0.0
    i = torch.arange(nx + 2 * HALO, device="cuda", dtype=torch.float64) - HALO + sx
    j = torch.arange(ny + 2 * HALO, device="cuda", dtype=torch.float64) - HALO + sy
    return (i / nx)[None, :], (j / ny)[:, None]


def _mask(nx, ny, islands, xperiodic, rng, small=False):
    msk = torch.zeros((ny + 2 * HALO, nx + 2 * HALO), dtype=torch.int8, device="cuda")
    msk[HALO:-HALO, slice(None) if xperiodic else slice(HALO, -HALO)] = 1
    x, y = _coords(nx, ny)
    lo, hi = (0.01, 0.04) if small else (0.03, 0.08)
    for _ in range(islands):
        xc, yc = rng.uniform(0.12, 0.88, 2)
        r = rng.uniform(lo, hi)
        msk[(x - xc) ** 2 + (y - yc) ** 2 < r * r] = 0
    return msk


def _vortices(x, y, n, radius, rng):
    w = 0.0
    for _ in range(n):
        xc, yc = rng.uniform(radius, 1 - radius, 2)
        gx, gy = (torch.exp(-(a - c) ** 2 / (2 * radius ** 2)) for a, c in ((x, xc), (y, yc)))
        w = w + (1.0 if rng.uniform() < 0.5 else -1.0) * gx * gy
    return w


def _turbulence(nx, ny, seed):
    """Unit-variance field of random phases at wavenumbers 4 to 32."""
    g = _generator(seed)
    k = torch.hypot(torch.fft.rfftfreq(nx, 1.0 / nx, device="cuda", dtype=torch.float64)[None, :],
                    torch.fft.fftfreq(ny, 1.0 / ny, device="cuda", dtype=torch.float64)[:, None])
    phase = torch.rand(k.shape, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
    spec = torch.polar(((k >= 4) & (k <= 32)).double(), phase)
    q = torch.fft.irfft2(spec, s=(ny, nx))
    q = (q - q.mean()) / q.std()
    return torch.nn.functional.pad(q, (HALO,) * 4)


def _periodic(a):
    a[:, :HALO] = a[:, -2 * HALO:-HALO]
    a[:, -HALO:] = a[:, HALO:2 * HALO]


def _inputs(case, seed, nx=None, ny=None, member=0):
    """{"msk", fields, parameters} of one model, as GPU tensors."""
    nx, ny = nx or case["nx"], ny or case["ny"]
    model, per = case["model"], case["xperiodic"]
    rng = np.random.default_rng([int(seed), member])
    # the islands are the basin's, not the seed's: the same for every seed
    # but drawn anew for every member
    msk = _mask(nx, ny, case["islands"], per, np.random.default_rng([91, member, nx, ny]),
                small=model == "qg")
    x, y = _coords(nx, ny)
    dx, dy = 1.0 / nx, 1.0 / ny
    area = dx * dy
    par, fields = {}, {}
    if model == "eulerpsi":
        fields["omega"] = _vortices(x, y, 8, 0.05, rng) * msk * area
    elif model == "qg":
        par = dict(f0=50.0, beta=1.0, g=1.0, H=1.0)
        fields["pv"] = (_turbulence(nx, ny, seed) + (y - 0.5)) * area * msk
        xv, yv = _coords(nx, ny, "v")
        par["f"] = (yv - 0.5) * area + 0 * xv
    elif model == "rsw":
        par = dict(f0=1.0, g=1.0, H=1.0)
        noise = torch.randn(msk.shape, generator=_generator(seed), device="cuda",
                            dtype=torch.float64)
        bump = torch.exp(-((x - rng.uniform(0.4, 0.6)) ** 2 + (y - 0.5) ** 2) / 0.02)
        fields["h"] = (1.0 + 0.1 * bump + 1e-3 * noise) * msk * area
    else:
        psi = _vortices(*_coords(nx, ny, "v"), 6, 0.08, rng) * (0.5 * area)
        ux, uy = torch.zeros_like(psi), torch.zeros_like(psi)
        ux[:-1, :] = -(psi[1:, :] - psi[:-1, :])
        uy[:, :-1] = psi[:, 1:] - psi[:, :-1]
        scale = 0.05 * float(torch.maximum(ux.abs().max(), uy.abs().max()))
        g = _generator(seed)
        for a in (ux, uy):
            a += scale * torch.randn(a.shape, generator=g, device="cuda", dtype=torch.float64)
        ux[:, 1:] *= msk[:, 1:] * msk[:, :-1]
        ux[:, 0] = 0
        uy[1:, :] *= msk[1:, :] * msk[:-1, :]
        uy[0, :] = 0
        fields.update({"u.x": ux, "u.y": uy})
        if model == "boussinesq":
            umax = float(torch.maximum(ux.abs().max(), uy.abs().max()))
            amp = 0.1 * umax ** 2 / (dy * dx ** 2)
            b = 0.5 * (y - 0.5) + 0 * x
            for _ in range(2):
                x0, y0 = rng.uniform(0.2, 0.8), rng.uniform(0.2, 0.5)
                b = b + rng.choice([-1.0, 1.0]) * torch.exp(
                    -((x - x0) ** 2 + (y - y0) ** 2) / rng.uniform(0.06, 0.12) ** 2)
            fields["b"] = amp * b * msk
    if case["tracer"]:
        fields["q"] = (0.5 * x + _vortices(x, y, 3, 0.1, rng)) * msk
    if per:
        for a in fields.values():
            _periodic(a)
    return dict(msk=msk, fields=fields, par=par)


def _cfl(model):
    return {"euler": 0.5, "boussinesq": 0.5, "eulerpsi": 0.8}.get(model, 0.9)


def _param(case, par):
    p = f2d.Param()
    p.model, p.nx, p.ny = case["model"], case["nx"], case["ny"]
    p.precision, p.xperiodic = case["precision"], case["xperiodic"]
    p.noslip = True if case["noslip"] else None
    p.tracer = "q" if case["tracer"] else None
    p.cfl = _cfl(case["model"])
    p.tend, p.maxite = 1e300, 10 ** 12
    for k in ("f0", "beta", "g", "H"):
        if k in par:
            setattr(p, k, par[k])
    return p


# ---- preparation and the pass -----------------------------------------------

def prepare(case, seed):
    if case["kind"] == "ensemble":
        return _prepare_ensemble(case, seed)
    inp = _inputs(case, seed)
    m = f2d.Model(_param(case, inp["par"]))
    m.mesh.msk[:] = inp["msk"].cpu().numpy()
    m.mesh.finalize()
    if "f" in inp["par"]:
        m.mesh.f = inp["par"]["f"].cpu().numpy()
    if case["kind"] == "adjoint":
        # a time step half of the initial flow's CFL limit, and a misfit's
        # gradient of the size of the vorticity
        w0 = inp["fields"]["omega"]
        m.state.omega[:] = w0.cpu().numpy()
        m.integrator.diag(m.state)
        m.set_dt()
        lam = _inputs(case, seed + 100003)["fields"]["omega"]
        return dict(case=case, m=m, w0=w0.requires_grad_(True), lam=lam, dt=0.5 * m.time.dt)
    s = m.state
    for k, v in inp["fields"].items():
        a = getattr(getattr(s, k[0]), k[2]) if "." in k else getattr(s, k)
        a[:] = v.cpu().numpy()
    m.integrator.diag(s)
    m.sync()
    names = FIELDS[case["model"]] + (("q",) if case["tracer"] else ())
    dtype = torch.float32 if case["precision"] == "fp32" else torch.float64
    out = {k: torch.empty(m.mesh.shape, dtype=dtype, pin_memory=True) for k in names}
    return dict(case=case, m=m, out=out)


def _prepare_ensemble(case, seed):
    sizes = _sizes(case, np.random.default_rng([17, case["members"], case["nx"]]))
    members = [_inputs(dict(case, islands=b % (case["islands"] + 1)), seed, nx, ny, b)
               for b, (nx, ny) in enumerate(sizes)]
    e = f2d.Ensemble(_param(case, {}), sizes, [c["msk"].cpu().numpy() for c in members])
    e.set_fields("omega", torch.cat([c["fields"]["omega"].ravel() for c in members]).cpu().numpy())
    e.diag()
    e.sync()
    n = e.packed_size()
    host = {k: torch.empty(n, dtype=torch.float64, pin_memory=True) for k in ("omega", "psi")}
    out = host if case["precision"] == "fp64" else \
        {k: torch.empty(n, dtype=torch.float32) for k in host}
    return dict(case=case, e=e, host=host, out=out)


def run(state):
    case = state["case"]
    if case["kind"] == "adjoint":
        wT = rollout(state["m"], state["w0"], case["steps"], state["dt"], every=10)
        (g,) = torch.autograd.grad((wT * state["lam"]).sum(), state["w0"])
        return {"omega": wT.detach(), "gradient": g}
    if case["kind"] == "ensemble":
        e = state["e"]
        e.run(case["steps"])
        for k, a in state["host"].items():
            check(lib().f2d_ensemble_fields_get(e._h, k.encode(), ctypes.c_void_p(a.data_ptr()),
                                                1))
        e.sync()
        if case["precision"] == "fp32":
            for k, a in state["host"].items():
                state["out"][k].copy_(a)
        return state["out"]
    m = state["m"]
    m.advance(case["steps"])
    get = lib().f2d_field_get_f32 if case["precision"] == "fp32" else lib().f2d_field_get
    for k, a in state["out"].items():
        name = "tracer" if k == "q" else k
        check(get(m._h, name.encode(), ctypes.c_void_p(a.data_ptr())))
    return state["out"]


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    """Bytes: per stage, every prognostic field and the solve's solution read
    once and written once, the mask read once; and the fields read back.
    Operations: the reconstructions and the update of the stage, and one
    V-cycle-sized pass (about 60 operations a point) for its solve."""
    word = 8 if case["precision"] == "fp64" else 4
    model, stages = case["model"], 3 * case["steps"]
    nprog = {"eulerpsi": 1, "qg": 1, "rsw": 3, "euler": 2, "boussinesq": 3}[model] + case["tracer"]
    solve = model != "rsw"
    nout = len(FIELDS[model]) + case["tracer"]
    if case["kind"] == "ensemble":
        points = sum((nx + 6) * (ny + 6) for nx, ny in
                     _sizes(case, np.random.default_rng([17, case["members"], case["nx"]])))
    else:
        points = (case["nx"] + 6) * (case["ny"] + 6)
    per_stage = 2 * word * nprog + 1 + (16 if solve else 0)
    flops = 2 * 90 * nprog + (60 if solve else 0)
    passes = 1
    if case["kind"] == "adjoint":  # forward, and twice that for the gradient
        passes = 3
    return {"bytes": float(points * (passes * stages * per_stage + nout * word)),
            "flops": float(points * passes * stages * flops)}


# ---- the same in plain FP64 torch -------------------------------------------

def exact(case, seed):
    cells = case["nx"] * case["ny"] * max(1, case["members"])
    if cells > 2_000_000:
        return None
    if case["kind"] == "ensemble":
        sizes = _sizes(case, np.random.default_rng([17, case["members"], case["nx"]]))
        parts = {"omega": [], "psi": []}
        for b, (nx, ny) in enumerate(sizes):
            c = dict(case, islands=b % (case["islands"] + 1), nx=nx, ny=ny)
            s = _Exact(c, _inputs(c, seed, nx, ny, b)).steps(case["steps"])
            for k, v in parts.items():
                v.append(s[k].ravel())
        return {k: torch.cat(v) for k, v in parts.items()}
    inp = _inputs(case, seed)
    ex = _Exact(case, inp)
    if case["kind"] == "adjoint":
        ex.diag()
        dt = 0.5 * ex.cfl_dt()
        lam = _inputs(case, seed + 100003)["fields"]["omega"]
        w0 = inp["fields"]["omega"].clone().requires_grad_(True)
        w = w0
        for _ in range(case["steps"]):
            w = torch.utils.checkpoint.checkpoint(ex.eulerpsi_step, w, dt, use_reentrant=False)
        (g,) = torch.autograd.grad((w * lam).sum(), w0)
        return {"omega": w.detach(), "gradient": g}
    s = ex.steps(case["steps"])
    names = FIELDS[case["model"]] + (("q",) if case["tracer"] else ())
    return {k: s[k] for k in names}


def _shift(a, n):
    """a at flat index + n."""
    return torch.roll(a.reshape(-1), -n).view_as(a)


def _weno5(a, b, c, d, e):
    q1 = a / 3 - 7 * b / 6 + 11 * c / 6
    q2 = -b / 6 + 5 * c / 6 + d / 3
    q3 = c / 3 + 5 * d / 6 - e / 6
    b1 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b2 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b3 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    tau = (b1 - b3).abs()
    w1, w2, w3 = (g * (1 + tau / (b + 1e-16)) for g, b in ((0.1, b1), (0.6, b2), (0.3, b3)))
    return (w1 * q1 + w2 * q2 + w3 * q3) / (w1 + w2 + w3)


def _weno3(a, b, c):
    b1, b2 = (b - a) ** 2, (c - b) ** 2
    tau = (b2 - b1).abs()
    w1, w2 = (1 + tau / (b1 + 1e-14)) / 3, 2 * (1 + tau / (b2 + 1e-14)) / 3
    return (w1 * (-0.5 * a + 1.5 * b) + w2 * 0.5 * (b + c)) / (w1 + w2)


def _reconstruct(order, U, w):
    """The upwind WENO value of the six-point window w at the order of each
    point (0: none)."""
    up = U > 0
    a, b, c, d, e = (torch.where(up, w[k], w[5 - k]) for k in range(5))
    r = torch.where(order > 4, _weno5(a, b, c, d, e), _weno3(b, c, d))
    return torch.where(order > 2, r, torch.where(order > 0, c, torch.zeros_like(c)))


def _orders(m, s):
    """Stencil order from the wet neighbours along the flat shift s (towards
    lower indices if s > 0)."""
    n, flat = m.numel(), m.reshape(-1).long()
    i = torch.arange(n, device=m.device)

    def at(k):
        return torch.where((i + k >= 0) & (i + k < n), torch.roll(flat, -k), -9)

    s2 = flat + at(-s)
    s4 = s2 + at(-2 * s) + at(s)
    s6 = s4 + at(-3 * s) + at(2 * s)
    o = torch.where(s6 == 6, 6, torch.where(s4 == 4, 4, torch.where(s2 == 2, 2, 0)))
    return o.view_as(m)


class _Elliptic:
    """The masked 5-point operator in FP64: conjugate gradients with the fast
    transform solve of the whole rectangle (Dirichlet vertices or Neumann
    cells, periodic in x or closed) as the preconditioner."""

    def __init__(self, wet, box, cx, cy, main, neumann, per):
        self.box, self.neumann, self.per, self.main = box, neumann, per, main
        self.wet = wet[box].double()
        w = self.wet
        self.faces = [(1, cx, (w * torch.roll(w, 1, 1)) if neumann else None),
                      (0, cy, (w * torch.roll(w, 1, 0)) if neumann else None)]
        if neumann:
            self.faces[1][2][0, :] = 0
            if not per:
                self.faces[0][2][:, 0] = 0
        self.c = (cx, cy)
        n = [w.shape[0], w.shape[1]]
        ext = [2 * n[0] if neumann else 2 * (n[0] + 1), n[1] if per else
               (2 * n[1] if neumann else 2 * (n[1] + 1))]
        lam = []
        for k, L in enumerate(ext):
            f = torch.arange(L, device=w.device, dtype=torch.float64)
            lam.append((cy if k == 0 else cx) * 2 * (torch.cos(2 * math.pi * f / L) - 1))
        sym = lam[0][:, None] + lam[1][None, :ext[1] // 2 + 1] - main
        if main == 0:  # the constant: not in the space (Dirichlet), or left out
            sym[0, 0] = 1.0
        self.sym, self.ext = sym, ext

    def apply(self, x):
        r = -self.main * x
        for dim, c, f in self.faces:
            if f is not None:
                flux = c * f * (x - torch.roll(x, 1, dim))
                r = r + torch.roll(flux, -1, dim) - flux
            else:
                pad = [1, 1, 0, 0] if dim == 1 else [0, 0, 1, 1]
                y = torch.nn.functional.pad(x, pad)
                a, b = (y[:, :-2], y[:, 2:]) if dim == 1 else (y[:-2], y[2:])
                r = r + c * ((a - x) + (b - x))
        return r * self.wet

    def _extend(self, x):
        for dim in (0, 1):
            if self.neumann and (dim == 0 or not self.per):
                x = torch.cat([x, x.flip(dim)], dim)
            elif not self.neumann:
                z = torch.zeros_like(x.narrow(dim, 0, 1))
                x = torch.cat([z, x, z, -x.flip(dim)], dim)
        return x

    def fast(self, r):
        ny, nx = r.shape
        y = torch.fft.irfft2(torch.fft.rfft2(self._extend(r)) / self.sym, s=self.ext)
        o = 0 if self.neumann else 1
        return self.centred(y[o:o + ny, o:o + nx] * self.wet)

    def centred(self, x):
        if not self.neumann:
            return x
        return (x - x.sum() / self.wet.sum()) * self.wet

    def solve(self, b):
        """The solution on the whole array (zero off the wet points)."""
        r = self.centred(b[self.box] * self.wet)
        x, p, rz = torch.zeros_like(r), None, None
        stop = 1e-14 * float(r.norm())
        for _ in range(400):
            z = self.fast(r)
            new = (r * z).sum()
            if float(new) == 0.0:
                break
            p = z if p is None else z + (new / rz) * p
            rz = new
            q = self.apply(p)
            a = rz / (p * q).sum()
            x, r = x + a * p, r - a * q
            if not float(r.norm()) > stop:
                break
        out = torch.zeros_like(b)
        out[self.box] = self.centred(x)
        return out


class _Solve(torch.autograd.Function):
    @staticmethod
    def forward(ctx, b, ell):
        ctx.ell = ell
        return ell.solve(b)

    @staticmethod
    def backward(ctx, g):
        return ctx.ell.solve(g), None


class _Exact:
    """The time step of the models in plain FP64 torch: masked C-grid, WENO
    reconstructions, SSP-RK3 with a CFL time step."""

    def __init__(self, case, inp):
        self.model, self.per = case["model"], case["xperiodic"]
        self.nx, self.ny = case["nx"], case["ny"]
        self.dx, self.dy = 1.0 / self.nx, 1.0 / self.ny
        self.area = self.dx * self.dy
        self.cfl, self.par = _cfl(self.model), inp["par"]
        self.prog = list(inp["fields"]) + (["u.x", "u.y"] if self.model == "rsw" else [])
        msk = inp["msk"].double()
        self.s = {k: torch.zeros_like(msk) for k in self.prog}
        self.s.update({k: v.clone() for k, v in inp["fields"].items()})
        Y = msk.shape[1]
        self.Y = Y
        self.msk = msk
        self.mskx, self.msky = torch.zeros_like(msk), torch.zeros_like(msk)
        self.mskx[:, 1:] = msk[:, 1:] * msk[:, :-1]
        self.msky[1:, :] = msk[1:, :] * msk[:-1, :]
        n = msk.clone()
        n[:, 1:] += msk[:, :-1]
        n[1:, :] += msk[:-1, :]
        n[1:, 1:] += msk[:-1, :-1]
        self.mskv = (n == 4).double()
        self.slip = n.clamp(max=1.0) if case["noslip"] else (n == 4).double()
        self.oc = (_orders(msk, 1), _orders(msk, Y))
        wetv = (self.slip > 0).double()
        self.ov = (_orders(wetv, -1) * self.msky.long(), _orders(wetv, -Y) * self.mskx.long())
        self.ok = (_orders(self.mskx, -1), _orders(self.msky, -Y))
        cx, cy, h = self.dy / self.dx, self.dx / self.dy, HALO
        if self.model in ("eulerpsi", "qg"):
            p = self.par
            main = self.area * p["f0"] ** 2 / (p["g"] * p["H"]) if self.model == "qg" else 0.0
            self.ell = _Elliptic(self.mskv, (slice(h + 1, -h), slice(h + 1, -h)), cx, cy, main,
                                 False, False)
        elif self.model != "rsw":
            self.ell = _Elliptic(msk, (slice(h, -h), slice(h, -h)), cx, cy, 0.0, True, self.per)

    def fill(self, *arrays):
        if self.per:
            for a in arrays:
                _periodic(a)

    # -- operators
    def div(self, fx, fy):
        d = torch.zeros_like(fx)
        d[:, :-1] = -(fx[:, 1:] - fx[:, :-1])
        d[:-1, :] -= fy[1:, :] - fy[:-1, :]
        return d * self.msk

    def divflux(self, q, Ux, Uy):
        f = [_reconstruct(o, U, [_shift(q, k * s) for k in range(-3, 3)]) * U
             for o, U, s in ((self.oc[0], Ux, 1), (self.oc[1], Uy, self.Y))]
        return self.div(*f)

    def vortexforce(self, V, q, o, s, s2, sign):
        Vm = 0.25 * (V + _shift(V, s) + _shift(V, -s2) + _shift(V, s - s2))
        r = sign * _reconstruct(o, Vm, [_shift(q, k * s) for k in range(-2, 4)]) * Vm
        return torch.where(o > 0, r, torch.zeros_like(r))

    def ke(self, ux, uy, Ux, Uy):
        k = 0.0
        for U, u, o, s in ((Ux, ux, self.ok[0], 1), (Uy, uy, self.ok[1], self.Y)):
            Um = 0.5 * (U + _shift(U, s))
            r = _reconstruct(o, Um, [_shift(u, j * s) for j in range(-2, 4)]) * Um
            k = k + torch.where(o > 0, r, torch.zeros_like(r))
        return k * self.msk * 0.5

    def addgrad(self, phi, dux, duy):
        dux[:, 1:] -= (phi[:, 1:] - phi[:, :-1]) * self.mskx[:, 1:]
        duy[1:, :] -= (phi[1:, :] - phi[:-1, :]) * self.msky[1:, :]

    def velocity(self, psi):
        ux = -(psi[1:, :] - psi[:-1, :]) * self.mskx[:-1, :] / self.dy ** 2
        uy = (psi[:, 1:] - psi[:, :-1]) * self.msky[:, :-1] / self.dx ** 2
        pad = torch.nn.functional.pad
        return pad(ux, (0, 0, 0, 1)), pad(uy, (0, 1, 0, 0))

    def to_vertices(self, c):
        v = 0.25 * (c[:-1, :-1] + c[1:, :-1] + c[:-1, 1:] + c[1:, 1:])
        return torch.nn.functional.pad(v, (1, 0, 1, 0)) * self.mskv

    # -- equations
    def diag(self):
        s = self.s
        if self.model in ("eulerpsi", "qg"):
            b = self.to_vertices(s["omega" if self.model == "eulerpsi" else "pv"])
            if self.model == "qg":
                b = b - self.par["f"]
            s["psi"] = self.ell.solve(b)
            s["U.x"], s["U.y"] = self.velocity(s["psi"])
            return
        ux, uy = s["u.x"], s["u.y"]
        if self.model != "rsw":
            d = self.div(ux / self.dx ** 2, uy / self.dy ** 2)
            s["p"] = self.ell.solve(-d * self.area)
            self.fill(s["p"])
            self.addgrad(s["p"], ux, uy)
            self.fill(ux, uy)
        s["U.x"], s["U.y"] = ux / self.dx ** 2, uy / self.dy ** 2
        w = torch.zeros_like(ux)
        w[1:, :] = -(ux[1:, :] - ux[:-1, :])
        w[:, 1:] += uy[:, 1:] - uy[:, :-1]
        s["omega"] = w * self.slip
        s["ke"] = self.ke(ux, uy, s["U.x"], s["U.y"])
        if self.model == "rsw":
            s["p"] = (self.par["g"] / self.area) * s["h"]
        self.fill(s["omega"], s["ke"])

    def rhs(self):
        s, Y = self.s, self.Y
        Ux, Uy, d = s["U.x"], s["U.y"], {}
        for k in self.prog:
            if k in ("omega", "pv", "h", "b", "q"):
                d[k] = self.divflux(s[k], Ux, Uy)
        if "u.x" in self.prog:
            dux = self.vortexforce(Uy, s["omega"], self.ov[1], Y, 1, 1.0)
            duy = self.vortexforce(Ux, s["omega"], self.ov[0], 1, Y, -1.0)
            if self.model == "rsw":
                f = self.par["f0"] * self.area * 0.25
                dux[:-1, 1:-1] += f * (Uy[:-1, :-2] + Uy[1:, :-2] + Uy[:-1, 1:-1] + Uy[1:, 1:-1])
                duy[1:-1, :-1] -= f * (Ux[:-2, :-1] + Ux[:-2, 1:] + Ux[1:-1, :-1] + Ux[1:-1, 1:])
            self.addgrad(s["ke"], dux, duy)
            if self.model == "rsw":
                self.addgrad(s["p"], dux, duy)
            if self.model == "boussinesq":
                duy[1:, :] += (0.5 * self.dy) * (s["b"][1:, :] + s["b"][:-1, :]) * self.msky[1:, :]
            d["u.x"], d["u.y"] = dux, duy
        self.fill(*d.values())
        return d

    def cfl_dt(self):
        if self.model == "rsw":
            c = (self.par["g"] * self.par["H"]) ** 0.5
            return self.cfl / (c / self.dx + c / self.dy)
        return self.cfl / (float(self.s["U.x"].abs().max() + self.s["U.y"].abs().max()) + 1e-99)

    def steps(self, n):
        self.diag()
        for _ in range(n):
            dt, ds = self.cfl_dt(), []
            for coefs in ((dt,), (-0.75 * dt, 0.25 * dt), (-dt / 12, -dt / 12, 2 * dt / 3)):
                ds.append(self.rhs())
                for k in self.prog:
                    self.s[k] = self.s[k] + sum(c * d[k] for c, d in zip(coefs, ds))
                self.diag()
        return self.s

    def eulerpsi_step(self, w, dt):
        """One step as a differentiable function of the vorticity."""
        ds = []
        for coefs in ((dt,), (-0.75 * dt, 0.25 * dt), (-dt / 12, -dt / 12, 2 * dt / 3)):
            U = self.velocity(_Solve.apply(self.to_vertices(w), self.ell))
            ds.append(self.divflux(w, *U))
            w = w + sum(c * d for c, d in zip(coefs, ds))
        return w
