"""The elliptic solves and the small-grid stage kernels at the sizes where
their rules change: a grid that is one dense level or just more, odd coarse
widths, one tile or just more, the sizes on both sides of the FP32 forms'
limits, and batches of uneven members.

Tolerances. Solves stop at a recurrence residual of 1e-12 |b|; the true one
drifts from it by rounding, iterations x eps x |A||x|/|b| <= 20 x 1.1e-16 x 4e4
(a 300-point basin) = 1e-10. A projected FP64 velocity has that divergence;
an FP32 one is rounded three times, 2^-24 each, and a divergence sums four of
them: 16 x 2^-24 |u|. Whole steps: 1e-10 per step as in the parity tests.

The FP32 divergence of two unconnected basins sums to 1e-7 in each instead of
0, and only the mean of both is taken off, so that system has no solution: the
solve reports its iteration limit.
"""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from fluids2d_gb300 import workloads as wl  # noqa: E402
from fluids2d_gb300._lib import F2DError, check, lib  # noqa: E402
from test_gpu_parity import (_ensemble, _model, _oracle_like, compare,  # noqa: E402
                             rel_l2)


def _mask(nx, ny, xper=False, islands=0, wall=False):
    msk = wl.default_mask(nx, ny, xperiodic=xper)
    rng = np.random.default_rng(nx * 1000 + ny)
    for _ in range(islands):
        j, i = int(rng.integers(4, ny)), int(rng.integers(6, nx))
        msk[j:j + max(2, ny // 9), i:i + max(2, nx // 11)] = 0
    if wall:  # two basins
        msk[3 + ny // 2] = 0
    if xper:
        msk[:, :3], msk[:, -3:] = msk[:, -6:-3], msk[:, 3:6]
    return msk


@pytest.mark.parametrize("model,nx,ny,precision,xper", [
    ("eulerpsi", 9, 7, "fp64", False),     # one dense level
    ("eulerpsi", 47, 45, "fp64", False),   # 46 x 44 nodes: the largest dense level
    ("eulerpsi", 48, 45, "fp64", False),   # just above it
    ("qg", 65, 64, "fp32", False),         # the same of the FP32 form: 4032 nodes
    ("qg", 67, 64, "fp32", False),
    ("qg", 48, 40, "fp64", True),
    ("qg", 45, 40, "fp64", True),          # odd periodic widths
    ("qg", 90, 61, "fp32", True),
    ("eulerpsi", 257, 33, "fp64", False),
    ("qg", 131, 97, "fp64", False),
    ("eulerpsi", 301, 287, "fp32", False),
    ("qg", 1450, 1400, "fp32", False),     # above 2M nodes: the level kernels
])
def test_vertex_solve(model, nx, ny, precision, xper):
    kw = dict(xperiodic=xper, f0=30.0 if model == "qg" else 0.0, g=1.0, H=1.0)
    msk = _mask(nx, ny, xper, islands=2 if min(nx, ny) > 30 else 0)
    m = _model(model, nx, ny, msk, precision=precision, **kw)
    solver = m.mesh.qg_helmholtz if model == "qg" else m.mesh.poisson_vertices
    b = np.random.default_rng(3).standard_normal(m.mesh.shape) * (m.mesh.G_vertices >= 0)
    x = np.zeros(m.mesh.shape)
    solver.solve(b, x)
    om = O.Mesh(O.Param(model=model, nx=nx, ny=ny, **kw))
    om.msk[:] = msk
    om.finalize()
    A, G = O.laplacian(om, om.maindiag if model == "qg" else 0.0)[:2]
    sel = G >= 0
    r = b[sel] - A @ x[sel]
    assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(b[sel])


@pytest.mark.parametrize("nx,ny,precision,xper,wall", [
    (8, 9, "fp64", False, False),
    (45, 45, "fp64", False, False),   # one dense level
    (46, 45, "fp64", False, True),    # just above it, two basins
    (41, 37, "fp64", True, False),    # odd periodic widths on every level
    (44, 61, "fp64", True, True),
    (131, 97, "fp64", False, True),
    (257, 160, "fp64", True, False),
    (45, 64, "fp32", False, False),   # between the FP32 form's two limits
    (64, 64, "fp32", True, False),
    (65, 64, "fp32", False, False),
    (65, 64, "fp32", False, True),
    (161, 300, "fp32", False, False),
])
def test_pressure_solve(nx, ny, precision, xper, wall):
    msk = _mask(nx, ny, xper, islands=1 if min(nx, ny) > 30 else 0, wall=wall)
    m = _model("euler", nx, ny, msk, precision=precision, xperiodic=xper, Lx=nx, Ly=ny)
    rng = np.random.default_rng(4)
    s = m.state
    for a, k in ((s.u.x, m.mesh.mskx), (s.u.y, m.mesh.msky)):
        v = rng.standard_normal(a.shape) * k
        if xper:
            v[:, :3], v[:, -3:] = v[:, -6:-3], v[:, 3:6]
        a[:] = v.astype(np.float32)
    fl = m.mesh.msk > 0
    if xper:
        fl[:, :3] = fl[:, -3:] = False

    def div():
        d = np.zeros(m.mesh.shape)
        d[:, :-1] = np.diff(s.u.x.astype(np.float64), axis=1)
        d[:-1] += np.diff(s.u.y.astype(np.float64), axis=0)
        return np.linalg.norm(d[fl])

    u0 = np.hypot(np.linalg.norm(s.u.x), np.linalg.norm(s.u.y))
    d0 = div()
    assert d0 > 0.1 * u0
    m.integrator.diag(s)
    if wall and precision == "fp32":
        with pytest.raises(F2DError, match="max iterations"):
            m.sync()
        return
    m.sync()
    s = m.state
    assert div() <= (1e-10 * d0 if precision == "fp64" else 16 * 2.0 ** -24 * u0)


@pytest.mark.parametrize("kind", ["eulerpsi", "rsw", "boussinesq"])
@pytest.mark.parametrize("nx,ny", [(26, 26), (27, 29), (90, 59),
                                   # 8 x 19 = 152 tiles of 32 x 8, and one row more
                                   (250, 146), (250, 147)])
def test_small_grid_stages(kind, nx, ny):
    make = {"eulerpsi": wl.eulerpsi_case, "rsw": wl.rsw_case,
            "boussinesq": wl.boussinesq_case}[kind]
    case = make(n=nx, ny=ny, seed=9, nislands=1)
    om = _oracle_like(case, kind, cfl=0.5)
    kw = dict(xperiodic=case.get("xperiodic", False), Lx=case["Lx"], Ly=case["Ly"],
              tend=1e300, maxite=10 ** 9, cfl=0.5)
    for k in ("f0", "g", "H", "beta"):
        if k in case:
            kw[k] = case[k]
    m = _model(kind, nx, ny, case["msk"], **kw)
    s = m.state
    for k, v in case["fields"].items():
        if "." in k:
            getattr(getattr(s, k.split(".")[0]), k.split(".")[1])[:] = v
        else:
            getattr(s, k)[:] = v
    m.integrator.diag(s)
    om.run_steps(2)
    m.advance(2)
    m.sync()
    compare(m, lambda k: om.s.get(k), 1e-10)


@pytest.mark.parametrize("sizes,precision,tol", [
    ([(20, 17), (47, 45), (48, 45), (129, 65), (250, 131)], "fp64", 1e-10),
    # above 1M nodes: the level kernels, against single models' persistent
    # solves (FP32: as for the members of the parity tests)
    ([(512, 512)] * 4 + [(33, 47)], "fp32", 1e-6),
])
def test_uneven_ensemble(sizes, precision, tol):
    cs = [wl.eulerpsi_case(n=nx, ny=ny, seed=20 + k, nislands=k % 3)
          for k, (nx, ny) in enumerate(sizes)]
    e = _ensemble(cs, precision)
    e.run(4)
    e.sync()
    for b, c in enumerate(cs):
        m = _model("eulerpsi", c["nx"], c["ny"], c["msk"], cfl=0.8, tend=1e300,
                   maxite=10 ** 9, precision=precision)
        m.state.omega[:] = c["fields"]["omega"]
        m.integrator.diag(m.state)
        m.advance(4)
        m.sync()
        assert rel_l2(e.get_field(b, "omega"), m.state.omega) <= tol, b
        assert rel_l2(e.get_field(b, "psi"), m.state.psi) <= tol, b


@pytest.mark.parametrize("nx,ny,precision,xper", [
    (32, 24, "fp64", False),   # one dense level
    (128, 96, "fp64", True),
    (32, 24, "fp32", True),
    (128, 96, "fp32", False),
])
def test_fluid_at_rest_stays_at_rest(nx, ny, precision, xper):
    """A zero right-hand side has the pressure 0, whatever was there before:
    a flow that is stopped does not start again. (Without a speed the time step
    is dtmax, whose default is beyond FP32's range.)"""
    case = wl.euler_case(n=nx, ny=ny, seed=8, nislands=1, xperiodic=xper)
    m = _model("euler", nx, ny, case["msk"], precision=precision, xperiodic=xper,
               Lx=case["Lx"], Ly=case["Ly"], cfl=0.5, dtmax=1.0, tend=1e300,
               maxite=10 ** 9)
    s = m.state
    s.u.x[:], s.u.y[:] = case["fields"]["u.x"], case["fields"]["u.y"]
    m.integrator.diag(s)
    m.advance(3)
    s = m.state
    s.u.x[:] = 0.0
    s.u.y[:] = 0.0
    m.integrator.diag(s)
    m.advance(2)
    m.sync()
    s = m.state
    for a in (s.u.x, s.u.y, s.p):
        assert np.all(a == 0)


@pytest.mark.parametrize("nx,ny", [(72, 72), (162, 60), (324, 100)])
def test_fp32_pressure_over_odd_periodic_widths(nx, ny):
    """The FP32 form's coarse matrix on x-periodic levels of odd width (9, 81):
    the same from every build, and the projection as good as elsewhere."""
    msk = _mask(nx, ny, True, islands=1)
    rng = np.random.default_rng(6)
    u = [rng.standard_normal(msk.shape) for _ in range(2)]
    out = []
    for _ in range(2):
        m = _model("euler", nx, ny, msk, precision="fp32", xperiodic=True, Lx=nx, Ly=ny)
        s = m.state
        for a, v, k in ((s.u.x, u[0], m.mesh.mskx), (s.u.y, u[1], m.mesh.msky)):
            a[:] = (v * k).astype(np.float32)
            a[:, :3], a[:, -3:] = a[:, -6:-3], a[:, 3:6]
        u0 = np.hypot(np.linalg.norm(s.u.x), np.linalg.norm(s.u.y))
        m.integrator.diag(s)
        m.sync()
        out.append(m.state.p.copy())
        s = m.state
        d = np.zeros(m.mesh.shape)
        d[:, :-1] = np.diff(s.u.x.astype(np.float64), axis=1)
        d[:-1] += np.diff(s.u.y.astype(np.float64), axis=0)
        fl = m.mesh.msk > 0
        fl[:, :3] = fl[:, -3:] = False
        assert np.linalg.norm(d[fl]) <= 16 * 2.0 ** -24 * u0
    assert np.array_equal(*out)


@pytest.mark.parametrize("nx,ny,precision,xper,want", [
    (256, 200, "fp64", False, 2), (256, 200, "fp32", False, 2),
    (1450, 1400, "fp32", False, 1),
    # 75 periodic columns: above the dense level (2048 unknowns; FP32 4096), or on it
    (300, 200, "fp64", True, 0), (300, 200, "fp32", True, 2), (300, 300, "fp32", True, 1),
])
def test_timed_leg_is_of_the_form_that_runs(nx, ny, precision, xper, want):
    m = _model("qg", nx, ny, _mask(nx, ny, xper), precision=precision, xperiodic=xper,
               f0=1.0, g=1.0, H=1.0)
    rng = np.random.default_rng(2)
    m.state.pv[:] = rng.standard_normal(m.mesh.shape) * (m.mesh.msk > 0)
    m.integrator.diag(m.state)
    m.sync()
    form, ms = ctypes.c_int(-1), ctypes.c_double()
    nodes, es = ctypes.c_int64(), ctypes.c_int()
    check(lib().f2d_solver_form(m._h, ctypes.byref(form)))
    assert form.value == want
    check(lib().f2d_time_solver(m._h, 3, 0, ctypes.byref(ms), ctypes.byref(nodes),
                                ctypes.byref(es)))
    assert ms.value > 0 and es.value == (8 if precision == "fp64" else 4)
    psi = m.state.psi.copy()
    m.integrator.diag(m.state)  # the hook leaves the solver as it was
    m.sync()
    assert rel_l2(m.state.psi, psi) <= 1e-10


@pytest.mark.parametrize("n,size,precision,want", [
    (152, (32, 32), "fp64", 2), (153, (32, 32), "fp64", 0), (153, (40, 36), "fp64", 2),
    (152, (48, 40), "fp32", 2), (153, (48, 40), "fp32", 1), (153, (16, 12), "fp32", 0),
    (1230, (40, 40), "fp64", 2),  # more than eight members to a block
])
def test_batches_around_the_number_of_sms(n, size, precision, want):
    """The form of batches with as many members as SMs (152 of them here) and
    one more, and their members against single models."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n += (sms - 152) * (n < 160)
    cs = [wl.eulerpsi_case(n=size[0], ny=size[1], seed=20 + k, nislands=k % 2)
          for k in range(4)]
    e = _ensemble([cs[b % 4] for b in range(n)], precision)
    form = ctypes.c_int(-1)
    check(lib().f2d_ensemble_solver_form(e._h, ctypes.byref(form)))
    assert form.value == want
    e.run(3)
    e.sync()
    tol = 1e-10 if precision == "fp64" else 1e-6
    for k, c in enumerate(cs):
        m = _model("eulerpsi", c["nx"], c["ny"], c["msk"], cfl=0.8, tend=1e300,
                   maxite=10 ** 9, precision=precision)
        m.state.omega[:] = c["fields"]["omega"]
        m.integrator.diag(m.state)
        m.advance(3)
        m.sync()
        for b in (k, n // 2 // 4 * 4 + k, (n - 1 - k) // 4 * 4 + k):
            if b >= n:
                continue
            assert rel_l2(e.get_field(b, "omega"), m.state.omega) <= tol, b
            assert rel_l2(e.get_field(b, "psi"), m.state.psi) <= tol, b


def _true_residual(m, model, b, x, msk, **kw):
    om = O.Mesh(O.Param(model=model, nx=m.param.nx, ny=m.param.ny, **kw))
    om.msk[:] = msk
    om.finalize()
    A, G = O.laplacian(om, om.maindiag if model == "qg" else 0.0)[:2]
    sel = G >= 0
    return np.linalg.norm(b[sel] - A @ x[sel]) / np.linalg.norm(b[sel])


def _rounds(m):
    n = ctypes.c_int64()
    check(lib().f2d_refine_rounds(m._h, ctypes.byref(n)))
    return n.value


@pytest.mark.parametrize("model,nx,ny", [("eulerpsi", 40, 36), ("eulerpsi", 97, 131),
                                         ("qg", 90, 61)])
def test_fp32_vertex_solve_from_a_far_start(model, nx, ny):
    """The FP32 form ends on the true residual: a start 1e10 times the
    solution leaves rounding of its own size in x, which the recurrence does
    not see. An ordinary start needs one check and no second start."""
    kw = dict(f0=30.0 if model == "qg" else 0.0, g=1.0, H=1.0)
    msk = _mask(nx, ny, islands=2)
    m = _model(model, nx, ny, msk, precision="fp32", **kw)
    solver = m.mesh.qg_helmholtz if model == "qg" else m.mesh.poisson_vertices
    rng = np.random.default_rng(5)
    wet = m.mesh.G_vertices >= 0
    b = rng.standard_normal(m.mesh.shape) * wet
    x = np.zeros(m.mesh.shape)
    solver.solve(b, x)
    assert _true_residual(m, model, b, x, msk, **kw) <= 1e-10
    assert _rounds(m) == 0
    x = 1e10 * np.abs(x).max() * rng.standard_normal(x.shape) * wet
    solver.solve(b, x)
    assert _true_residual(m, model, b, x, msk, **kw) <= 1e-10
    assert solver.last_relres <= 1e-10
    assert _rounds(m) >= 1
    m.sync()


def test_fp32_ensemble_from_a_far_start():
    """The same for one member of a batch, the others being done."""
    sizes = [(40, 36), (97, 131), (64, 64)]
    cs = [wl.eulerpsi_case(n=nx, ny=ny, seed=20 + k, nislands=1)
          for k, (nx, ny) in enumerate(sizes)]
    e, far = _ensemble(cs, "fp32"), _ensemble(cs, "fp32")
    rng = np.random.default_rng(6)
    psi = far.get_field(1, "psi")
    far.set_field(1, "psi", 1e10 * rng.standard_normal(psi.shape) * psi)
    far.diag()
    far.sync()
    assert far.stats()["refine_rounds"] >= 1 and e.stats()["refine_rounds"] == 0
    for b in range(len(cs)):
        assert rel_l2(far.get_field(b, "psi"), e.get_field(b, "psi")) <= 1e-10, b


def test_fp32_iteration_limit_counts_rounds():
    """poisson_maxit = 5 allows the FP32 form two rounds of 30 iterations,
    whichever kernels run it (a solve from zero takes 12 to 20)."""
    case = wl.eulerpsi_case(n=96, ny=80, seed=3, nislands=2)
    m = _model("eulerpsi", 96, 80, case["msk"], precision="fp32", poisson_maxit=5)
    m.state.omega[:] = case["fields"]["omega"]
    m.integrator.diag(m.state)
    m.sync()


def test_memory_of_an_fp64_model():
    """Of its grid's arrays of 8 bytes an FP64 eulerpsi model holds 24.6 of its
    own, one for the coarse levels, and two of the persistent solve (its others
    are the level kernels'), with its dense inverse half of one: 28.3, and 1.7
    for small buffers and the driver."""
    m = _model("eulerpsi", 32, 32)
    m.integrator.diag(m.state)  # (the library's own memory)
    m.sync()
    n = 3072
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    m = _model("eulerpsi", n, n)
    check(lib().f2d_diag(m._h))
    check(lib().f2d_run(m._h, 1))
    m.sync()
    form = ctypes.c_int(-1)
    check(lib().f2d_solver_form(m._h, ctypes.byref(form)))
    assert form.value == 2
    used = free - torch.cuda.mem_get_info()[0]
    assert used <= 30 * 8 * ((n + 6 + 15) // 16 * 16) * (n + 6)
