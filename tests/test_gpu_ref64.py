"""The FP64 form with constants outside the fast arithmetic's range (a density
or sound-speed floor of zero or far below it): the kernels in the reference's
arithmetic.  Bit for bit against the CPU oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_five_eq_gb300 import configs  # noqa: E402
from godunov_five_eq_gb300.implem import GodunovImplemGB300  # noqa: E402
from oracle.oracle import Oracle, derived  # noqa: E402
from tests.helpers import amr_mesh, smooth_state, water_air_params  # noqa: E402

pytestmark = pytest.mark.gpu

FLOORS = {"smallc0": dict(smallc=0.0), "smallr0": dict(smallr=0.0), "smallr-70": dict(smallr=1e-70)}


def build(dim, b, floor, gas=None, **kw):
    """A state on a mesh with coarse/fine faces (gas None), or a JWL tube."""
    if gas:
        mesh, t, p, U = configs.mg_shock_tube(gas, "air", bsize=b, nx_blocks=6, dim=dim)
        for k, v in {**FLOORS[floor], **kw}.items():
            setattr(p, k, v)
        return t, p, U
    mesh, t = amr_mesh(dim=dim, b=b, nref=3, lmin=1, lmax=2, seed=5)
    p = water_air_params(t, dim=dim, b=b, **FLOORS[floor], **kw)
    return t, p, smooth_state(mesh, t, p, seed=2)


def device(U):
    d_U = torch.from_numpy(U).cuda()
    return d_U, torch.zeros_like(d_U)


@pytest.mark.parametrize("floor", sorted(FLOORS))
@pytest.mark.parametrize("dim,b,gas", [(2, 16, None), (2, 8, None), (3, 8, None), (2, 16, "jwl"), (3, 8, "jwl")])
def test_fields_and_cfl_rate(dim, b, gas, floor):
    t, p, U = build(dim, b, floor, gas)
    o = Oracle(t, p)
    o.fill_outside(U)
    d_U, _ = device(U)
    impl = GodunovImplemGB300(p, t)
    n = t.n_owned
    codes = [64 + q for q in range(8)] + [1, 0]
    every = impl.pack_fields(d_U, codes).cpu().numpy()
    for q in range(8):
        ref = np.asarray(derived(p, U, q)).reshape(U.shape[0], -1)
        assert np.array_equal(every[q], ref[:n], equal_nan=True), q
        assert np.array_equal(impl.pack_fields(d_U, [3, 64 + q]).cpu().numpy()[1], ref[:n], equal_nan=True), q
        assert np.array_equal(impl.derived_quantity(d_U, q).cpu().numpy()[:n, 0], ref[:n], equal_nan=True), q
    assert np.array_equal(every[8], U[:n, 1]) and np.array_equal(every[9], U[:n, 0])
    assert np.array_equal(impl.compute_inv_dt(d_U).cpu().numpy(), o.inv_dt(U))


CASES = [
    # dim, block, law, options
    (2, 16, None, {}),
    (2, 16, None, dict(thinc=1, source_term=1)),
    (2, 16, None, dict(integrator=1, slope_type=2.0)),
    (2, 8, None, dict(slope_type=0.0)),
    (2, 8, None, dict(thinc=1, slope_type=2.0)),
    (2, 8, "jwl", dict(thinc=1)),
    (2, 16, "shockwave", dict(source_term=1)),
    (3, 8, None, {}),
    (3, 8, None, dict(thinc=1, source_term=1, slope_type=2.0)),
    (3, 8, None, dict(integrator=1)),
    (3, 8, "jwl", dict(thinc=1)),
]


@pytest.mark.parametrize("floor", sorted(FLOORS))
@pytest.mark.parametrize("dim,b,gas,kw", CASES, ids=["-".join([str(c[0]), str(c[1]), str(c[2])] + sorted(c[3])) for c in CASES])
def test_step(dim, b, gas, kw, floor):
    t, p, U = build(dim, b, floor, gas, **kw)
    o = Oracle(t, p)
    o.fill_outside(U)
    dt = 0.5 * o.dt(U)
    ref = o.step(U, dt)
    impl = GodunovImplemGB300(p, t)
    d_U, d_U2 = device(U)
    inv = torch.zeros(t.n_inst, dtype=torch.float64, device="cuda")
    impl.do_time_step(d_U, d_U2, dt, mode="fp64", inv_dt_out=inv)
    n = t.n_owned
    assert np.array_equal(d_U2.cpu().numpy()[:n], ref[:n], equal_nan=True)
    full = np.zeros_like(U)
    full[:n] = ref[:n]
    assert np.array_equal(inv.cpu().numpy(), o.inv_dt(full))


@pytest.mark.parametrize("dim,b", [(2, 16), (2, 8), (3, 8)])
@pytest.mark.parametrize("integrator", [0, 2])
@pytest.mark.parametrize("thinc", [0, 1])
def test_solver_loop(dim, b, integrator, thinc):
    """Walls, coarse/fine records and the boundary fill inside the step, five
    steps of the device-driven loop; RK2's combination with its CFL rate."""
    mesh, t = amr_mesh(dim=dim, b=b, periodic=False, nref=4, lmin=1, lmax=3, seed=9)
    p = water_air_params(t, dim=dim, b=b, bc=(2, 2, 3, 3, 2, 3), integrator=integrator, thinc=thinc, smallc=0.0)
    U = smooth_state(mesh, t, p, seed=3)
    ref, hist = Oracle(t, p).run(U.copy(), 5)
    impl = GodunovImplemGB300(p, t)
    d_U, d_U2 = device(U)
    dts = torch.zeros((5, 1), dtype=torch.float64, device="cuda")
    impl.run(d_U, d_U2, 5, mode="fp64", dt_hist=dts)
    assert impl.status() == 0
    assert np.array_equal(dts.cpu().numpy().ravel(), np.asarray(hist).ravel())
    assert np.array_equal(d_U.cpu().numpy(), ref)


@pytest.mark.parametrize("dim,b", [(2, 16), (2, 8), (3, 8)])
def test_host_step_and_shapes(dim, b):
    """Chunks with work lists, and every launch shape, give the plain step's bits."""
    t, p, U = build(dim, b, "smallc0")
    o = Oracle(t, p)
    o.fill_outside(U)
    dt = o.dt(U)
    ref = o.step(U, dt)[: t.n_owned]
    impl = GodunovImplemGB300(p, t)
    hU, hU2 = torch.from_numpy(U.copy()).pin_memory(), torch.zeros(U.shape, dtype=torch.float64).pin_memory()
    impl.do_time_step_host(hU, hU2, dt, mode="fp64")
    torch.cuda.synchronize()
    assert np.array_equal(hU2.numpy()[: t.n_owned], ref)
    d_U, d_U2 = device(U)
    for ctas in (1, 2, 0):
        for claim in (0, 1):
            impl.set_shape("fp64", ctas_per_sm=ctas, claim=claim, walk_cf_first=claim)
            d_U2.zero_()
            impl.do_time_step(d_U, d_U2, dt, mode="fp64")
            assert np.array_equal(d_U2.cpu().numpy()[: t.n_owned], ref)
