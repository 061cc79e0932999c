"""The FP64 form's fast arithmetic (csrc/g5_fast64.cuh) where its shortcuts
could fail: zeros, pure materials, values outside its range (which take the
reference arithmetic), non-physical states, every constant of the mixture.
Bit for bit against the CPU oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_five_eq_gb300 import configs  # noqa: E402
from godunov_five_eq_gb300.implem import GodunovImplemGB300  # noqa: E402
from oracle.oracle import Oracle  # noqa: E402
from tests.helpers import amr_mesh, smooth_state, water_air_params  # noqa: E402

pytestmark = pytest.mark.gpu

GASES = {"ideal": ((1.4, 1.648), (0.0, 0.0)), "first": ((4.4, 1.4), (6e8, 0.0)), "second": ((1.4, 4.4), (0.0, 6e8)), "both": ((4.4, 3.0), (6e8, 1e8))}


def build(dim, b, kind, gas, **kw):
    mesh, t = amr_mesh(dim=dim, b=b, nref=3, lmin=1, lmax=2, seed=5)
    p = water_air_params(t, dim=dim, b=b, **kw)
    p.gamma, p.pinf = GASES[gas]
    U = smooth_state(mesh, t, p)
    I = configs.ids(dim)
    n = t.n_owned
    V = U[:n]
    rng = np.random.default_rng(3)
    mom = [I["IU"], I["IV"]] + ([I["IW"]] if dim == 3 else [])

    def state(a0, vel):
        pr = np.full_like(a0, 1e5)
        pr[: n // 2] = 1.3e5
        U[:n] = np.moveaxis(configs.prim_to_cons(dim, p, a0, a0 * 1000.0, (1.0 - a0) * 1.2, pr, vel), 0, 1)

    a0 = V[:, I["IA0"]].copy()
    zero = [0.0 * a0 for _ in range(dim)]
    if kind == "rest":
        state(a0, zero)
    elif kind == "pure":
        state(np.where(a0 > 0.5, 1.0, 0.0), [7.0 + 0.0 * a0] + zero[1:])
    elif kind in ("tiny", "subnormal", "huge", "nan"):
        # a few cells far from the rest: the last owned blocks only, so that both arithmetics run
        val = {"tiny": 1e-280, "subnormal": 3e-310, "huge": 1e215, "nan": np.nan}[kind]
        state(a0, [1e-200 * rng.standard_normal(a0.shape) for _ in range(dim)])
        for v in mom[:2] if kind != "nan" else mom[:1]:
            V[-1, v, rng.integers(0, t.ncell, 5)] = val
    elif kind == "negative":
        cells = rng.random(a0.shape) < 0.02
        V[:, I["IE"]] = np.where(cells, V[:, I["IE"]] * 0.2, V[:, I["IE"]])
    return t, p, U


CASES = [
    (2, 16, "smooth", "ideal", {}),
    (2, 16, "smooth", "second", dict(slope_type=2.0, source_term=1)),
    (2, 8, "smooth", "both", dict(thinc=1, source_term=1)),
    (2, 8, "smooth", "first", dict(integrator=1, slope_type=0.0)),
    (2, 16, "rest", "first", {}),
    (2, 8, "rest", "ideal", dict(slope_type=2.0)),
    (2, 16, "pure", "first", {}),
    (2, 8, "pure", "ideal", dict(thinc=1)),
    (2, 16, "tiny", "ideal", {}),
    (2, 8, "subnormal", "first", {}),
    (2, 16, "huge", "ideal", {}),
    (2, 16, "nan", "ideal", {}),
    (2, 8, "negative", "ideal", {}),
    (2, 16, "negative", "both", dict(slope_type=2.0)),
    (3, 8, "smooth", "first", {}),
    (3, 8, "smooth", "second", dict(thinc=1, slope_type=2.0, source_term=1)),
    (3, 8, "smooth", "both", dict(integrator=1, slope_type=0.0)),
    (3, 8, "rest", "ideal", dict(thinc=1)),
    (3, 8, "pure", "first", {}),
    (3, 8, "tiny", "ideal", dict(source_term=1)),
    (3, 8, "subnormal", "first", {}),
    (3, 8, "huge", "ideal", dict(thinc=1)),
    (3, 8, "nan", "ideal", {}),
    (3, 8, "negative", "ideal", dict(slope_type=2.0)),
]


@pytest.mark.parametrize("dim,b,kind,gas,kw", CASES, ids=["-".join([str(c[0]), str(c[1]), c[2], c[3]] + sorted(c[4])) for c in CASES])
def test_fast64_step_matches_oracle(dim, b, kind, gas, kw):
    t, p, U = build(dim, b, kind, gas, **kw)
    o = Oracle(t, p)
    o.fill_outside(U)
    dt = 1e-6
    with np.errstate(all="ignore"):
        ref = o.step(U, dt)[: t.n_owned]
        full = np.zeros_like(U)
        full[: t.n_owned] = ref
        inv_ref = o.inv_dt(full)
    impl = GodunovImplemGB300(p, t)
    d_U = torch.from_numpy(U).cuda()
    d_U2 = torch.zeros_like(d_U)
    inv = torch.zeros(t.n_inst, dtype=torch.float64, device="cuda")
    impl.do_time_step(d_U, d_U2, dt, mode="fp64", inv_dt_out=inv)
    torch.cuda.synchronize()
    got = d_U2.cpu().numpy()[: t.n_owned]
    assert np.array_equal(got, ref, equal_nan=True), f"{(~((got == ref) | (np.isnan(got) & np.isnan(ref)))).sum()} values differ"
    if kind == "nan":
        assert impl.status() != 0
    else:
        assert np.array_equal(inv.cpu().numpy(), inv_ref)


@pytest.mark.parametrize("dim,b", [(2, 16), (2, 8), (3, 8)])
@pytest.mark.parametrize("er,ec", [(0.1, 0.0125), (0.0, 0.0), (0.5, 0.5), (1.0, 1.0), (2.0, 1e-60), (0.25, 0.9)])
def test_gradient_flags_match_oracle(dim, b, er, ec):
    """Indicators exactly on a threshold, of tiny, huge, zero and NaN densities."""
    mesh, t = amr_mesh(dim=dim, b=b, nref=3, lmin=1, lmax=2, seed=7)
    p = water_air_params(t, dim=dim, b=b)
    I = configs.ids(dim)
    rng = np.random.default_rng(11)
    n = t.n_owned
    U = smooth_state(mesh, t, p)
    for k, v in enumerate((I["IAD0"], I["IAD1"])):
        base = rng.choice([1.0, 0.001, 1000.0, 1e-4, 1e60], size=(n, 1))
        step = rng.choice([0.0, 1e-6, er, ec, 0.3, 3.0], size=(n, 1)) * rng.integers(0, 2, (n, t.ncell))
        U[:n, v] = base * (1.0 - np.minimum(step, 0.999999) * (k + 1) / 2)
    U[0, I["IAD0"], :3] = (np.nan, 0.0, -0.5)
    U[1, I["IAD1"], 5] = np.inf
    o = Oracle(t, p)
    o.fill_outside(U)
    for lmin, lmax in ((0, 3), (1, 2), (2, 2)):
        with np.errstate(all="ignore"):
            ref = o.refine_flags(U, 0, er, ec, 0.02, lmin, lmax)
        got = GodunovImplemGB300(p, t).refine_flags(torch.from_numpy(U).cuda(), 0, er, ec, 0.02, lmin, lmax)
        assert np.array_equal(got.cpu().numpy(), ref)


@pytest.mark.parametrize("dim,b,kind,gas", [(2, 16, "pure", "first"), (2, 8, "subnormal", "both"), (2, 16, "rest", "ideal"), (3, 8, "tiny", "second"), (3, 8, "negative", "ideal")])
def test_fields_match_single_quantities_and_oracle(dim, b, kind, gas):
    from oracle.oracle import derived

    t, p, U = build(dim, b, kind, gas)
    U[0, 0, :4] *= 1.0 + 2e-16 * np.arange(4)  # ID apart from the partial densities
    impl = GodunovImplemGB300(p, t)
    d_U = torch.from_numpy(U).cuda()
    codes = [64 + q for q in range(8)] + [1, 0]
    got = impl.pack_fields(d_U, codes).cpu().numpy()
    for q in range(8):
        with np.errstate(all="ignore"):
            ref = np.asarray(derived(p, U, q)).reshape(U.shape[0], -1)[: t.n_owned]
        assert np.array_equal(got[q], ref, equal_nan=True), q
        one = impl.derived_quantity(d_U, q).cpu().numpy()[: t.n_owned, 0]
        assert np.array_equal(one, ref, equal_nan=True), q
    assert np.array_equal(got[8], U[: t.n_owned, 1]) and np.array_equal(got[9], U[: t.n_owned, 0])
    with np.errstate(all="ignore"):
        inv = Oracle(t, p).inv_dt(U)
    assert np.array_equal(impl.compute_inv_dt(d_U).cpu().numpy(), inv)


@pytest.mark.parametrize("law,other,dim,kw", [("jwl", "air", 2, {}), ("jwl", None, 2, dict(source_term=1)), ("shockwave", "air", 2, {}), ("shockwave2", "jwl", 2, {}), ("jwl", "air", 3, {}), ("jwl", "shockwave", 3, dict(source_term=1))])
@pytest.mark.parametrize("thinc", [0, 1])
def test_mie_grueneisen_step_and_fields_match_oracle(law, other, dim, kw, thinc):
    """Laws and mixture rules on the integer pipes, with an absent material
    (reference density) and a cell outside the range."""
    from oracle.oracle import derived

    mesh, t, p, U = configs.mg_shock_tube(law, other, bsize=8 if dim == 3 else 16, nx_blocks=6, dim=dim, **kw)
    p.thinc = thinc
    I = configs.ids(dim)
    rng = np.random.default_rng(2)
    n = t.n_owned
    U[:n, I["IU"]] += U[:n, I["ID"]] * 50.0 * rng.standard_normal((n, t.ncell))
    a = U[1, I["IA0"], :7]
    U[1, I["IAD1"], :7] += U[1, I["IAD0"], :7]
    a[:] = 0.0
    U[1, I["IAD0"], :7] = 0.0
    U[1, I["IA1"], :7] = 1.0
    U[2, I["IV"], 3] = 1e-290
    o = Oracle(t, p)
    o.fill_outside(U)
    dt = 0.2 * o.dt(U)
    ref = o.step(U, dt)[:n]
    full = np.zeros_like(U)
    full[:n] = ref
    impl = GodunovImplemGB300(p, t)
    d_U = torch.from_numpy(U).cuda()
    d_U2 = torch.zeros_like(d_U)
    inv = torch.zeros(1, dtype=torch.float64, device="cuda")
    impl.do_time_step(d_U, d_U2, dt, mode="fp64", inv_dt_out=inv)
    got = d_U2.cpu().numpy()[:n]
    assert np.array_equal(got, ref, equal_nan=True)
    assert np.array_equal(inv.cpu().numpy(), o.inv_dt(full))
    assert np.array_equal(impl.compute_inv_dt(d_U).cpu().numpy(), o.inv_dt(U))
    f = impl.pack_fields(d_U, [64 + q for q in range(8)]).cpu().numpy()
    for q in range(8):
        assert np.array_equal(f[q], np.asarray(derived(p, U, q)).reshape(U.shape[0], -1)[:n], equal_nan=True), q


@pytest.mark.parametrize("nref,thinc", [(1, 0), (2, 1), (40, 0), (40, 1)])
def test_half_block_round_in_the_solver_loop(nref, thinc):
    """16x16 blocks few enough for a last round in halves (and more): walls,
    coarse/fine records and the boundary fill inside the step, five steps."""
    mesh, t = amr_mesh(dim=2, b=16, periodic=False, nbrick=(3, 2), nref=nref, lmin=1, lmax=4, seed=nref)
    p = water_air_params(t, b=16, bc=(2, 2, 3, 3, 1, 1), thinc=thinc)
    p.gamma, p.pinf = GASES["ideal"]
    U = smooth_state(mesh, t, p)
    o = Oracle(t, p)
    ref, hist = o.run(U.copy(), 5)
    impl = GodunovImplemGB300(p, t)
    d_U = torch.from_numpy(U).cuda()
    d_U2 = torch.zeros_like(d_U)
    dts = torch.zeros((5, 1), dtype=torch.float64, device="cuda")
    impl.run(d_U, d_U2, 5, mode="fp64", dt_hist=dts)
    torch.cuda.synchronize()
    assert impl.status() == 0
    assert np.array_equal(dts.cpu().numpy().ravel(), np.asarray(hist).ravel())
    assert np.array_equal(d_U.cpu().numpy(), ref)


@pytest.mark.parametrize("dim,b", [(2, 16), (2, 8), (3, 8)])
@pytest.mark.parametrize("thinc", [0, 1])
def test_flow_from_rest_matches_oracle(dim, b, thinc):
    """A pressure jump in a gas at rest: ahead of the waves the velocities fall
    off to nothing, so that blocks hold cells and faces inside and outside the
    fast form's range side by side."""
    mesh, t = amr_mesh(dim=dim, b=b, nref=2, lmin=1, lmax=2, seed=5)
    p = water_air_params(t, dim=dim, b=b, thinc=thinc, source_term=thinc)
    p.gamma, p.pinf = GASES["first"]
    xc = configs.cell_centers(mesh, t)
    d = xc[:, 0] + 0.3 * xc[:, 1] + (0.2 * xc[:, 2] if dim == 3 else 0.0)
    a0 = np.where(np.abs(d - 1.1) < 0.2, 1.0 - 1e-6, 1e-6)
    pr = np.where(d < 0.7, 1.4e5, 1e5)
    U = np.zeros((t.n_total, t.nv, t.ncell))
    U[: t.n_owned] = np.moveaxis(configs.prim_to_cons(dim, p, a0, a0 * 1000.0, (1.0 - a0) * 1.2, pr, [0.0 * a0] * dim), 0, 1)
    nsteps = 24
    ref, _ = Oracle(t, p).run(U, nsteps)
    I = configs.ids(dim)
    v = np.abs(ref[: t.n_owned, I["IV"]])
    assert ((v > 0) & (v < 1e-136)).any() and (v > 1e-20).any()
    impl = GodunovImplemGB300(p, t)
    d_U = torch.from_numpy(U).cuda()
    d_U2 = torch.zeros_like(d_U)
    impl.run(d_U, d_U2, nsteps, mode="fp64")
    torch.cuda.synchronize()
    assert impl.status() == 0
    assert np.array_equal(d_U.cpu().numpy()[: t.n_owned], ref[: t.n_owned])
