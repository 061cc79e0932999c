"""FP32-bulk 3D step: one copy of the face code for the three directions (the
normal velocity swapped at run time).  Every kernel case against the CPU
oracle, and the flow turned through the axes: the same values, turned."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_five_eq_gb300 import configs  # noqa: E402
from godunov_five_eq_gb300.implem import GodunovImplemGB300  # noqa: E402
from godunov_five_eq_gb300.metrics import l1_relative  # noqa: E402
from oracle.oracle import Oracle  # noqa: E402
from tests.helpers import amr_mesh, smooth_state, water_air_params  # noqa: E402

pytestmark = pytest.mark.gpu

L1_TOL = 1e-5  # the FP32-bulk form's bound, as in the other parity tests


def one_step(t, p, U, dt):
    impl = GodunovImplemGB300(p, t)
    d_U = torch.from_numpy(U).cuda()
    d_U2 = torch.zeros_like(d_U)
    impl.do_time_step(d_U, d_U2, dt, mode="mixed")
    torch.cuda.synchronize()
    assert impl.status() == 0
    return d_U2.cpu().numpy()


@pytest.mark.parametrize("thinc", [0, 1])
@pytest.mark.parametrize("gas", ["ideal", "stiff", "jwl"])
@pytest.mark.parametrize("integrator", [0, 1])
def test_mixed_3d_step_every_case(gas, thinc, integrator):
    if gas == "jwl":
        mesh, t, p, U = configs.mg_shock_tube("jwl", "air", bsize=8, nx_blocks=6, dim=3)
        p.thinc, p.integrator = thinc, integrator
    else:
        mesh, t = amr_mesh(dim=3, b=8, nref=3, lmin=1, lmax=2, seed=5)
        p = water_air_params(t, dim=3, b=8, thinc=thinc, integrator=integrator)
        if gas == "ideal":
            p.pinf = (0.0, 0.0)
        U = smooth_state(mesh, t, p, seed=4)
    o = Oracle(t, p)
    o.fill_outside(U)
    dt = o.dt(U)
    ref = o.step(U, dt)
    got = one_step(t, p, U, dt)
    assert np.all(np.isfinite(got[: t.n_owned]))
    assert l1_relative(t, got, ref).max() <= L1_TOL


@pytest.mark.parametrize("thinc", [0, 1])
def test_mixed_3d_step_turned_through_the_axes(thinc):
    """Random layers along x, y or z: the cells of a layer stay alike bit for
    bit, and the three runs agree as far as the form is accurate."""
    mesh, t = amr_mesh(dim=3, b=8, nref=0, lmin=1, lmax=1, seed=5, nbrick=(2, 2, 2))
    p = water_air_params(t, dim=3, b=8, thinc=thinc)
    I = configs.ids(3)
    rng = np.random.default_rng(1)
    nl = 32
    a0, pr, un = rng.uniform(0.05, 0.95, nl), rng.uniform(0.9e5, 1.1e5, nl), rng.uniform(-30, 30, nl)
    dx = float(t.level_dx[t.level[0]])
    xc = configs.cell_centers(mesh, t)
    pos = [np.floor(xc[:, d] / dx).astype(int) for d in range(3)]
    assert all(L.min() == 0 and L.max() == nl - 1 for L in pos)
    out = []
    for d in range(3):
        L = pos[d]
        vel = [np.zeros(L.shape) for _ in range(3)]
        vel[d] = un[L]
        U = np.zeros((t.n_total, t.nv, t.ncell))
        U[: t.n_owned] = np.moveaxis(configs.prim_to_cons(3, p, a0[L], a0[L] * 1000.0, (1 - a0[L]) * 1.2, pr[L], vel), 0, 1)
        got = one_step(t, p, U, 1e-7)[: t.n_owned]
        m = [I["IU"], I["IV"], I["IW"]]
        got[:, [m[0], m[d]]] = got[:, [m[d], m[0]]]
        line = np.zeros((t.nv, nl))
        for v in range(t.nv):
            line[v, L.ravel()] = got[:, v].ravel()
            assert np.array_equal(line[v][L], got[:, v])
        out.append(line)
    scale = np.abs(out[0]).max(axis=1, keepdims=True)
    for d in (1, 2):
        assert np.all(np.abs(out[d] - out[0]) <= L1_TOL * scale)
