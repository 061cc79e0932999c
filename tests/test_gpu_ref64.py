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
