"""Device memory that g5_remap keeps between calls (its tables' pool): counted by
the context's memory size, bounded, given back with the context."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from godunov_five_eq_gb300.implem import GodunovImplemGB300  # noqa: E402
from godunov_five_eq_gb300.mesh import RemapTable  # noqa: E402
from tests.helpers import amr_mesh, water_air_params  # noqa: E402

pytestmark = pytest.mark.gpu

KEEP = 32 << 20  # what the pool may keep


def copies(n_old, n_new):
    """n_new copies of old blocks."""
    src = np.zeros((n_new, 4), np.int32)
    src[:, 0] = np.arange(n_new) % n_old
    return RemapTable(dim=2, bsize=8, n_old=n_old, kind=np.zeros(n_new, np.int8), src=src)


def test_remap_pool_is_counted_and_bounded():
    mesh, t = amr_mesh(dim=2, b=8, nref=1, lmin=1, lmax=2, seed=5)
    impl = GodunovImplemGB300(water_air_params(t), t)
    none = impl.total_mem_size_in_bytes()
    U = torch.rand((t.n_owned, t.nv, t.ncell), dtype=torch.float64, device="cuda")
    kept = []
    # a table within the bound, the same again, one beyond it, a small one after that
    for n_new in (1000, 1000, 1 << 21, 1000):
        rt = copies(t.n_owned, n_new)
        U_new = torch.zeros((n_new, t.nv, t.ncell), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        impl.remap(rt, U, U_new)
        torch.cuda.synchronize()
        kept.append(impl.total_mem_size_in_bytes() - none)
        if len(kept) == 1:
            assert kept[0] == free - torch.cuda.mem_get_info()[0]
        last = U_new[-1].cpu()
        assert torch.equal(last, U[rt.src[-1, 0]].cpu())
        del U_new
    assert min(kept) > 0 and max(kept) <= KEEP and kept[1] == kept[0]
    impl.close()
