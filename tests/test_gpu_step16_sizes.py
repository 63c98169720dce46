"""16-bit steps on both sides of the grid size up to which they run with more
registers (75,776 nodes on 148 SMs), rows of whole warps and rows that leave
warps across x-rows, whose warps take the tested update for all their nodes.
Against the FP64 oracle, with the bound of the smaller sizes: within
4 (n + 1) u of the largest after n steps."""
import numpy as np
import pytest

from helpers import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,u", [("f16s", 2.0 ** -11), ("bf16s", 2.0 ** -8)])
@pytest.mark.parametrize("collision", ["bgk", "regularized"])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("lx,ly,lz", [(64, 36, 32), (64, 37, 33), (63, 36, 32), (65, 36, 33), (16, 3, 1600)])
def test_step16_by_grid_size(lbm, oracle_mod, storage, u, collision, periodic, lx, ly, lz):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    o = oracle_mod.Oracle(oracle_mod.make_params(lx, ly, lz, rayleigh=2e4, periodic_sides=periodic))
    o.set_collision(collision)
    o.init_conduction(31, 1e-2)
    p = lbm.make_params(lx, ly, lz, rayleigh=2e4, storage=storage,
                        sides=lbm.SIDES_PERIODIC if periodic else lbm.SIDES_WALL)
    with lbm.Case(p) as c:
        c.set_collision(collision)
        c.init_conduction(31, 1e-2)
        for n in (1, 2, 3):
            o.step(1)
            c.step(1)
            got = c.store_ref_state(("f", "g"))
            for k in ("f", "g"):
                assert relerr(got[k], np.asarray(o.field(k))) <= 4 * (n + 1) * u, (k, n)
