"""The FP32 regularised step at the sizes where its two paths part (rows that
end inside, at and beyond a warp, few interior rows), both AA layouts, against
the FP64 oracle.  Tolerance: an FP32 step rounds a population in ~30
operations of relative 2^-24 on values within a factor 4 of the largest, and
passes an error on by a factor below 4: 4 * 30 * 2^-24 * (n + 1) after n
steps, relative to the largest."""
import numpy as np
import pytest

from helpers import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("lx,ly,lz", [(31, 6, 3), (33, 7, 5), (64, 5, 4), (65, 3, 2), (2, 4, 3)])
def test_reg32_against_the_oracle(lbm, oracle_mod, periodic, lx, ly, lz):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    o = oracle_mod.Oracle(oracle_mod.make_params(lx, ly, lz, rayleigh=2e4, periodic_sides=periodic))
    o.set_collision("regularized")
    o.init_conduction(31, 1e-2)
    p = lbm.make_params(lx, ly, lz, rayleigh=2e4, storage="f32",
                        sides=lbm.SIDES_PERIODIC if periodic else lbm.SIDES_WALL)
    with lbm.Case(p) as c:
        c.set_collision("regularized")
        c.init_conduction(31, 1e-2)
        for n in (1, 2, 3, 6):
            more = n - c.step_count
            o.step(more)
            c.step(more)
            got = c.store_ref_state(("f", "g"))
            for k in ("f", "g"):
                assert relerr(got[k], np.asarray(o.field(k))) <= 120 * 2.0 ** -24 * (n + 1), (k, n)
