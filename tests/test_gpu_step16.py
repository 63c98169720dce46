"""The 16-bit step at the sizes where its paths part: rows that end inside,
at and beyond a warp, x-wall nodes alone in a warp, few interior rows, after
odd and even step counts (both AA layouts), with both collision models.

Tolerance: each step rounds every stored value once, to u = 2^-11 (FP16) or
2^-8 (BF16) relative, on top of the rounding of the start; one step passes
an error on by a factor below 4 (|1 - 1/tau| <= 1 per population and the
moments' share in the equilibria).  So after n <= 5 steps the populations
are within 4 (n + 1) u of the oracle's, relative to the largest."""
import numpy as np
import pytest

from helpers import relerr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("storage,u", [("f16s", 2.0 ** -11), ("bf16s", 2.0 ** -8)])
@pytest.mark.parametrize("collision", ["bgk", "regularized"])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("lx,ly,lz", [(31, 6, 3), (33, 7, 5), (64, 5, 4), (65, 3, 2), (96, 4, 7)])
def test_step16_against_the_oracle(lbm, oracle_mod, storage, u, collision, periodic, lx, ly, lz):
    o = oracle_mod.Oracle(oracle_mod.make_params(lx, ly, lz, rayleigh=2e4, periodic_sides=periodic))
    o.set_collision(collision)
    o.init_conduction(31, 1e-2)
    p = lbm.make_params(lx, ly, lz, rayleigh=2e4, storage=storage,
                        sides=lbm.SIDES_PERIODIC if periodic else lbm.SIDES_WALL)
    with lbm.Case(p) as c:
        c.set_collision(collision)
        c.init_conduction(31, 1e-2)
        for n in (1, 2, 3, 5):
            more = n - c.step_count
            o.step(more)
            c.step(more)
            got = c.store_ref_state(("f", "g"))
            for k in ("f", "g"):
                assert relerr(got[k], np.asarray(o.field(k))) <= 4 * (n + 1) * u, (k, n)


@pytest.mark.parametrize("storage", ["f16s", "bf16s"])
@pytest.mark.parametrize("collision", ["bgk", "regularized"])
def test_tile_walk_is_bitwise_the_single_case_step(lbm, storage, collision):
    """Both kernels inline the same 16-bit update."""
    shapes = [(33, 7, 5), (64, 5, 4), (160, 16, 9)]
    pairs = []
    for i, s in enumerate(shapes):
        both = [lbm.Case(lbm.make_params(*s, rayleigh=1e5, storage=storage)) for _ in range(2)]
        for c in both:
            c.set_collision(collision)
            c.init_conduction(40 + i, 1e-2)
        both[0].step(5)
        pairs.append(both)
    with lbm.Batch(storage) as b:
        for _, c in pairs:
            b.add(c)
        b.step(5)
        for x, y in pairs:
            want, got = x.store_ref_state(("f", "g", "phi")), y.store_ref_state(("f", "g", "phi"))
            for k in want:
                assert np.array_equal(want[k], got[k]), k
    for both in pairs:
        for c in both:
            c.close()
