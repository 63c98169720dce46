"""Rows and plane sums of observed steps at the warps where they part: rows
of nodes that fill warps, end inside them, and are shorter than one (a warp
over many x-rows, over a whole plane stack, and past the last node), few
planes (the six plane terms overlap), one and several reduction blocks.
Against lbm_get_observables of the same states; both sum in FP64, in other
orders: 1e-11 relative, as in the observed-step tests, and 1e-13 of the
temperature scale for Nu_top and Nu_bottom, LY times a difference of means."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f64", "f32", "f16s"])
@pytest.mark.parametrize("lx,ly,lz", [(2, 3, 2), (3, 4, 5), (7, 9, 3), (32, 3, 2), (33, 7, 5), (64, 5, 40), (40, 30, 70)])
def test_rows_match_the_reduction(lbm, storage, lx, ly, lz):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = lbm.make_params(lx, ly, lz, rayleigh=1e4, storage=storage, sides=lbm.SIDES_PERIODIC)
    with lbm.Case(p) as a, lbm.Case(p) as b:
        for c in (a, b):
            c.init_conduction(9, 1e-2)
        for _ in range(4):
            want = b.observables()
            b.step(1)
            got = a.step_observed(1)[0]
            for k in want:
                scale = abs(want[k]) + (1e-2 * ly if k in ("nu_top", "nu_bottom") else 1e-4)
                assert abs(got[k] - want[k]) <= 1e-11 * scale, (k, got[k], want[k])
