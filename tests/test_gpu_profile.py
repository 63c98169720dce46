"""The vertical profile over its split into chunks per plane, against the
same averages of the exported fields: planes smaller than a block, of one
and of several uneven chunks, few and many planes.  The fields are exact
copies of what the kernel averages (FP64, and FP32 read exactly), so only
the order of ~1e4 FP64 additions differs: 1e4 * 2^-53, and its square root in
the rms, a difference of squares."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("lx,ly,lz", [(2, 3, 2), (16, 5, 16), (33, 4, 31), (100, 3, 77), (5, 300, 3)])
def test_profile_is_the_plane_average(lbm, storage, periodic, lx, ly, lz):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = lbm.make_params(lx, ly, lz, rayleigh=1e4, storage=storage,
                        sides=lbm.SIDES_PERIODIC if periodic else lbm.SIDES_WALL)
    with lbm.Case(p) as c:
        c.init_conduction(3, 1e-2)
        for steps in (2, 1):   # both layouts
            c.step(steps)
            s = c.store_ref_state(("ux", "uy", "uz", "phi"))
            got = c.profile()
            for k, name in enumerate(("ux", "uy", "uz", "phi")):
                assert np.max(np.abs(got[:, k] - s[name].mean(axis=(0, 2)))) <= 1e4 * 2.0 ** -53, name
            rms = s["phi"].std(axis=(0, 2))
            assert np.max(np.abs(got[:, 4] - rms)) <= (1e4 * 2.0 ** -53) ** 0.5
