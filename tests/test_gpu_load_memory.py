"""lbm_load_ref_state where the device has room for the FP64 values of one
field but not of two, as it has always needed: the state is bitwise the one
loaded with room to spare."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "ux", "uy", "uz", "phi", "f", "g")


@pytest.mark.parametrize("storage", ["f64", "f16s"])
def test_load_with_little_device_memory(lbm, storage):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from test_gpu_obs_tail_rows import _cudart

    rt = _cudart()
    p = lbm.make_params(127, 96, 129, rayleigh=1e5, storage=storage)
    with lbm.Case(p) as c:
        c.init_conduction(5, 1e-2)
        c.step(4)
        state = c.store_ref_state()
        images = []
        for room in (None, 12 * c.n):
            fill = C.c_void_p()
            if room:
                c.init_conduction(6, 1e-2)   # something else
                torch.cuda.empty_cache()
                free, total = C.c_size_t(), C.c_size_t()
                assert rt.cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
                assert rt.cudaMalloc(C.byref(fill), C.c_size_t(free.value - room)) == 0
            try:
                c.load_ref_state(*[state[k] for k in FIELDS])
            finally:
                rt.cudaFree(fill)
            images.append(np.zeros(c.checkpoint_bytes(), dtype=np.uint8))
            c.save_state(images[-1])
            torch.cuda.synchronize()
        pops = 256 + 2 * 27 * -(-c.n // 128) * 128 * (8 if storage == "f64" else 2)
        row = c.n * (8 if storage == "f64" else 4)
        assert np.array_equal(images[0][:256], images[1][:256])
        assert np.array_equal(images[0][pops:pops + row], images[1][pops:pops + row])
        got = c.store_ref_state()
        c.load_ref_state(*[state[k] for k in FIELDS])
        want = c.store_ref_state()
        for k in FIELDS:
            assert np.array_equal(got[k], want[k]), k
