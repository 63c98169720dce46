"""Observed steps whose last block holds warps without nodes (up to three in
FP64, one in FP32 and 16-bit storage), with the rows' memory taken from
freed memory full of NaN: such a warp writes no plane sums, and none may be
read for it.  Nu_top and Nu_bottom (and the rest) against lbm_get_observables
of the same states, tolerances as for the rows of whole warps: both sum in
FP64 in other orders, 1e-11 relative, and 1e-13 of the temperature scale for
the plates' differences of means."""
import ctypes as C
import glob
import os

import pytest

pytestmark = pytest.mark.gpu


def _cudart():
    import torch

    site = os.path.dirname(os.path.dirname(torch.__file__))
    for name in glob.glob(os.path.join(site, "nvidia", "cuda_runtime", "lib", "libcudart.so*")):
        return C.CDLL(name)
    return C.CDLL("libcudart.so.12")


def _leave_nan_behind(sizes):
    """Blocks of these sizes, filled with NaN and freed (every other one, so
    the pages they came from stay with the process)."""
    rt = _cudart()
    blocks = []
    for size in sizes:
        for _ in range(16):
            p = C.c_void_p()
            assert rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0
            assert rt.cudaMemset(p, 0xFF, C.c_size_t(size)) == 0
            blocks.append(p)
    assert rt.cudaDeviceSynchronize() == 0
    for p in blocks[::2]:
        assert rt.cudaFree(p) == 0
    return rt, blocks[1::2]


@pytest.mark.parametrize("storage", ["f64", "f32", "f16s"])
@pytest.mark.parametrize("periodic", [True, False])
# nodes mod 128: 12, 3, 32, 36, 80, 16, 112; mod 64: 12, 3, 32, 36, 16, 16, 48
@pytest.mark.parametrize("lx,ly,lz", [(2, 3, 2), (33, 7, 5), (48, 5, 6), (20, 7, 3), (16, 5, 17), (40, 30, 70),
                                      (40, 6, 9)])
def test_no_plane_sums_past_the_last_node(lbm, storage, periodic, lx, ly, lz):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = lbm.make_params(lx, ly, lz, rayleigh=1e4, storage=storage,
                        sides=lbm.SIDES_PERIODIC if periodic else lbm.SIDES_WALL)
    with lbm.Case(p) as a, lbm.Case(p) as b:
        for c in (a, b):
            c.init_conduction(9, 1e-2)
        rows = -(-lx * ly * lz // 128) * 4   # 14 doubles each, and the partial sums behind them
        rt, kept = _leave_nan_behind([rows * 14 * 8 + 13 * 8 * (rows // 64 + k) for k in (1, 2)] + [512, 1 << 16])
        for _ in range(3):
            want = b.observables()
            b.step(1)
            got = a.step_observed(1)[0]
            for k in want:
                scale = abs(want[k]) + (1e-2 * ly if k in ("nu_top", "nu_bottom") else 1e-4)
                assert abs(got[k] - want[k]) <= 1e-11 * scale, (k, got[k], want[k])
        for q in kept:
            rt.cudaFree(q)
