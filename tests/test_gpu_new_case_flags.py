"""A case's error flag and count of finished blocks are clear before anything
reads them, though the case is created while the legacy default stream is
busy, initialised and read on a non-blocking stream, in memory that holds
something else."""
import numpy as np
import pytest

from test_gpu_obs_tail_rows import _leave_nan_behind

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["init", "restore"])
@pytest.mark.parametrize("n", [16, 40])
def test_new_case_beside_a_busy_default_stream(lbm, how, n):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = lbm.make_params(n, n, n, rayleigh=1e4, storage="f32")
    s = torch.cuda.Stream()
    with lbm.Case(p) as ref:
        ref.init_conduction(9, 1e-2, stream=s)
        want = ref.observables(stream=s)
        image = np.zeros(ref.checkpoint_bytes(), dtype=np.uint8)
        ref.save_state(image, stream=s)
        s.synchronize()
        rt, kept = _leave_nan_behind([1 << k for k in range(9, 20)])
        torch.cuda._sleep(400_000_000)   # a fifth of a second of the default stream
        with lbm.Case(p) as c:
            if how == "init":
                c.init_conduction(9, 1e-2, stream=s)
            else:
                c.restore_state(image, stream=s)
            got = [c.observables(stream=s) for _ in range(2)]
            torch.cuda.synchronize()
            got.append(c.observables(stream=s))
        assert got == [want] * 3
        for q in kept:
            rt.cudaFree(q)
