"""Steps launched to overlap the end of the previous kernel: small grids
(where the next launch is waiting before the last one is done), plain and
observed steps mixed, other work of the stream before and after, and a
captured graph, against the same steps with a device synchronisation after
each.  Bitwise: the same kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(c):
    s = c.store_ref_state(("f", "g", "phi"))
    return np.concatenate([s[k].reshape(-1) for k in ("f", "g", "phi")])


@pytest.mark.parametrize("storage", ["f64", "f32", "f16s", "bf16s"])
@pytest.mark.parametrize("lx,ly,lz", [(2, 3, 2), (32, 32, 32), (65, 40, 33)])
def test_overlapped_steps_are_the_same_steps(lbm, storage, lx, ly, lz):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = lbm.make_params(lx, ly, lz, rayleigh=2e4, storage=storage)
    with lbm.Case(p) as a, lbm.Case(p) as b:
        for c in (a, b):
            c.init_conduction(4, 1e-2)
        want = []
        for i in range(60):
            if i % 7 == 3:
                want += b.step_observed(1)
            else:
                b.step(1)
            torch.cuda.synchronize()
        got = []
        i = 0
        while i < 60:
            if i % 7 == 3:
                got += a.step_observed(1)
                i += 1
            else:
                n = 1
                while (i + n) % 7 != 3 and i + n < 60:
                    n += 1
                a.step(n)
                i += n
        assert np.array_equal(_state(a), _state(b))
        assert got == want


def test_captured_steps_replay(lbm):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = lbm.make_params(40, 16, 24, rayleigh=2e4, storage="f32")
    x, y = torch.zeros(1 << 20, device="cuda"), torch.ones(1 << 20, device="cuda")
    with lbm.Case(p) as a, lbm.Case(p) as b:
        for c in (a, b):
            c.init_conduction(4, 1e-2)
            c.step(2)
        s = torch.cuda.Stream()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            x.copy_(y)
            b.step(4, stream=s)
            y.mul_(2.0)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        a.step(12)
        assert np.array_equal(_state(a), _state(b))
