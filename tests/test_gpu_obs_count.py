"""The reductions' count of finished blocks after a misuse: reductions of one
case enqueued on two streams at once spoil each other's records (the header
forbids it), but once both are done, later calls report the state they are
given: the count is a multiple of the blocks again, whatever the order in
which the blocks counted."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f64", "f16s"])
@pytest.mark.parametrize("n", [32, 64])
def test_a_misused_call_does_not_spoil_later_ones(lbm, storage, n):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    p = lbm.make_params(n, n, n, rayleigh=1e4, storage=storage)
    gate, s1, s2 = (torch.cuda.Stream() for _ in range(3))
    with lbm.Case(p) as a, lbm.Case(p) as b, lbm.Batch(storage) as batch:
        for c in (a, b):
            c.init_conduction(9, 1e-2)
        batch.add(a)
        spoilt = lbm.ObservablesBuffer(1)
        for i in range(24):
            for late in range(1000 * i, 1000 * i + 1000, 250):   # cycles by which one starts after the other
                with torch.cuda.stream(gate):
                    torch.cuda._sleep(200_000)
                for s in (s1, s2):
                    s.wait_stream(gate)
                    if s is s2:
                        with torch.cuda.stream(s):
                            torch.cuda._sleep(late)
                    for _ in range(4):
                        batch.observables_async(spoilt, stream=s)
                torch.cuda.synchronize()
            batch.step(1)
            b.step(1)
            torch.cuda.synchronize()
            assert a.observables() == b.observables()
            batch.observables_async(spoilt, stream=s1)
            s1.synchronize()
            assert spoilt[0] == b.observables()
