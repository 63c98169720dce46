"""The tile walk passes up to 32, or else about 140 to 190, members per launch
in its kernel parameters: batches on both sides of 32 and of the larger limit
(several launches per step), one block per tile and persistent blocks, equal
the single-case step bit for bit (FP64 and 16-bit storage)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f64", "f16s"])
@pytest.mark.parametrize("members,per_sm", [(32, 0), (33, 0), (200, 0), (200, 1)])
def test_members_over_several_launches(lbm, storage, members, per_sm):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    shapes = [(9, 4, 3), (33, 3, 2), (16, 8, 5)]

    def cases():
        out = []
        for i in range(members):
            c = lbm.Case(lbm.make_params(*shapes[i % 3], rayleigh=1e4 + 10 * i, storage=storage))
            c.set_collision("regularized" if i % 5 == 0 else "bgk")
            c.init_conduction(i, 1e-2)
            out.append(c)
        return out

    solo, batched = cases(), cases()
    for c in solo:
        c.step(3)
    with lbm.Batch(storage) as b:
        b.set_config(128, per_sm)
        for c in batched:
            b.add(c)
        b.step(1)
        b.step(2)
        for i, (x, y) in enumerate(zip(solo, batched)):
            want, got = x.store_ref_state(("f", "g", "phi")), y.store_ref_state(("f", "g", "phi"))
            for k in want:
                assert np.array_equal(want[k], got[k]), (i, k)
    for c in solo + batched:
        c.close()
