"""Batches that are stepped from tables in global memory (persistent blocks,
and more members than one launch's parameters hold, if they are small) and
the changes between the two ways: members beyond a table's first size,
members leaving, another block size, persistent blocks on and off, the
per-case launch in between.  Bitwise the single-case step, FP64 and 16-bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f64", "f16s"])
def test_table_steps_are_the_single_case_steps(lbm, storage):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    shapes = [(9, 4, 3), (33, 3, 2), (16, 8, 5), (40, 10, 12)]

    def case(i):
        c = lbm.Case(lbm.make_params(*shapes[i % 4], rayleigh=1e4 + 10 * i, storage=storage))
        c.set_collision("regularized" if i % 7 == 0 else "bgk")
        c.init_conduction(i, 1e-2)
        return c

    solo, batched = [case(i) for i in range(420)], [case(i) for i in range(420)]
    with lbm.Batch(storage) as b:
        def run(n):
            for c in solo[:len(b.members)]:
                c.step(n)
            b.step(n)

        for c in batched[:20]:
            b.add(c)
        b.set_config(128, 2)            # tables for few members
        run(3)
        for x, y in zip(solo[20:], batched[20:]):
            x.step(2)                   # in the other layout than the first members
            y.step(2)
            b.add(y)
        run(2)
        for i in range(0, 420, 3):
            b.remove(batched[i])
            b.add(batched[i])
        run(1)
        b.set_config(128, 0)            # tables for many
        run(3)
        b.set_config(256, 0)
        run(1)
        b.set_launch("per_case")
        run(2)
        b.set_launch("tiles")
        run(2)
        b.set_config(256, 3, False)
        run(2)
        for i, (x, y) in enumerate(zip(solo, batched)):
            want, got = x.store_ref_state(("f", "g", "phi")), y.store_ref_state(("f", "g", "phi"))
            for k in want:
                assert np.array_equal(want[k], got[k]), (i, k)
    for c in solo + batched:
        c.close()
