"""The combining of a system's partials by the warp that arrives last: its 32
lanes load what other blocks wrote, behind lane 0's acquire and a warp barrier.
A partial read too early is one of an earlier phase, which moves a dot and with
it the iterates, so solves of the same systems have to give the same bits every
time.  Systems of more segments than a warp has lanes, and of one segment."""
import numpy as np
import pytest

from conftest import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides", [(180,), (150, 4, 90, 3, 33), (12, 70, 9, 70, 5, 70, 8, 70)])
def test_solves_repeat_bit_for_bit(native, ctx, problems, sides):
    systems = [problems.config0(side=side, bs=1 + i % 4, seed=20 + i) for i, side in enumerate(sides)]
    batch = native.Batch(ctx, systems)
    rhs = np.concatenate([s.rhs for s in systems])
    b = native.Vector(ctx, rhs.size, 0, 1).upload(rhs)
    x = native.Vector(ctx, rhs.size, 0, 1)
    first = None
    for run in range(12):
        x.fill(0.0)
        results = [{k: v for k, v in r.as_dict().items() if k != "solve_seconds"} for r in batch.solve(b, x)]
        assert results[0]["status"] == 0
        if first is None:
            first = x.download(), results
        assert_bitwise(x.download(), first[0], f"solve {run}")
        assert results == first[1], f"solve {run}"
