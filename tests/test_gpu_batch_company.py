"""A subset's results do not depend on the batch it is solved in, to the last
bit, at either precision."""
import numpy as np
import pytest

import matrices as M
from gpu_util import upload
from single_svdlib import randomized

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("rank,over", [(10, 7), (30, 10), (5, 3)])
def test_same_bits_alone_and_with_others(rank, over, precision):
    A = upload("csr", M.poisson_rows(5003, 611, 12, 9))
    rng = np.random.default_rng(3)
    subsets = [np.sort(rng.choice(611, int(k), replace=False)) for k in rng.integers(60, 500, 40)]

    def solve(which):
        return randomized.RandomizedBatch(A, [subsets[i] for i in which], rank, over, 1, seed=5,
                                          precision=precision).run()

    alone = {i: solve([i])[0] for i in (0, 1)}
    for which in ([1, 0], [0, 1, 2, 3, 4, 5, 6], [1] + list(range(2, 40)) + [0]):
        got = solve(which)
        for i in (0, 1):
            r = got[which.index(i)]
            for name in ("u", "s", "vt"):
                np.testing.assert_array_equal(getattr(r, name), getattr(alone[i], name), err_msg=f"{name} of {i} in {len(which)}")
