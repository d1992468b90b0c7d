"""The work list that two-sweep passes of a batch get before each segment."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


# boxes with and without remainders of the 32 x 8 tile, of one cell in y and z,
# of fewer planes than the shortest run; they leave at different checks, in
# another order than they are listed, until one is left
@pytest.mark.parametrize("zrun", [1, 5, 64])
def test_uneven_batch_equals_single_sweeps(zrun):
    shapes = [(32, 8, 40), (70, 9, 33), (2, 1, 1), (33, 17, 3), (5, 40, 66), (64, 24, 16), (31, 7, 130)]
    boxes = [wavy_box(s, i % 2) for i, s in enumerate(shapes)]
    counts = [[30, 60, 10, 50, 20, 10, 40], [10, 20, 60, 30, 10, 50, 20]]
    got = []
    for z in (0, zrun):
        b = L.Batch([p for p, _ in boxes], [f for _, f in boxes])
        b.set_tuning(32, 8, 4, 4, z)
        b.set_poisson(check_interval=10)
        b.step_replay(counts)
        got.append([b.download_fields(i) for i in range(len(boxes))])
        b.close()
    for i in range(len(boxes)):
        for k in L.FIELDS:
            assert np.array_equal(got[0][i][k], got[1][i][k]), (i, k)
