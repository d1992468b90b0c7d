"""Both tiles of a batch's two-sweep passes: bitwise the single sweeps."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


# rows that whole 32 x 8 tiles cover, and rows of which they would leave a third
# or more empty (16 x 8 then); remainders in y and z, one plane
@pytest.mark.parametrize("shapes", [[(64, 9, 33), (32, 40, 10), (96, 8, 70), (32, 17, 1)],
                                    [(48, 9, 33), (16, 40, 10), (33, 8, 70), (7, 17, 1), (80, 5, 20)]])
@pytest.mark.parametrize("zrun", [7, 32])
def test_tiles_of_the_two_sweep_passes(shapes, zrun):
    boxes = [wavy_box(s, i % 2) for i, s in enumerate(shapes)]
    counts = [[20 + 10 * (3 * i % 5) for i in range(len(shapes))], [40] * len(shapes)]
    got = []
    for z in (0, zrun):
        b = L.Batch([p for p, _ in boxes], [f for _, f in boxes])
        b.set_tuning(32, 8, 4, 4, z)
        b.set_poisson(check_interval=10)
        b.step_replay(counts)
        got.append([b.download_fields(i) for i in range(len(boxes))])
        assert (b.timing()["fused_sweeps"] > 0) == (z > 0)
        b.close()
    for i in range(len(boxes)):
        for k in L.FIELDS:
            assert np.array_equal(got[0][i][k], got[1][i][k]), (i, k)
