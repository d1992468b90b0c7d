"""The adjoint's transposed pull: all populations at once (the transposed sweep
and the adjoint Krylov operator) against one at a time."""
import pytest

import lbm_b200 as L

pytestmark = pytest.mark.gpu


# both walls in one cell's neighbourhood (2 and 3 columns), one row, one plane, a
# CTA's remainder
@pytest.mark.parametrize("shape", [(2, 1, 1), (2, 3, 4), (3, 1, 5), (4, 6, 1), (17, 5, 3), (33, 9, 10)])
@pytest.mark.parametrize("periodic", [False, True])
def test_all_populations_at_once(shape, periodic):
    assert L.selftest_transposed_pull(*shape, periodic) == 0


def test_refused_boxes():
    for shape in ((1, 4, 4), (4, 0, 4), (4, 4, 0), (4096, 4096, 2)):
        with pytest.raises(L.LBMError) as e:
            L.selftest_transposed_pull(*shape, False)
        assert e.value.status == 4
