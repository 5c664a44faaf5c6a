"""Row-major fills on either side of the window length from which they go through
bulk copies; the same comparison with NumPy sums as the longer windows'."""

import pytest

from test_gpu_fill_bulk import test_row_major_fill as row_major_fill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 32, 47, 48, 49])
@pytest.mark.parametrize("B", [3, 2001])
def test_short_windows(M, B):
    row_major_fill(M, B)
