"""gaussMLE reads its array's values in Fortran order whatever the array's memory order: square windows,
and the first sz x sz values of one window that is wider than high."""
import numpy as np
import pytest

from bamf_gb300 import frontend

pytestmark = pytest.mark.gpu


def test_order_of_a_stack_that_is_copied_in_pieces(cuda_lib):
    """Above 256 MB a C-ordered stack goes to the device in pieces; the last one here is short."""
    rng = np.random.default_rng(2)
    g = np.arange(21) - 10
    base = rng.poisson(20 + 300 * np.exp(-(g[:, None, None] ** 2 + g[None, :, None] ** 2) / 3.4) +
                       np.zeros((1, 1, 997))).astype(np.float32)
    d = np.tile(base, (1, 1, 161))[:, :, :160_005]  # 282 MB
    want = frontend.gaussMLE(np.asfortranarray(base), "Basic", "CCD", 1.3, Iterations=2)
    got = frontend.gaussMLE(np.ascontiguousarray(d), "Basic", "CCD", 1.3, Iterations=2)
    for k in want:
        np.testing.assert_array_equal(got[k], np.tile(want[k], 161)[:160_005], err_msg=k)


@pytest.mark.parametrize("rows,cols,n", [(7, 7, 1), (7, 7, 40), (7, 9, 1), (8, 21, 1), (7, 9, 5), (1, 3, 2)])
def test_memory_order_does_not_matter(cuda_lib, rows, cols, n):
    rng = np.random.default_rng(rows * cols + n)
    a = np.arange(rows)[:, None, None] - (rows - 1) / 2, np.arange(cols)[None, :, None] - (rows - 1) / 2
    d = rng.poisson(20 + 300 * np.exp(-(a[0] ** 2 + a[1] ** 2) / 3.4) + np.zeros((1, 1, n))).astype(np.float32)
    for fit in ("Basic", "Sigma"):
        want = frontend.gaussMLE(np.asfortranarray(d), fit, "CCD", 1.3)
        got = frontend.gaussMLE(np.ascontiguousarray(d), fit, "CCD", 1.3)
        for k in want:
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"{fit} {k}")
