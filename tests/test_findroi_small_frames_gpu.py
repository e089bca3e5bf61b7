"""Boxes larger than the frame: the crop stays inside the stack."""
import numpy as np
import pytest

from bamf_gb300 import frontend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ys,xs", [(7, 7), (16, 7), (7, 16), (5, 5)])
def test_crops_of_frames_smaller_than_the_box(cuda_lib, ys, xs):
    rng = np.random.default_rng(ys * xs)
    st = rng.poisson(5.0, (ys, xs, 6)).astype(np.float32)
    st[ys // 2, xs // 2, :] += 4000.0  # a maximum in every frame, the first among them
    SMD, rois, coords = frontend.findROI(st, 1.3, 2.6, 8, 1.0)
    assert (coords[:, 2] == 1).any()
    flat = np.ascontiguousarray(st.ravel(order="F"))
    for b in range(len(coords)):
        col, row = np.meshgrid(np.arange(8), np.arange(8))
        at = ((coords[b, 2] - 1) * ys * xs + (SMD["XBoxCorner"][b] - 1 + col) * ys + SMD["YBoxCorner"][b] - 1 + row)
        want = np.where(at >= 0, flat[np.maximum(at, 0)], 0.0)
        np.testing.assert_array_equal(rois[:, :, b], want)
