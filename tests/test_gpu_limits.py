"""Calls at the limits of a launch, a row or the device: more slices than a grid dimension
holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_more_slices_than_a_launch_takes():
    """Slices too wide for the two-pass resize, more of them than a grid's y dimension: the
    ones past 65,535 too are resized and colored."""
    pytest.importorskip("cv2")
    from astroflow_b200 import postprocess
    from oracle import cv2_images as CVI

    target, width, n = 8, 2000, 70000
    raw = np.random.default_rng(7).integers(0, 1 << 20, (1, width + 16)).astype(np.uint32)
    d = torch.from_numpy(raw.view(np.int32)).cuda().view(torch.uint32)
    starts = np.arange(n) % 7
    got = postprocess.device_images(d, starts, np.full(n, width), target=target).cpu().numpy()
    want = np.stack([CVI.image(raw[:, s:s + width], target) for s in range(7)])
    assert np.array_equal(got, want[starts])
