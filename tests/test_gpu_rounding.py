"""Every culling kernel rounds each product and each sum by itself, as the
shader's arithmetic does: lights whose radius only just reaches a cluster's
box, so that a sum rounded once instead of twice moves a light in or out of a
list, and cameras whose rotation and translation make the light transform round
too.  Bit for bit against the oracle."""
import numpy as np
import pytest

from gpu_helpers import assert_matches_oracle, run_pipeline
from hellovulkan_gb300 import scenes
from hellovulkan_gb300.camera import look_at_rh
from test_gpu_mask import MASK
from test_gpu_one_launch import SHAPES, one_launch_tuning
from test_gpu_parity import TUNINGS

pytestmark = pytest.mark.gpu

CAMERAS = [np.eye(4, dtype=np.float32), look_at_rh((3.7, 2.3, 11.9), (0.6, -1.3, -20.1))]


def borderline_view(oracle, camera, n, seed):
    """A view of n lights, each with the smallest radius whose square reaches
    its squared distance to some cluster's box: half of them touch that box by
    an ulp or not at all."""
    view = scenes.custom_view((16, 9, 24), 1920, 1080, 0.1, 300.0, view=camera)
    rng = np.random.default_rng(seed)
    world = rng.uniform([-30, -15, -60], [30, 15, -5], size=(n, 3)).astype(np.float32)
    m = np.array(list(view.ubo.cameraView), np.float32)  # column major
    x, y, z = world.T
    pos = np.stack([((m[r] * x + m[4 + r] * y) + m[8 + r] * z) + m[12 + r] for r in range(3)], axis=1)
    a = oracle.generate_aabbs(view.ubo)
    box = a[rng.integers(0, a.shape[0], n)]
    d = np.maximum(np.maximum(box[:, 0:3] - pos, pos - box[:, 4:7]), np.float32(0))
    sq = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
    r = np.sqrt(sq)
    for _ in range(2):
        low = np.nextafter(r, np.float32(0))
        r = np.where(low * low >= sq, low, r)
    r = np.where(r * r < sq, np.nextafter(r, np.float32(np.inf)), r)
    assert r.dtype == np.float32
    view.lights = scenes.make_lights(world, r)
    return view


@pytest.mark.parametrize("camera", [0, 1])
@pytest.mark.parametrize("tuning", ["auto", MASK] + SHAPES + TUNINGS)
def test_lights_on_the_border_of_a_box(gpu, oracle, tuning, camera):
    for seed in (3, 4, 5):
        v = borderline_view(oracle, CAMERAS[camera], 1000, seed)
        t = None if tuning == "auto" else tuning
        if tuning in SHAPES:
            t = one_launch_tuning(v.clusters, v.light_count, None, tuning)
        assert_matches_oracle(oracle, v, *run_pipeline(gpu, v, t))
