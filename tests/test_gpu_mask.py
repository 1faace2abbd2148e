"""GPU parity of the hit-mask culling path (cf_mask.cu), bit for bit against
the oracle: light counts around a list segment's and a mask's edges, grids
whose slices end in a short group or hold a single cluster, more survivors
than a warp keeps masks for (the second scan), lists that reach the cap in the
middle of a mask, non-finite lights in a mask of finite ones."""
import numpy as np
import pytest

from gpu_helpers import assert_matches_oracle, run_pipeline
from hellovulkan_gb300 import scenes
from test_gpu_fuzz import mismatch, random_view

pytestmark = pytest.mark.gpu

MASK = (4, 8, 32, 1, 1)


@pytest.mark.parametrize("n_lights", [0, 1, 31, 33, 255, 256, 257, 2049, 4096, 4097, 8192, 8193])
def test_light_counts_around_segments(gpu, oracle, n_lights):
    rng = np.random.default_rng(41 + n_lights)
    v = scenes.custom_view((15, 9, 17), 1920, 1080, 0.1, 300.0,
                           lights=scenes.uniform_box_lights(rng, n_lights, [-30, -15, -60], [30, 15, -5], 1.0, 6.0))
    assert_matches_oracle(oracle, v, *run_pipeline(gpu, v, MASK))


@pytest.mark.parametrize("grid", [(1, 1, 1), (1, 1, 40), (31, 1, 7), (32, 1, 2), (33, 1, 16), (8, 8, 33), (64, 36, 24)])
def test_group_and_slice_edges(gpu, oracle, grid):
    rng = np.random.default_rng(sum(grid))
    lights = scenes.uniform_box_lights(rng, 700, [-30, -15, -60], [30, 15, 2], 0.5, 8.0)
    lights[[3, 100, 301], 0] = np.nan
    lights[7, 1], lights[9, 2], lights[600, 2] = np.inf, -np.inf, np.nan
    v = scenes.custom_view(grid, 1920, 1080, 0.1, 300.0, lights=lights)
    assert_matches_oracle(oracle, v, *run_pipeline(gpu, v, MASK))


@pytest.mark.parametrize("cap", [1, 31, 150, 4096])
@pytest.mark.parametrize("radius", [(0.02, 0.3), (30.0, 60.0)])
def test_more_survivors_than_kept_masks(gpu, oracle, cap, radius):
    """9000 lights inside two slices of two groups: small ones reach few
    clusters each (every warp sees far more survivors than it keeps masks
    for, and tests them again to write them), large ones reach all of them."""
    rng = np.random.default_rng(cap)
    v = scenes.custom_view((8, 8, 2), 512, 512, 5.0, 60.0, cap=cap,
                           lights=scenes.uniform_box_lights(rng, 9000, [-6, -6, -50], [6, 6, -6], *radius))
    assert_matches_oracle(oracle, v, *run_pipeline(gpu, v, MASK))


def test_random_views(gpu, oracle):
    rng = np.random.default_rng(43)
    failures = []
    for case in range(60):
        v = random_view(rng)
        m = mismatch(oracle, v, *run_pipeline(gpu, v, MASK))
        if m:
            failures.append((case, v.name, m))
    assert not failures, failures[:5]


def borderline_lights(oracle, view, n, seed):
    """n lights, each with the smallest radius whose square reaches its squared
    distance to some cluster's box (float32, each product and sum rounded):
    half of them then touch that box by an ulp or not at all, and a sum
    rounded once instead of twice decides otherwise."""
    rng = np.random.default_rng(seed)
    a = oracle.generate_aabbs(view.ubo)
    pos = rng.uniform([-30, -15, -60], [30, 15, -5], size=(n, 3)).astype(np.float32)
    box = a[rng.integers(0, a.shape[0], n)]
    d = np.maximum(np.maximum(box[:, 0:3] - pos, pos - box[:, 4:7]), np.float32(0))
    sq = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
    r = np.sqrt(sq)
    for _ in range(2):
        low = np.nextafter(r, np.float32(0))
        r = np.where(low * low >= sq, low, r)
    r = np.where(r * r < sq, np.nextafter(r, np.float32(np.inf)), r)
    return scenes.make_lights(pos, r)


def test_sums_are_rounded_as_the_shader_rounds_them(gpu, oracle):
    import torch

    from hellovulkan_gb300.batch import Batch, BatchBuffers
    v = scenes.custom_view((32, 18, 24), 2560, 1440, 0.1, 300.0)  # identity view: positions are view space
    v.lights = borderline_lights(oracle, v, 6000, 47)
    assert_matches_oracle(oracle, v, *run_pipeline(gpu, v, MASK))
    bufs = BatchBuffers([v])
    b = Batch(gpu)
    b.set_views(bufs.batch_views())
    s = torch.cuda.Stream()
    b.generate_aabbs(s)
    b.cull(s)
    assert_matches_oracle(oracle, v, *bufs.read(0))
    b.close()


@pytest.mark.parametrize("grid", [(8, 8, 2), (15, 9, 13), (33, 1, 7), (5, 1, 255), (3, 1, 257)])
def test_batches_of_few_and_many_units(gpu, oracle, grid):
    """A batch whose groups have from no unit to more than a warp adds up by
    itself (eight of 128 candidates), side by side in one block, with slices
    that the quick test of four at a time passes over; numbers of groups and of
    slices that are no multiple of four; the most slices of the hit-mask path
    and one more."""
    from hellovulkan_gb300.batch import Batch, BatchBuffers
    views = []
    for n in (0, 90, 1100, 3000):
        rng = np.random.default_rng(n)
        near = scenes.uniform_box_lights(rng, n, [-3, -2, -4], [3, 2, -3.5], 0.1, 0.6)
        far = scenes.uniform_box_lights(rng, 60, [-60, -30, -200], [60, 30, -5], 1.0, 9.0)
        views.append(scenes.custom_view(grid, 1920, 1080, 0.1, 300.0, lights=np.concatenate([far[:30], near, far[30:]])))
    bufs = BatchBuffers(views)
    b = Batch(gpu)
    b.set_views(bufs.batch_views())
    b.generate_aabbs()
    b.cull()
    for q, v in enumerate(views):
        assert_matches_oracle(oracle, v, *bufs.read(q))
    b.close()


@pytest.mark.parametrize("grid", [(16, 9, 24), (33, 1, 13)])
def test_boxes_of_other_shapes(gpu, oracle, grid):
    """Boxes that a caller made, not the generator: z bounds that differ within
    a group (no squared z distance to share), one group whose bounds differ in
    a single cluster, a box with a NaN bound; in a batch, and with more lights
    than a warp's groups of few units go with."""
    from hellovulkan_gb300.batch import Batch, BatchBuffers
    rng = np.random.default_rng(53)
    views = [scenes.custom_view(grid, 1920, 1080, 0.1, 300.0,
                                lights=scenes.uniform_box_lights(rng, n, [-30, -15, -60], [30, 15, -5], 1.0, 6.0))
             for n in (300, 9000)]
    bufs = BatchBuffers(views)
    b = Batch(gpu)
    b.set_views(bufs.batch_views())
    b.generate_aabbs()
    given = []
    for q, v in enumerate(views):
        a = oracle.generate_aabbs(v.ubo)
        xy = grid[0] * grid[1]
        a[:5 * xy, 2] -= rng.uniform(0, 2, 5 * xy).astype(np.float32)
        a[5 * xy: 9 * xy, 6] += rng.uniform(0, 1, 4 * xy).astype(np.float32)
        a[9 * xy + 7, 6] += np.float32(0.5)
        a[10 * xy + 3, 0] = np.nan
        import torch
        bufs.aabbs[q].copy_(torch.from_numpy(a).reshape(bufs.aabbs[q].shape))
        given.append(a)
    b.cull()
    for q, v in enumerate(views):
        _, cells, idx = bufs.read(q)
        oc, oi, _ = oracle.cull(v.ubo, given[q], v.lights, v.cap)
        assert np.array_equal(cells, oc) and np.array_equal(idx, oi), q
    b.close()


@pytest.mark.parametrize("grid", [(8, 8, 16), (16, 9, 24), (8, 10, 30)])
@pytest.mark.parametrize("n_lights", [2303, 2304])
def test_the_line_between_brute_force_and_hit_masks(gpu, oracle, grid, n_lights):
    """More lights than one launch takes, on both sides of the line: the chosen
    kernels, and their output."""
    from hellovulkan_gb300.pipelines import PipelineLightCulling, ResourcesClusterForward, ResourcesLight
    rng = np.random.default_rng(n_lights)
    v = scenes.custom_view(grid, 1920, 1080, 0.1, 300.0,
                           lights=scenes.uniform_box_lights(rng, n_lights, [-30, -15, -60], [30, 15, -5], 1.0, 6.0))
    rl, rc = ResourcesLight(gpu), ResourcesClusterForward(gpu)
    rl.add_lights(v.lights)
    rc.create_buffers(*v.grid, v.cap)
    cull = PipelineLightCulling(gpu, rl, rc)
    cull.set_cluster_forward_ubo(v.ubo)
    if n_lights == 2304:
        assert cull.tuning() == MASK
    else:
        assert cull.tuning()[4] == 0
    for o in (cull, rc, rl):
        o.close()
    assert_matches_oracle(oracle, v, *run_pipeline(gpu, v))
