"""Views in which more lights than a list holds reach whole depth slices: the
hit-mask kernels end such a slice's candidates where its lists are full for
certain, with the oracle's lists bit for bit."""
import numpy as np
import pytest

from gpu_helpers import assert_matches_oracle, run_pipeline
from hellovulkan_gb300 import scenes
from test_gpu_mask import MASK

pytestmark = pytest.mark.gpu


def view(grid, n, radius, cap, seed=61):
    rng = np.random.default_rng(seed + n)
    return scenes.custom_view(grid, 1920, 1080, 0.1, 300.0, cap=cap,
                              lights=scenes.uniform_box_lights(rng, n, [-40, -40, -40], [40, 40, 40], *radius))


def pad(n):  # lights as the kernels' arrays hold them, at most
    return -(-n // 1024) * 1024


# segments of 256, 512 and 1024 lights; caps below, at and above what a warp or a segment holds
@pytest.mark.parametrize("n", [300, 3000, 6000, 9000])
@pytest.mark.parametrize("cap", [1, 31, 32, 150, 256, 1500])
def test_lights_that_reach_everything(gpu, oracle, n, cap):
    from hellovulkan_gb300.pipelines import (PipelineAABBGenerator, PipelineLightCulling, ResourcesClusterForward,
                                             ResourcesLight)
    v = view((9, 7, 20), n, (900.0, 2000.0), cap)
    rl, rc = ResourcesLight(gpu), ResourcesClusterForward(gpu)
    rl.add_lights(v.lights)
    rc.create_buffers(*v.grid, v.cap)
    gen = PipelineAABBGenerator(gpu, rc)
    gen.set_cluster_forward_ubo(v.ubo)
    gen.fill_command_buffer()
    cull = PipelineLightCulling(gpu, rl, rc)
    cull.set_tuning(*MASK)
    cull.set_cluster_forward_ubo(v.ubo)
    cull.enable_work_counters()
    cull.fill_command_buffer()
    cells, idx = rc.read_outputs()
    assert_matches_oracle(oracle, v, rc.read_aabbs(), cells, idx)
    # every light against every slice, then of each slice no more than the lights that fill its lists, up to the
    # end of a warp's 32 where one segment of 256 has them, else of a segment of at most 1024, against two groups
    tests, _ = cull.read_work_counters()
    needed = min(-(-cap // 32) * 32 if cap <= 256 else -(-cap // 1024) * 1024, pad(n))
    assert tests <= 20 * pad(n) + 20 * 2 * needed
    for o in (cull, gen, rc, rl):
        o.close()


@pytest.mark.parametrize("grid", [(9, 7, 20), (33, 1, 40), (1, 1, 256)])
@pytest.mark.parametrize("n", [1200, 5000, 20000])
@pytest.mark.parametrize("cap", [20, 150, 1500])
def test_lights_that_reach_the_near_slices(gpu, oracle, grid, n, cap):
    """Some slices full after one segment, some after several, some never; a
    few lights with odd values among them."""
    v = view(grid, n, (15.0, 70.0), cap)
    v.lights[::97, 0], v.lights[5::211, 8], v.lights[7::331, 2], v.lights[11::173, 8] = np.nan, np.inf, -np.inf, np.nan
    assert_matches_oracle(oracle, v, *run_pipeline(gpu, v, MASK))


@pytest.mark.parametrize("slices", [1, 3, 4])
def test_few_slices_are_left_to_the_other_kernels(gpu, oracle, slices):
    from hellovulkan_gb300.batch import Batch, BatchBuffers
    from hellovulkan_gb300.pipelines import PipelineLightCulling, ResourcesClusterForward, ResourcesLight
    v = view((30, 20, slices), 9000, (1.0, 60.0), 20)
    rl, rc = ResourcesLight(gpu), ResourcesClusterForward(gpu)
    rl.add_lights(v.lights)
    rc.create_buffers(*v.grid, v.cap)
    cull = PipelineLightCulling(gpu, rl, rc)
    cull.set_cluster_forward_ubo(v.ubo)
    assert (cull.tuning() == MASK) == (slices == 4)
    for o in (cull, rc, rl):
        o.close()
    assert_matches_oracle(oracle, v, *run_pipeline(gpu, v))
    bufs = BatchBuffers([v])
    b = Batch(gpu)
    b.set_views(bufs.batch_views())
    assert (b.info()["bucket_configs"][0]["config"] == list(MASK[:4])) == (slices == 4)
    b.generate_aabbs()
    b.cull()
    assert_matches_oracle(oracle, v, *bufs.read(0))
    b.close()


@pytest.mark.parametrize("n", [2000, 9000])
def test_boxes_the_wrong_way_round(gpu, oracle, n):
    """A box whose lower bounds lie above its upper ones is further from a
    light than any corner of its slice's box need be (all kernels take the
    larger of its two distances, the shader their sum); with it, boxes without
    extent, infinite ones and NaN bounds.  The hit masks against the staged
    kernels, and against the oracle but for the boxes the wrong way round."""
    import torch
    from hellovulkan_gb300.batch import Batch, BatchBuffers
    grid = (16, 9, 24)
    xy = grid[0] * grid[1]
    views = [view(grid, n, (25.0, 90.0), 150), view(grid, n, (900.0, 2000.0), 150, 67)]
    bufs = BatchBuffers(views)
    b = Batch(gpu)
    b.set_views(bufs.batch_views())
    b.generate_aabbs()
    given, turned = [], [40, 3 * xy + 43, 7 * xy + 47]
    for q, v in enumerate(views):
        a = oracle.generate_aabbs(v.ubo)
        for k, axis in ((0, 0), (3, 1), (7, 2)):  # bounds of one cluster exchanged, and far apart
            lo, hi = a[k * xy + 40 + k, axis], a[k * xy + 40 + k, 4 + axis]
            a[k * xy + 40 + k, axis], a[k * xy + 40 + k, 4 + axis] = hi + 120, lo - 120
        a[10 * xy + 5, 4:7] = a[10 * xy + 5, 0:3]
        a[12 * xy + 9, 0], a[12 * xy + 9, 4] = -np.inf, np.inf
        a[14 * xy + 9, 0], a[14 * xy + 9, 4] = np.inf, np.inf
        a[16 * xy + 1, 5] = np.nan
        bufs.aabbs[q].copy_(torch.from_numpy(a).reshape(bufs.aabbs[q].shape))
        given.append(a)
    b.cull()
    masks = [bufs.read(q)[1:] for q in range(2)]
    b.set_tuning(xy, 2, 8, 1024, 2)
    b.cull()
    for q, v in enumerate(views):
        _, cells, idx = bufs.read(q)
        assert np.array_equal(cells, masks[q][0]) and np.array_equal(idx, masks[q][1]), q
        oc, oi, _ = oracle.cull(v.ubo, given[q], v.lights, v.cap)
        for c in set(range(v.clusters)) - set(turned):
            assert np.array_equal(idx[cells[c, 0]:cells[c].sum()], oi[oc[c, 0]:oc[c].sum()]), (q, c)
    b.close()
