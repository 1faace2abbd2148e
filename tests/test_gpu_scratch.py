"""Views whose hit masks need more scratch than the caller brings: the other
kernels take them, with the same output, and none is refused that they fit."""
import ctypes as C
import re

import numpy as np
import pytest

from hellovulkan_gb300 import scenes
from test_gpu_failures import STALL_BRUTE_FORCE, hooks  # noqa: F401 (a fixture)
from test_zz_no_alloc import _inputs, _oracle, _outputs, _read, _with_static_scratch

pytestmark = pytest.mark.gpu

CF_ERROR_CAPACITY = 4


def view(grid, n_lights, cap=32):
    rng = np.random.default_rng(n_lights)
    return scenes.custom_view(grid, 1920, 1080, 0.1, 300.0, cap=cap,
                              lights=scenes.uniform_box_lights(rng, n_lights, [-30, -15, -60], [30, 15, -5], 0.5, 3.0))


# brute force and, for the last two, the staged kernels without the hit masks
@pytest.mark.parametrize("grid, n_lights", [((8, 8, 16), 2400), ((2, 1, 200), 4000), ((24, 14, 32), 9000), ((5, 1, 255), 14000)])
def test_a_workspace_that_holds_the_other_kernels_is_taken(cflib, oracle, grid, n_lights):
    import torch
    v = view(grid, n_lights)
    aabbs, lights = _inputs(v)
    o_cells, o_idx = _oracle(oracle, v, aabbs)
    reported = C.c_uint64()
    assert cflib.cf_cull_workspace_size(C.byref(v.ubo), v.light_count, v.cap, C.byref(reported)) == 0

    def cull(ws_bytes):
        cells, idx, total = _outputs(v)
        ws = torch.zeros(max(ws_bytes, 1), dtype=torch.uint8, device="cuda")
        st = cflib.cf_cull_lights(C.byref(v.ubo), aabbs.data_ptr(), lights.data_ptr(), v.light_count, v.cap,
                                  cells.data_ptr(), idx.data_ptr(), v.clusters * v.cap, total.data_ptr(), ws.data_ptr(),
                                  ws_bytes, torch.cuda.current_stream().cuda_stream)
        return st, _read(v, cells, idx, total) if st == 0 else None

    st, _ = cull(0)
    assert st == CF_ERROR_CAPACITY
    least = int(re.search(rb"< (\d+) needed", cflib.cf_last_error_message()).group(1))
    assert least < reported.value
    assert cull(least - 1)[0] == CF_ERROR_CAPACITY
    for size in (least, reported.value - 1, reported.value):
        st, out = cull(size)
        assert st == 0 and np.array_equal(out[0], o_cells) and np.array_equal(out[1], o_idx), size


# staged layout 23 and 20 MiB, hit masks 36 and 41 MiB, static scratch 32 MiB
@pytest.mark.parametrize("grid, n_lights", [((32, 18, 48), 22000), ((64, 36, 64), 8000)])
def test_static_scratch_takes_the_staged_kernels_before_brute_force(cflib, hooks, oracle, grid, n_lights):  # noqa: F811
    """With the brute-force kernel's first tile withheld, its bounded waits
    run out and the error word says so; it must not have been used."""
    v = view(grid, n_lights, cap=16)
    aabbs, lights = _inputs(v)
    assert cflib.cf_testing_set_wait_limit_ns(20_000_000) == 0
    assert cflib.cf_testing_inject_stall(STALL_BRUTE_FORCE) == 0
    try:
        cells, idx, _ = _with_static_scratch(v, aabbs, lights)  # asserts that the error word is clear
    finally:
        cflib.cf_testing_inject_stall(0)
        cflib.cf_testing_set_wait_limit_ns(0)
    o_cells, o_idx = _oracle(oracle, v, aabbs)
    assert np.array_equal(cells, o_cells) and np.array_equal(idx, o_idx)


def pipeline(gpu, v):
    from hellovulkan_gb300.pipelines import (PipelineAABBGenerator, PipelineLightCulling, ResourcesClusterForward,
                                             ResourcesLight)
    rl, rc = ResourcesLight(gpu), ResourcesClusterForward(gpu)
    rl.add_lights(v.lights)
    rc.create_buffers(*v.grid, v.cap)
    gen, cull = PipelineAABBGenerator(gpu, rc), PipelineLightCulling(gpu, rl, rc)
    gen.set_cluster_forward_ubo(v.ubo)
    gen.fill_command_buffer()
    cull.set_cluster_forward_ubo(v.ubo)
    return cull, rc, (cull, gen, rc, rl)


STAGED, MASK = (2, 8, 1024, 2, 1), (4, 8, 32, 1, 1)


# units of 128 lights and a group: 100 bytes each, half a gigabyte or twice the lists' bytes at most
@pytest.mark.parametrize("grid, n_lights, want", [((128, 128, 24), 32768, MASK), ((128, 128, 24), 65536, STAGED),
                                                  ((64, 36, 4), 3500000, STAGED), ((64, 18, 4), 1000000, MASK)])
def test_views_whose_masks_would_take_too_much_memory(gpu, oracle, grid, n_lights, want):
    """The choice on both sides of the line, for a pipeline and for a batch,
    and the same lists from both sides."""
    import torch

    from hellovulkan_gb300.batch import Batch, BatchBuffers
    v = view(grid, n_lights, cap=4)
    cull, rc, objects = pipeline(gpu, v)
    assert cull.tuning() == want
    cull.fill_command_buffer()
    cells, idx = rc.read_outputs()
    cells, idx = cells.copy(), idx.copy()
    cull.set_tuning(*(STAGED if want == MASK else MASK))
    cull.fill_command_buffer()
    other = rc.read_outputs()
    assert np.array_equal(cells, other[0]) and np.array_equal(idx, other[1])
    for o in objects:
        o.close()
    bufs = BatchBuffers([v])
    b = Batch(gpu)
    b.set_views(bufs.batch_views())
    assert b.info()["bucket_configs"][0]["config"] == list(want[:4])
    b.generate_aabbs()
    b.cull()
    torch.cuda.synchronize()
    _, c, i = bufs.read(0)
    assert np.array_equal(cells, c) and np.array_equal(idx, i)
    b.close()


def test_without_room_for_the_masks_the_other_kernels_run(gpu, hooks, oracle):  # noqa: F811
    from hellovulkan_gb300.batch import Batch, BatchBuffers
    v = view((16, 9, 24), 6000, cap=150)
    a = oracle.generate_aabbs(v.ubo)
    oc, oi, _ = oracle.cull(v.ubo, a, v.lights, v.cap)
    cull, rc, objects = pipeline(gpu, v)
    assert cull.tuning() == MASK
    hooks.cf_testing_fail_allocation_after(0)  # the workspace with hit masks
    for _ in range(2):
        cull.fill_command_buffer()
        cells, idx = rc.read_outputs()
        assert np.array_equal(cells, oc) and np.array_equal(idx, oi)
        assert cull.tuning() == STAGED
    hooks.cf_testing_fail_allocation_after(-1)
    rc.create_buffers(*v.grid, v.cap)
    assert cull.tuning() == MASK
    for o in objects:
        o.close()
    bufs = BatchBuffers([v])
    b = Batch(gpu)
    hooks.cf_testing_fail_allocation_after(0)
    b.set_views(bufs.batch_views())
    hooks.cf_testing_fail_allocation_after(-1)
    assert b.info()["bucket_configs"][0]["config"] == list(STAGED[:4])
    b.generate_aabbs()
    b.cull()
    _, c, i = bufs.read(0)
    assert np.array_equal(oc, c) and np.array_equal(oi, i)
    b.close()


def test_without_room_for_any_the_failure_is_reported(gpu, hooks):  # noqa: F811
    from hellovulkan_gb300._lib import CfError
    v = view((16, 9, 24), 6000)
    cull, rc, objects = pipeline(gpu, v)
    cull.set_tuning(*MASK)  # asked for by name: nothing takes its place
    hooks.cf_testing_fail_allocation_after(0)
    with pytest.raises(CfError) as e:
        cull.fill_command_buffer()
    assert e.value.status == 2  # CF_ERROR_OUT_OF_MEMORY
    hooks.cf_testing_fail_allocation_after(-1)
    for o in objects:
        o.close()
