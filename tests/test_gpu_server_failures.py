"""A served batch whose launches fail in the middle."""
import numpy as np
import pytest

from hellovulkan_gb300 import scenes

pytestmark = pytest.mark.gpu

CF_ERROR_CUDA = 3


def test_a_failed_batch_gives_its_memory_back_once_its_kernels_are_done(gpu, cflib, oracle):
    """Batches that fail after the light transform and the slice lists of
    large views (some 100 us of work): their requests report the failure,
    nothing of theirs is in flight when their memory returns to the arena,
    and the batches that get this memory, on another stream too, are right."""
    from hellovulkan_gb300.server import Server
    rng = np.random.default_rng(61)
    views = [scenes.plain_large(seed, n_lights=30000) for seed in (2, 5)] + [scenes.batch_view(rng) for _ in range(4)]
    want = []
    for v in views:
        a = oracle.generate_aabbs(v.ubo)
        want.append(oracle.cull(v.ubo, a, v.lights, 150)[:2])
    before = cflib.cf_testing_early_batch_releases()
    srv = Server(gpu, budget_bytes=512 << 20, max_batch_views=8, streams=2)
    sets = [srv.register(v.lights) for v in views]
    try:
        for _ in range(5):
            cflib.cf_testing_fail_server_batches(1)
            failing = {srv.submit(views[0].ubo, sets[0])}
            failed = srv.wait_all(1)
            assert {c.request_id for c in failed} == failing and failed[0].status == CF_ERROR_CUDA
            ids = {srv.submit(v.ubo, s): q for q, (v, s) in enumerate(zip(views, sets))}
            done = srv.wait_all(len(ids))
            assert len(done) == len(ids)
            for c in done:
                assert c.status == 0
                cells, idx = srv.read(c)
                assert np.array_equal(cells, want[ids[c.request_id]][0])
                assert np.array_equal(idx, want[ids[c.request_id]][1])
                srv.release(c.request_id)
        assert cflib.cf_testing_early_batch_releases() == before
    finally:
        cflib.cf_testing_fail_server_batches(0)
        srv.close()
