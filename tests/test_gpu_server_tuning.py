"""The server's tuning call: what it takes, it can launch."""
import numpy as np
import pytest

from hellovulkan_gb300 import scenes

pytestmark = pytest.mark.gpu

CF_ERROR_INVALID_ARGUMENT = 1


def served(srv, view, set_id):
    rid = srv.submit(view.ubo, set_id)
    (c,) = srv.wait_all(1)
    assert c.request_id == rid
    out = srv.read(c) if c.status == 0 else None
    if out:
        srv.release(rid)
    return c.status, out


def test_a_tuning_without_served_kernels_is_refused(gpu, cflib, oracle):
    """(4, 8, 32, 1), the hit masks, is what cf_batch_get_info may report and
    no configuration of the served kernels: refused, and the grid's requests
    go on as before; a staged configuration is taken."""
    from hellovulkan_gb300.server import Server
    v = scenes.plain_small(3)
    xy = v.grid[0] * v.grid[1]
    oc, oi, _ = oracle.cull(v.ubo, oracle.generate_aabbs(v.ubo), v.lights, 150)
    srv = Server(gpu, budget_bytes=64 << 20, streams=2)
    sid = srv.register(v.lights)
    for tuning, taken in (((4, 8, 32, 1), False), ((3, 5, 7, 9), False), ((2, 8, 256, 4), True), ((0, 0, 0, 0), True)):
        status = cflib.cf_server_set_tuning(srv.handle, xy, *tuning)
        assert status == (0 if taken else CF_ERROR_INVALID_ARGUMENT), tuning
        st, out = served(srv, v, sid)
        assert st == 0 and np.array_equal(out[0], oc) and np.array_equal(out[1], oi), tuning
    srv.close()
