"""GPU tests of the consumers' tiled kernels (cf_lookup_clusters,
cf_shade_clusters) where they can go wrong, bit for bit against the oracle:
images at and around the tiles' sides and too narrow for tiles, light sets
around what the shared-memory table holds, unaligned outputs, lists that do not
ascend or hold no light, and texels and lights for which the shading's reach
test may not be taken — texels out of its bounds, non-finite and degenerate
values, lights at exactly their radius, falloffs at and past its limit."""
import ctypes as C

import numpy as np
import pytest

from gpu_helpers import run_pipeline
from hellovulkan_gb300 import scenes
from hellovulkan_gb300._lib import CfPBRPushConstant, check, lib
from test_gpu_lookup import device_lookup, same

pytestmark = pytest.mark.gpu


def view_of(res, n_lights, grid=(5, 4, 12), seed=0, r=(0.5, 6.0)):
    rng = np.random.default_rng(seed + n_lights + res[0])
    return scenes.custom_view(grid, *res, 0.1, 300.0,
                              lights=scenes.uniform_box_lights(rng, n_lights, [-20, -10, -60], [20, 10, -1], *r)), rng


RESOLUTIONS = [(1, 1), (7, 300), (300, 7), (15, 16), (16, 16), (33, 31), (97, 64), (1001, 701), (1201, 1051)]


@pytest.mark.parametrize("res", RESOLUTIONS)
def test_lookup_images(gpu, oracle, res):
    v, rng = view_of(res, 400)
    aabbs, cells, idx = run_pipeline(gpu, v)
    depth = scenes.depth_log_uniform(rng, *res, 0.1, 300.0, far_plane_fraction=0.05)
    depth.reshape(-1)[::37] = rng.choice([0.0, 1.0, -0.5, 1.5, np.nan, np.inf], depth.reshape(-1)[::37].size)
    for check_all in (False, True):
        got = device_lookup(v, depth, cells, idx, aabbs, check_all)
        want = oracle.lookup_clusters(v.ubo, depth, cells, idx, v.lights, v.cap, aabbs, check_all)
        nan = np.isnan(want["view_z"]) & np.isnan(got["view_z"])  # a NaN's payload is not pinned
        nan_l = np.isnan(want["linear_depth"]) & np.isnan(got["linear_depth"])
        got["view_z"][nan] = want["view_z"][nan] = 0
        got["linear_depth"][nan_l] = want["linear_depth"][nan_l] = 0
        assert same(got, want)


@pytest.mark.parametrize("n_lights", [0, 1, 31, 33, 63, 65, 1023, 1024, 1025, 1088, 2048, 2500])
def test_lookup_light_tables(gpu, oracle, n_lights):
    v, rng = view_of((160, 96), n_lights)
    if n_lights > 31:
        v.lights[5, 0], v.lights[9, 1], v.lights[20, 8] = np.nan, np.inf, np.inf
    aabbs, cells, idx = run_pipeline(gpu, v)
    depth = scenes.depth_log_uniform(rng, 160, 96, 0.1, 300.0)
    got = device_lookup(v, depth, cells, idx, aabbs, True)
    assert same(got, oracle.lookup_clusters(v.ubo, depth, cells, idx, v.lights, v.cap, aabbs, True))


@pytest.mark.parametrize("depths", ["scattered", "one", "ramp"])
@pytest.mark.parametrize("res", [(96, 64), (512, 320)])
def test_lookup_lists_read_by_a_warp(gpu, oracle, res, depths):
    """Lists of no light to five times a warp's width, with non-finite lights
    and entries that are no light in them: clusters with a few of a warp's
    pixels each, with all of them, and with fragments whose box few of the
    listed lights reach; images on both sides of a tile per SM."""
    v, rng = view_of(res, 1500, grid=(3, 2, 16), r=(0.2, 9.0))
    v.lights[[5, 400], 0], v.lights[9, 1], v.lights[20, 8] = np.nan, -np.inf, np.inf
    aabbs, cells, idx = run_pipeline(gpu, v)
    assert cells[:, 1].max() > 96 and (cells[:, 1] < 8).any()
    idx = idx.copy()
    idx[rng.integers(0, idx.size, 40)] = rng.choice([1500, 0xFFFFFFFF], 40)
    if depths == "scattered":
        depth = scenes.depth_log_uniform(rng, *res, 0.1, 300.0)
    else:
        lin = np.full(res[::-1], 20.0) if depths == "one" else np.broadcast_to(np.linspace(2.0, 59.0, res[0]), res[::-1])
        depth = ((0.1 * 300.0 / lin - 300.0) / (0.1 - 300.0)).astype(np.float32)
    got = device_lookup(v, depth, cells, idx, aabbs, False)
    assert same(got, oracle.lookup_clusters(v.ubo, depth, cells, idx, v.lights, v.cap, aabbs, False))


def test_lookup_lists_that_do_not_ascend(gpu, oracle):
    """A walk over all lights in order matches a list up to its first entry
    that does not ascend or is no light; the lights after that count as
    missing even where the list holds them."""
    v, rng = view_of((96, 64), 300, r=(4.0, 12.0))
    aabbs, cells, idx = run_pipeline(gpu, v)
    idx = idx.copy()
    hit = rng.integers(0, idx.size, idx.size // 8)
    idx[hit] = rng.choice([0, 7, 299, 300, 0xFFFFFFFF], hit.size)
    depth = scenes.depth_log_uniform(rng, 96, 64, 0.1, 300.0)
    got = device_lookup(v, depth, cells, idx, aabbs, True)
    want = oracle.lookup_clusters(v.ubo, depth, cells, idx, v.lights, v.cap, aabbs, True)
    prefix = cells.copy()
    for c, (off, n) in enumerate(cells):
        k, last = 0, -1
        while k < n and last < int(idx[off + k]) < 300:
            last, k = int(idx[off + k]), k + 1
        prefix[c, 1] = k
    none = np.zeros_like(cells)
    every = oracle.lookup_clusters(v.ubo, depth, none, idx, v.lights, v.cap, aabbs, True)["missing"]
    matched = oracle.lookup_clusters(v.ubo, depth, prefix, idx, v.lights, v.cap, aabbs, False)["covering"]
    want["missing"] = every - matched
    assert same(got, want)


def test_lookup_into_an_unaligned_buffer(gpu, oracle):
    import torch
    v, rng = view_of((64, 48), 200)
    aabbs, cells, idx = run_pipeline(gpu, v)
    depth = scenes.depth_log_uniform(rng, 64, 48, 0.1, 300.0)
    d = {k: torch.from_numpy(np.ascontiguousarray(a)).cuda() for k, a in
         (("z", depth), ("c", cells.view(np.int32)), ("i", idx.view(np.int32)), ("l", v.lights), ("a", aabbs))}
    out = torch.zeros(64 * 48 * 32 + 16, dtype=torch.uint8, device="cuda")
    check(lib().cf_lookup_clusters(C.byref(v.ubo), d["z"].data_ptr(), 64, 48, d["c"].data_ptr(), d["i"].data_ptr(),
                                   idx.size, d["l"].data_ptr(), 200, v.cap, d["a"].data_ptr(), 0, out.data_ptr() + 4, None))
    torch.cuda.synchronize()
    from hellovulkan_gb300._lib import FRAGMENT_DTYPE
    got = out.cpu().numpy()[4:4 + 64 * 48 * 32].copy().view(FRAGMENT_DTYPE).reshape(48, 64)
    assert same(got, oracle.lookup_clusters(v.ubo, depth, cells, idx, v.lights, v.cap, aabbs, False))


def shade(view, g, cells, idx, pc, cam):
    import torch
    from hellovulkan_gb300.consumer import shade_clusters
    d_idx = torch.from_numpy(idx.view(np.int32).copy() if idx.size else np.zeros(1, np.int32)).cuda()
    lights = torch.from_numpy(np.ascontiguousarray(view.lights)).cuda()
    return shade_clusters(view.ubo, cam, pc, torch.from_numpy(np.ascontiguousarray(g)).cuda(),
                          torch.from_numpy(cells.view(np.int32)).cuda(), d_idx, idx.size, lights,
                          view.light_count).cpu().numpy()


def same_shading(got, want):
    nan = np.isnan(got) & np.isnan(want)  # a NaN's payload is not pinned
    return np.array_equal(np.where(nan, 0, got).view(np.uint32), np.where(nan, 0, want).view(np.uint32))


PC = CfPBRPushConstant(1.75, 0.01, 0.0, 0.1, 0.1)


@pytest.mark.parametrize("res", RESOLUTIONS)
def test_shading_images(gpu, oracle, res):
    v, rng = view_of(res, 400)
    _, cells, idx = run_pipeline(gpu, v)
    g = scenes.gbuffer(rng, v.ubo, far_plane_fraction=0.05)
    cam = scenes.camera_position(v.ubo)
    assert same_shading(shade(v, g, cells, idx, PC, cam), oracle.shade_clusters(v.ubo, cam, PC, g, cells, idx, v.lights))


@pytest.mark.parametrize("n_lights", [0, 1, 31, 1023, 1024, 1025, 2500])
def test_shading_light_tables(gpu, oracle, n_lights):
    v, rng = view_of((160, 96), n_lights)
    _, cells, idx = run_pipeline(gpu, v)
    idx = idx.copy()
    if idx.size:
        idx[rng.integers(0, idx.size, 1 + idx.size // 50)] = 0xFFFFFFFF  # no light
    g = scenes.gbuffer(rng, v.ubo)
    cam = scenes.camera_position(v.ubo)
    assert same_shading(shade(v, g, cells, idx, PC, cam), oracle.shade_clusters(v.ubo, cam, PC, g, cells, idx, v.lights))


ODD = np.array([0.0, -0.0, 1e-30, -1e-3, 1.0, 1.8, 1.9, 2.0, 1e7, 1e30, np.inf, -np.inf, np.nan], np.float32)


@pytest.mark.parametrize("depths", ["scattered", "one"])
@pytest.mark.parametrize("r", [(0.2, 1.5), (0.2, 9.0)])
def test_shading_lists_read_by_a_warp(gpu, oracle, r, depths):
    """Lists that each texel walks itself and lists, of up to five times a
    warp's width, that a warp reads for all its texels of a cluster; clusters
    with a few of its texels and with all; entries that are no light."""
    v, rng = view_of((96, 64), 1500, grid=(3, 2, 16), r=r)
    _, cells, idx = run_pipeline(gpu, v)
    if r[1] > 5:
        assert cells[:, 1].max() > 96
    cells, idx = cells.copy(), idx.copy()
    if r[1] < 5:
        cells[:, 1] = np.minimum(cells[:, 1], rng.integers(0, 8, cells.shape[0]))  # around what counts as short
    idx[rng.integers(0, idx.size, 40)] = rng.choice([1500, 0xFFFFFFFF], 40)
    g = scenes.gbuffer(rng, v.ubo)
    if depths == "one":
        g[..., 3] = np.float32((0.1 * 300.0 / 20.0 - 300.0) / (0.1 - 300.0))
    cam = scenes.camera_position(v.ubo)
    assert same_shading(shade(v, g, cells, idx, PC, cam), oracle.shade_clusters(v.ubo, cam, PC, g, cells, idx, v.lights))


@pytest.mark.parametrize("falloff", [0.1, 0.0, 2.0, -1.5, 60.0, 120.0, 121.0, np.inf, np.nan])
@pytest.mark.parametrize("intensity", [1.75, 0.0, np.inf])
def test_shading_odd_texels_and_lights(gpu, oracle, falloff, intensity):
    """Every field of some texels and lights replaced by a value that breaks
    an assumption of the reach test, lights at a texel's own position, behind
    it on the camera's ray, and at exactly their radius from it."""
    v, rng = view_of((128, 96), 300, r=(1.0, 10.0))
    g = scenes.gbuffer(rng, v.ubo)
    cam = scenes.camera_position(v.ubo)
    flat = g.reshape(-1, 12)
    n = flat.shape[0]
    for field in (0, 1, 4, 5, 7, 8, 9, 11):
        rows = rng.integers(0, n, n // 40)
        flat[rows, field] = rng.choice(ODD, rows.size)
    rows = rng.integers(0, n, n // 20)
    flat[rows, 4:7] *= rng.uniform(0.0, 3.0, (rows.size, 1)).astype(np.float32)  # normals of other lengths
    rows = rng.integers(0, n, n // 20)
    to = cam - flat[rows, 0:3]  # the normal along the view ray, on a mirror
    with np.errstate(invalid="ignore"):
        flat[rows, 4:7] = (to / np.linalg.norm(to, axis=1, keepdims=True)).astype(np.float32)
    flat[rows, 11] = rng.choice([0.0, 0.03, 0.056, 0.06], rows.size)
    L = v.lights
    at = flat[rng.integers(0, n, 100), 0:3]
    L[0:30, 0:3] = at[0:30]  # at a texel
    L[30:60, 0:3] = cam + (at[30:60] - cam) * 1.5  # behind it
    L[60:100, 0:3] = at[60:100] + np.float32([0, 3, 4])  # 5 away, radius 5
    L[60:100, 8] = 5.0
    for field in (4, 5, 8):
        L[rng.integers(100, 300, 12), field] = rng.choice(ODD, 12)
    L[np.isnan(L).any(1) | np.isinf(L).any(1), 0:3] = rng.uniform([-10, -5, -40], [10, 5, -2], (int((np.isnan(L).any(1) |
                                                                  np.isinf(L).any(1)).sum()), 3))
    L[110, 0], L[111, 1] = np.nan, np.inf
    # every cluster lists every light, in order: the test must hold for any pair
    c = v.clusters
    cells = np.stack([np.zeros(c, np.uint32), np.full(c, 300, np.uint32)], axis=1)
    idx = np.arange(300, dtype=np.uint32)
    pc = CfPBRPushConstant(intensity, 0.01, 0.0, falloff, -0.0)
    assert same_shading(shade(v, g, cells, idx, pc, cam), oracle.shade_clusters(v.ubo, cam, pc, g, cells, idx, v.lights))


@pytest.mark.parametrize("res, grid, n_lights", [((96, 64), (40, 24, 30), 4000), ((20, 3000), (16, 9, 24), 3500),
                                                 ((330, 200), (64, 60, 20), 2500), ((900, 500), (90, 70, 12), 2500)])
def test_lookup_of_many_clusters_per_warp(gpu, oracle, res, grid, n_lights):
    """Clusters of a few pixels or less: each pixel of a warp walks its own
    list, of none to over a hundred entries, some of them no light."""
    v, rng = view_of(res, n_lights, grid=grid, r=(0.2, 5.0))
    v.lights[[5, 400], 0], v.lights[9, 1], v.lights[20, 8] = np.nan, -np.inf, np.inf
    aabbs, cells, idx = run_pipeline(gpu, v)
    assert cells[:, 1].max() > 64
    idx = idx.copy()
    idx[rng.integers(0, idx.size, idx.size // 200)] = rng.choice([n_lights, 0xFFFFFFFF], idx.size // 200)
    cells = cells.copy()
    cells[rng.integers(0, cells.shape[0], 5)] = [idx.size - 2, 3]  # no cell of this list
    depth = scenes.depth_log_uniform(rng, *res, 0.1, 300.0, far_plane_fraction=0.02)
    got = device_lookup(v, depth, cells, idx, aabbs, False)
    assert same(got, oracle.lookup_clusters(v.ubo, depth, cells, idx, v.lights, v.cap, aabbs, False))


@pytest.mark.parametrize("res, grid, n_lights", [((96, 64), (40, 24, 30), 4000), ((20, 3000), (16, 9, 24), 3500),
                                                 ((330, 200), (64, 60, 20), 2500)])
def test_shading_of_many_clusters_per_warp(gpu, oracle, res, grid, n_lights):
    """As the lookup's: each texel walks its own list, some of whose entries
    are no light, and warps on both sides of the rule."""
    v, rng = view_of(res, n_lights, grid=grid, r=(0.2, 5.0))
    _, cells, idx = run_pipeline(gpu, v)
    assert cells[:, 1].max() > 64
    idx = idx.copy()
    idx[rng.integers(0, idx.size, idx.size // 200)] = rng.choice([n_lights, 0xFFFFFFFF], idx.size // 200)
    g = scenes.gbuffer(rng, v.ubo, far_plane_fraction=0.02)
    cam = scenes.camera_position(v.ubo)
    assert same_shading(shade(v, g, cells, idx, PC, cam), oracle.shade_clusters(v.ubo, cam, PC, g, cells, idx, v.lights))


@pytest.mark.parametrize("res, grid, n_lights", [((19, 886), (20, 8, 55), 150), ((97, 64), (22, 20, 24), 70),
                                                 ((1001, 701), (90, 70, 12), 40), ((1201, 1051), (120, 105, 6), 33)])
def test_shading_of_lists_that_all_reach(gpu, oracle, res, grid, n_lights):
    """Every light reaches every texel, with a few texels to a cluster: a
    texel's pairs are gathered 32 at a time, and the sums keep the list's
    order; an entry that is no light in the middle of some lists."""
    v, rng = view_of(res, n_lights, grid=grid, r=(500.0, 2000.0))
    _, cells, idx = run_pipeline(gpu, v)
    assert cells[:, 1].min() == n_lights
    idx = idx.copy()
    idx[rng.integers(0, idx.size, idx.size // 500)] = n_lights
    g = scenes.gbuffer(rng, v.ubo, far_plane_fraction=0.02)
    cam = scenes.camera_position(v.ubo)
    assert same_shading(shade(v, g, cells, idx, PC, cam), oracle.shade_clusters(v.ubo, cam, PC, g, cells, idx, v.lights))


@pytest.mark.parametrize("res", [(31, 400), (97, 64), (1001, 701)])
def test_shading_of_unlit_tiles(gpu, oracle, res):
    """An image whose tiles are unlit but for those around a few small lights:
    unlit clusters, texels outside of the grid and cells that are none, in
    tiles of their own and beside lit ones; a black albedo's sign."""
    v, rng = view_of(res, 12, grid=(16, 12, 24), r=(0.05, 0.8))
    v.lights[:, 0:3] *= np.float32(0.2)
    _, cells, idx = run_pipeline(gpu, v)
    lit = cells[:, 1] > 0
    assert 0 < lit.sum() < 0.1 * lit.size
    cells = cells.copy()
    cells[rng.integers(0, cells.shape[0], 40)] = [idx.size, 1]  # no cell of this list
    g = scenes.gbuffer(rng, v.ubo, far_plane_fraction=0.02)
    w, h = res
    g[: h // 3, :, 3] = 1.0
    g[h // 2:, : w // 2, 3] = rng.choice([1.0, -0.5, 1.5, np.nan], (h - h // 2, w // 2))
    g[:, :, 8:11] = np.where(rng.uniform(size=(h, w, 1)) < 0.1, np.float32(-0.0), g[:, :, 8:11])
    cam = scenes.camera_position(v.ubo)
    assert same_shading(shade(v, g, cells, idx, PC, cam), oracle.shade_clusters(v.ubo, cam, PC, g, cells, idx, v.lights))


@pytest.mark.parametrize("res, grid, n_lights, r", [((96, 64), (40, 24, 30), 4000, (0.2, 5.0)), ((20, 3000), (16, 9, 24), 1500, (0.2, 5.0)),
                                                    ((330, 200), (64, 60, 20), 900, (0.2, 9.0)), ((17, 56), (122, 61, 2), 27, (500.0, 900.0))])
def test_check_of_many_clusters_per_warp(gpu, oracle, res, grid, n_lights, r):
    """As the lookup's, with the all-lights check: each pixel of a warp walks its
    own list, up to the entry that does not ascend or is no light for what
    the list lacks."""
    v, rng = view_of(res, n_lights, grid=grid, r=r)
    v.lights[5, 0], v.lights[9, 1], v.lights[20, 8] = np.nan, -np.inf, np.inf
    aabbs, cells, idx = run_pipeline(gpu, v)
    idx = idx.copy()
    at = rng.integers(0, idx.size, idx.size // 40)
    idx[at] = rng.choice([n_lights, 0xFFFFFFFF, 0, n_lights - 1], at.size)
    depth = scenes.depth_log_uniform(rng, *res, 0.1, 300.0, far_plane_fraction=0.02)
    got = device_lookup(v, depth, cells, idx, aabbs, True)
    want = oracle.lookup_clusters(v.ubo, depth, cells, idx, v.lights, v.cap, aabbs, True)
    # what is missing, from the part of each list that a walk over all lights matches
    last = np.concatenate([[-1], idx[:-1].astype(np.int64)])
    last[np.minimum(cells[:, 0], idx.size - 1)] = -1
    good = (idx < n_lights) & (idx.astype(np.int64) > last)
    bad_before = np.concatenate([[0], np.cumsum(~good)])
    prefix = cells.copy()
    for c in np.nonzero(cells[:, 1])[0]:
        off, n = cells[c]
        prefix[c, 1] = np.searchsorted(bad_before[off + 1:off + n + 1], bad_before[off], side="right")
    every = oracle.lookup_clusters(v.ubo, depth, np.zeros_like(cells), idx, v.lights, v.cap, aabbs, True)["missing"]
    matched = oracle.lookup_clusters(v.ubo, depth, prefix, idx, v.lights, v.cap, aabbs, False)["covering"]
    want["missing"] = every - matched
    assert want["missing"].max() > 0
    assert same(got, want)


@pytest.mark.parametrize("res, grid, n_lights, cap", [((31, 200), (62, 40, 3), 450, 500), ((31, 6000), (62, 50, 3), 150, 150),
                                                      ((28, 300), (24, 40, 3), 400, 500)])
@pytest.mark.parametrize("check_all", [False, True])
def test_lookup_of_long_lists_of_many_clusters(gpu, oracle, res, grid, n_lights, cap, check_all):
    """A cluster or more for each pixel of a warp, with lists longer than the
    rule by length takes: each pixel walks its own all the same; and 24
    clusters or a few less."""
    v, rng = view_of(res, n_lights, grid=grid, r=(500.0, 900.0))
    v.cap = cap
    aabbs, cells, idx = run_pipeline(gpu, v)
    assert cells[:, 1].min() == n_lights
    depth = scenes.depth_log_uniform(rng, *res, 0.1, 300.0, far_plane_fraction=0.02)
    depth[:, :] = depth[:, :1]  # a row at one depth: its pixels lie in the columns' clusters
    got = device_lookup(v, depth, cells, idx, aabbs, check_all)
    assert same(got, oracle.lookup_clusters(v.ubo, depth, cells, idx, v.lights, v.cap, aabbs, check_all))
