"""The warp-cooperative traversal (csrc/warptrace.cuh) on scenes and ray counts
at its edges: trees deep enough to drop short-stack entries, leaves of more than
four triangles, partial warps and groups, each launch rule's limits, and a BVH
buffer that starts on 16 bytes only. Hits and distances bit-exact vs the oracle.
"""
import numpy as np
import pytest

import oracle.binding as ob
import restir_b200 as rb
from restir_b200.abi import RestirScene
from tests.helpers import SceneSetup, make_scene, seeded_rays

KINDS = [rb.TRACE_CLOSEST, rb.TRACE_ANY, rb.TRACE_CLOSEST_STACKLESS, rb.TRACE_CLOSEST_QUEUE]


def large_leaves(setup: SceneSetup) -> SceneSetup:
    """setup with a tree of this test's own over its triangles: leaves of 5 to 12 of them, sorted by x."""
    data = setup.bvh.data.reshape(-1, 4)
    n, offset = setup.bvh.desc.triangle_count, setup.bvh.desc.triangle_offset
    triangles = data[offset:].reshape(n, 4, 4)
    triangles = triangles[np.argsort(triangles[:, :3, 0].mean(1), kind="stable")]
    bounds = np.concatenate([[0], np.cumsum(np.tile([5, 12, 9, 7, 8], n // 41 + 1))])
    bounds = np.append(bounds[bounds < n], n)
    nodes = []

    def build(lo, hi):
        corners = triangles[bounds[lo]:bounds[hi], :3, :3].reshape(-1, 3)
        index = len(nodes)
        nodes.append(None)
        if hi - lo == 1:
            a, b = bounds[lo], bounds[hi] - bounds[lo]
        else:
            build(lo, (lo + hi) // 2)
            a = len(nodes)
            build((lo + hi) // 2, hi)
            b = -len(nodes) - 1
        nodes[index] = [[*corners.min(0), a], [*corners.max(0), b]]

    build(0, len(bounds) - 1)
    rows = np.concatenate([np.array(nodes, np.float32).reshape(-1, 4), triangles.reshape(-1, 4)]).astype(np.float32)
    setup.bvh_data, setup.node_count, setup.triangle_offset = rows.reshape(-1), len(nodes), 2 * len(nodes)
    return setup


def check(setup, rays, kind, offset=0):
    import torch
    n = len(rays)
    ids, t = np.zeros(n, np.int32), np.zeros(n, np.float32)
    ob.load().oracle_trace(None, setup.host_scene(), rays.ctypes.data, ids.ctypes.data, t.ctypes.data, n, kind)
    scene = setup.device_scene()
    data = setup.bvh_data if setup.bvh_data is not None else setup.bvh.data
    rows = torch.zeros(data.size + 8, dtype=torch.float32, device="cuda")
    rows[offset:offset + data.size] = torch.from_numpy(data).cuda()
    scene.bvh = rows[offset:].data_ptr()
    d_rays = torch.from_numpy(rays).cuda()
    d_ids, d_t = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.float32, device="cuda")
    rb.check(rb.load().restir_trace(None, scene, d_rays.data_ptr(), d_ids.data_ptr(), d_t.data_ptr(), n, kind, None),
             "restir_trace")
    torch.cuda.synchronize()
    np.testing.assert_array_equal(d_ids.cpu().numpy(), ids)
    np.testing.assert_array_equal(d_t.cpu().numpy().view(np.uint32), t.view(np.uint32))
    rb.status_flags()  # some of these rays reach the step cap, as the oracle's do


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 31, 33, 1000, 37_888, 37_889, 303_105])
def test_ray_counts(kind, n):
    setup = make_scene(rb.SCENE_CITY, 0, 60_000)
    check(setup, seeded_rays(setup, 303_105, seed=5)[::-1][:n].copy(), kind)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("triangles", [300, 4_000, 120_000])
def test_scene_sizes(kind, triangles):
    setup = make_scene(rb.SCENE_COURTYARD, 1, triangles)
    check(setup, seeded_rays(setup, 50_000, seed=6), kind)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [500, 310_000])
def test_large_leaves(kind, n):
    setup = large_leaves(make_scene(rb.SCENE_COURTYARD, 2, 20_000))
    assert setup.node_count > 4096
    check(setup, seeded_rays(setup, n, seed=7), kind)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_unaligned_rows(kind):
    """16 bytes past a 32-byte boundary: the nodes are read with 128-bit loads."""
    setup = make_scene(rb.SCENE_CITY, 0, 60_000)
    check(setup, seeded_rays(setup, 20_000, seed=8), kind, offset=4)


def test_wide_rows_rule():
    """32-byte reads need the nodes and the triangles on 32 bytes: a buffer on 16 bytes only, or an odd number of rows
    before the triangles, takes the 16-byte ones."""
    scene = RestirScene()
    for address, offset, wide in ((4096, 86, 1), (4096, 87, 0), (4112, 86, 0), (4112, 87, 0), (4128, 0, 1)):
        scene.bvh, scene.node_count, scene.triangle_offset, scene.triangle_count = address, 43, offset, 36
        assert rb.load().restir_bvh_wide_rows(scene) == wide, (address, offset)
    assert rb.load().restir_bvh_wide_rows(None) == 0


def padded(setup: SceneSetup, rows: int) -> SceneSetup:
    """setup with rows of padding between its nodes and its triangles."""
    data, offset = setup.bvh.data.reshape(-1, 4), setup.bvh.desc.triangle_offset
    setup.bvh_data = np.concatenate([data[:offset], np.full((rows, 4), np.nan, np.float32), data[offset:]]).reshape(-1)
    setup.node_count, setup.triangle_offset = setup.bvh.desc.node_count, offset + rows
    return setup


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS + [rb.TRACE_CLOSEST_WATERTIGHT, rb.TRACE_ANY_WAVE])
@pytest.mark.parametrize("rows", [1, 2, 3])
def test_padding_before_the_triangles(kind, rows):
    """Triangles that start on 16 bytes only, and on 32 again."""
    setup = padded(make_scene(rb.SCENE_CITY, 0, 60_000), rows)
    check(setup, seeded_rays(setup, 20_000, seed=9), kind)


@pytest.mark.gpu
def test_more_than_2_31_rays():
    """Indices past 2^31: a set of rays that end before they start, and at its end real ones, through one thread per
    ray, the nearest parts with their re-walk, and the lane walks. 86 GB of rays and hits."""
    import torch
    n, real = (1 << 31) + 77, 300
    if torch.cuda.mem_get_info()[0] < 40 * n + (8 << 30):
        pytest.skip("needs 94 GB of device memory")
    rays = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
    rays[:, 3] = -1.0
    ids, t = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.float32, device="cuda")
    small, large = make_scene(rb.SCENE_CORNELL), make_scene(rb.SCENE_CITY, 0, 200_000)
    for setup, kind in ((small, rb.TRACE_CLOSEST), (large, rb.TRACE_CLOSEST_QUEUE), (large, rb.TRACE_CLOSEST_STACKLESS),
                        (large, rb.TRACE_ANY)):
        host = seeded_rays(setup, real, seed=10)
        rays[n - real:] = torch.from_numpy(host).cuda()
        want, distance = np.zeros(real, np.int32), np.zeros(real, np.float32)
        ob.load().oracle_trace(None, setup.host_scene(), host.ctypes.data, want.ctypes.data, distance.ctypes.data, real, kind)
        ids.fill_(7)
        t.fill_(7.0)
        rb.check(rb.load().restir_trace(None, setup.device_scene(), rays.data_ptr(), ids.data_ptr(), t.data_ptr(), n, kind,
                                        None), "restir_trace")
        torch.cuda.synchronize()
        np.testing.assert_array_equal(ids[n - real:].cpu().numpy(), want)
        np.testing.assert_array_equal(t[n - real:].cpu().numpy().view(np.uint32), distance.view(np.uint32))
        assert ids[:n - real].min() == -1 and ids[:n - real].max() == -1
        assert t[:n - real].min() == -1.0 and t[:n - real].max() == -1.0
    rb.status_flags()
    del rays, ids, t
    torch.cuda.empty_cache()


@pytest.mark.gpu
@pytest.mark.parametrize("triangles", [2_000, 30_000, 100_000])
@pytest.mark.parametrize("n", [127, 128, 151_553, 227_329, 454_657])
def test_nearest_hits_on_both_sides_of_each_line(triangles, n):
    """The sizes of scene and ray set between which restir_trace changes its kernel for nearest hits."""
    setup = make_scene(rb.SCENE_CITY, 0, triangles)
    assert {2_000: 4_096, 30_000: 131_072, 100_000: 1 << 30}[triangles] > setup.bvh.desc.node_count \
        > {2_000: 0, 30_000: 4_096, 100_000: 131_072}[triangles]
    check(setup, seeded_rays(setup, n, seed=11), rb.TRACE_CLOSEST)
    check(setup, seeded_rays(setup, n - 1, seed=12), rb.TRACE_CLOSEST)


@pytest.mark.gpu
@pytest.mark.parametrize("kind, counted", [(rb.TRACE_CLOSEST, 0), (rb.TRACE_ANY, 0), (rb.TRACE_CLOSEST_STACKLESS, 0),
                                           (rb.TRACE_ANY_WAVE, 0), (rb.TRACE_CLOSEST_QUEUE, 1)])
@pytest.mark.parametrize("n", [40, 40_000, 400_000])
def test_empty_scene(kind, counted, n):
    """Rays in a scene without nodes hit nothing, and only the queue's kind counts them."""
    import ctypes as C
    import torch
    scene = make_scene(rb.SCENE_CORNELL).device_scene()
    scene.node_count = 0
    rays = torch.ones((n, 8), dtype=torch.float32, device="cuda")
    ids, t = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.float32, device="cuda")
    values = (C.c_uint64 * 8)()
    rb.check(rb.load().restir_counters(1, values), "counters")
    rb.check(rb.load().restir_trace(None, scene, rays.data_ptr(), ids.data_ptr(), t.data_ptr(), n, kind, None), "restir_trace")
    torch.cuda.synchronize()
    rb.check(rb.load().restir_counters(0, values), "counters")
    assert (ids == -1).all() and (t == 1.0).all()
    assert sum(values[0:4]) == counted * n


class Shifted(SceneSetup):
    """A scene whose device rows start 16 bytes past a 32-byte boundary."""

    def device_scene(self):
        import torch
        scene = super().device_scene()
        data = self.bvh_data if self.bvh_data is not None else self.bvh.data
        rows = torch.zeros(data.size + 4, dtype=torch.float32, device="cuda")
        rows[4:] = torch.from_numpy(data).cuda()
        self.keep.append(rows)
        scene.bvh = rows[4:].data_ptr()
        return scene


@pytest.mark.gpu
@pytest.mark.parametrize("wavefront", [False, True])
@pytest.mark.parametrize("rows", ["shifted", "padded"])
def test_frame_of_rows_on_16_bytes(rows, wavefront):
    """Every pass that traces, through its instance for rows that cannot be read 32 bytes at a time: a buffer on 16
    bytes, and one row of padding before the triangles."""
    from oracle.frame import run_checked
    setup = make_scene(rb.SCENE_COURTYARD, 3, 20_000, extra_lights=8)
    if rows == "padded":
        padded(setup, 1)
    else:
        setup = Shifted(setup.mesh, setup.bvh, setup.lights, setup.settings, setup.materials)
    assert not rb.load().restir_bvh_wide_rows(setup.device_scene())
    setup.settings.grid_mode = rb.GRID_DETERMINISTIC
    report, _, _ = run_checked(setup, 112, 62, 3, setup.settings, gi_wavefront=wavefront)
    assert report == {}, report


@pytest.mark.gpu
def test_watertight_unaligned_rows():
    setup = make_scene(rb.SCENE_CITY, 0, 60_000)
    check(setup, seeded_rays(setup, 20_000, seed=8), rb.TRACE_CLOSEST_WATERTIGHT, offset=4)
