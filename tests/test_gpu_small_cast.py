"""Launches of few rays (their own kernel, then one wave without a work counter) give the bits of the same rays
in a large launch, at the sizes where the kernel, its rays per warp and its blocks change."""
import functools

import numpy as np
import pytest

import phantasyenginetestbed_gb300 as P
from oracle import oracle as O
from tests.helpers import C1_CAM, built_scene, cam_struct, device_empty, from_device, random_rays, to_device

pytestmark = pytest.mark.gpu
N = 400_000   # more than one wave of any device of 152 SMs


@functools.lru_cache(maxsize=None)
def _large(name):
    """The scene, N rays on the device and their results in one launch of the persistent kernels."""
    import torch
    if name == "one_leaf":
        b = P.build_sbvh(np.array([[0, 0, 0, 1, 0, 0, 0, 1, 0], [0, 0, 0.5, 1, 0, 0.5, 0, 1, 0.5]], np.float32))
        k = 1.0
    else:
        s, b = built_scene(name)
        k = s.scale
    scene = P.Scene(b.nodes, b.verts)
    rays = random_rays(N, [0, 0, 0.01 * k], [k, k, 0.3 * k], 21)
    d_rays = to_device(rays)
    hits, vis = device_empty(N, P.RAY_HIT_DTYPE), device_empty(N, np.uint8)
    P.cast_closest(scene, d_rays, hits, N)
    P.cast_any(scene, d_rays, vis, N)
    torch.cuda.synchronize()
    return b, scene, rays, d_rays, from_device(hits, P.RAY_HIT_DTYPE), from_device(vis, np.uint8)


@pytest.mark.parametrize("name", ["c1_64_100", "c2_256_2000", "one_leaf"])
@pytest.mark.parametrize("n", [1, 31, 33, 152 * 32 + 1, 152 * 16 * 4, 152 * 16 * 4 + 1, 152 * 16 * 8 + 1, 49152, 49153,
                               152 * 16 * 32, 152 * 16 * 32 + 1, 152 * 1280, 152 * 1280 + 1])
def test_small_launches_give_the_large_launch(name, n):
    import torch
    b, scene, rays, d_rays, hits, vis = _large(name)
    for cast in (P.cast_closest, P.cast_closest_plain):
        out = device_empty(n, P.RAY_HIT_DTYPE)
        cast(scene, d_rays, out, n)
        torch.cuda.synchronize()
        assert np.array_equal(from_device(out, np.uint8), hits[:n].view(np.uint8))
    order = np.random.default_rng(n).permutation(n).astype(np.uint32)
    for scatter in (None, order):
        out = torch.full((n + 16,), 7, dtype=torch.uint8, device="cuda")
        P.cast_any(scene, d_rays, out, n, scatter=None if scatter is None else to_device(scatter))
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert np.array_equal(got[:n] if scatter is None else got[:n][order], vis[:n])
        assert np.all(got[n:] == 7)
    assert scene.status() == 0
    if n == 33:
        assert np.array_equal(vis[:20000], O.any_rays(b.nodes, b.verts, rays[:20000]))
        orc = O.cast_rays(b.nodes, b.verts, rays[:20000], mode=O.MODE_GPU)
        assert O.compare_closest(hits[:20000], orc, rays[:20000], b.slot_to_tri, b.verts)["ok"]


@pytest.mark.parametrize("shift", [0, 16])   # the buffer aligned to 32 bytes or to 16 only
@pytest.mark.parametrize("res,order", [((1, 1), 0), ((257, 3), 0), ((100, 77), 0), ((8, 8), 1), ((264, 24), 1)])
def test_primary_rays_at_block_edges(res, order, shift):
    import math

    import torch
    cam = O.camera_def(C1_CAM["pos"], C1_CAM["dir"], C1_CAM["up"], math.radians(60), res)
    n = res[0] * res[1]
    buf = torch.full((shift + n * 32 + 32,), 7, dtype=torch.uint8, device="cuda")
    P.gen_primary_rays(buf[shift:], cam_struct(cam), res, jitter=(0.25, -0.125), order=order)
    torch.cuda.synchronize()
    got = buf.cpu().numpy()
    want = O.gen_primary(cam, res, jitter=(0.25, -0.125), order=order)
    assert np.array_equal(got[shift:shift + n * 32], want.view(np.uint8))
    assert np.all(got[:shift] == 7) and np.all(got[shift + n * 32:] == 7)


@pytest.mark.parametrize("n", [152 * 1280 + 1, 300_001])
def test_counter_cleared_in_and_out_of_a_graph(n):
    """Rays written by the work before on the stream; cleared by a kernel that runs beside the cast, or by a memset
    inside a graph, replayed."""
    import torch
    _, scene, _, d_rays, hits, vis = _large("c2_256_2000")
    stream = torch.cuda.Stream()
    rays, out = torch.empty_like(d_rays), device_empty(n, P.RAY_HIT_DTYPE)
    lit = device_empty(n, np.uint8)

    def work():
        rays.copy_(d_rays)
        P.cast_closest(scene, rays, out, n, stream=stream)
        rays.zero_()
        rays.copy_(d_rays)
        P.cast_any(scene, rays, lit, n, stream=stream)
        rays.zero_()

    def check():
        stream.synchronize()
        assert np.array_equal(from_device(out, np.uint8), hits[:n].view(np.uint8))
        assert np.array_equal(from_device(lit, np.uint8), vis[:n])
        assert scene.status() == 0
        out.zero_()
        lit.zero_()
        torch.cuda.synchronize()

    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for _ in range(2):
            work()
        check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        work()
    for _ in range(2):
        with torch.cuda.stream(stream):
            graph.replay()
        check()


@pytest.mark.parametrize("n", [k * 152 * 7 + d for k in (4, 8, 16) for d in (0, 1)])
def test_any_hit_where_the_rays_per_warp_change(n):
    import torch
    _, scene, _, d_rays, _, vis = _large("c2_256_2000")
    order = np.random.default_rng(n).permutation(n).astype(np.uint32)
    out = torch.full((n + 16,), 7, dtype=torch.uint8, device="cuda")
    P.cast_any(scene, d_rays, out, n, scatter=to_device(order))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.array_equal(got[:n][order], vis[:n]) and np.all(got[n:] == 7)
