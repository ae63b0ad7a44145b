"""The packed triangle test's edges: its reciprocal against the correctly rounded one on every float in
range, and rays whose direction lies on either side of the bound that selects it (DeviceScene::dirLimit)."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import phantasyenginetestbed_gb300 as P
from oracle import oracle as O
from phantasyenginetestbed_gb300 import build as B
from tests.helpers import device_empty, from_device, random_rays, to_device

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def test_reciprocal_is_correctly_rounded_in_range(tmp_path):
    out = tmp_path / "reciprocal_test"
    subprocess.run([B._nvcc(), *B.ARCH, "-std=c++17", "-fmad=false", f"-I{ROOT / 'include'}", f"-I{B.CSRC / 'device'}",
                    str(ROOT / "tests/cpp/reciprocal_test.cu"), "-o", str(out)], check=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("scene_exp,dir_exp", [(0, 0), (0, 100), (0, -100), (40, 0), (40, 45), (40, 57), (40, 70)])
def test_long_directions_on_large_scenes(scene_exp, dir_exp):
    """Vertices scaled by 2^scene_exp, directions by 2^dir_exp: determinants from small to beyond 2^126 (where
    the reciprocal is subnormal) and to overflow. Hit or miss and visibility as the oracle's; every reported hit
    is what the oracle's triangle test gives for that triangle, bit for bit; and the oracle's hit, where no
    hit is a NaN (the overflowing determinants accept triangles with NaN u or v, and which of them
    is kept depends on the order of the visits)."""
    import torch
    s = P.generate_scene(24, 20, True, 5)
    scale = np.float32(2.0) ** np.float32(scene_exp)
    b = P.build_sbvh(s.tri_verts * scale)
    scene = P.Scene(b.nodes, b.verts)
    k = s.scale
    rays = random_rays(20011, [0, 0, 0.02 * k], [k, k, 0.3 * k], 9, tmin=0.0)
    rays["origin"] *= scale
    rays["dir"] *= np.float32(2.0) ** np.float32(dir_exp)
    d_rays = to_device(rays)
    orc = O.cast_rays(b.nodes, b.verts, rays, mode=O.MODE_GPU)
    for cast in (P.cast_closest, P.cast_closest_plain):
        d_hits = device_empty(len(rays), P.RAY_HIT_DTYPE)
        cast(scene, d_rays, d_hits, len(rays))
        torch.cuda.synchronize()
        hits = from_device(d_hits, P.RAY_HIT_DTYPE)
        hit = np.nonzero(hits["triangleIndex"] != 0xFFFFFFFF)[0]
        assert np.array_equal(hits["triangleIndex"] == 0xFFFFFFFF, orc["triangleIndex"] == 0xFFFFFFFF)
        for i in hit[::7]:
            ok, *tuv = O.intersect_tri(b.verts[hits["triangleIndex"][i]], rays["origin"][i], rays["dir"][i])
            assert ok and np.array_equal(np.float32(tuv), [hits[f][i] for f in ("t", "u", "v")], equal_nan=True), i
        if not np.isnan(orc["u"] + orc["v"]).any():
            rep = O.compare_closest(hits, orc, rays, b.slot_to_tri, b.verts)
            assert rep["ok"] and rep["near_ties"] <= 2, rep
    d_vis = device_empty(len(rays), np.uint8)
    P.cast_any(scene, d_rays, d_vis, len(rays))
    torch.cuda.synchronize()
    assert np.array_equal(from_device(d_vis, np.uint8), O.any_rays(b.nodes, b.verts, rays))
    assert scene.status() == 0
    if scene_exp == 0 and dir_exp == 0:
        assert (orc["triangleIndex"] != 0xFFFFFFFF).sum() > 1000


def test_triangles_with_an_edge_that_is_not_finite():
    """Vertices at infinity and NaN in a quarter of the slots: their triangles are never hit, as in the oracle, and the
    rays of the scene take the fast path in every layout."""
    import torch
    s = P.generate_scene(24, 20, True, 5)
    b = P.build_sbvh(s.tri_verts)
    verts = b.verts.copy()
    rng = np.random.default_rng(3)
    for i in rng.permutation(len(verts))[:len(verts) // 4]:
        verts[("v0", "v1", "v2")[rng.integers(3)]][i, rng.integers(3)] = (np.inf, -np.inf, np.nan)[rng.integers(3)]
    k = s.scale
    rays = random_rays(60011, [0, 0, 0.02 * k], [k, k, 0.3 * k], 9, tmin=0.0)
    rays["dir"][::5, 2] = 0.0   # products of 0 and infinity
    d_rays = to_device(rays)
    orc = O.cast_rays(b.nodes, verts, rays, mode=O.MODE_GPU)
    lit = O.any_rays(b.nodes, verts, rays)
    slots = orc["triangleIndex"][orc["triangleIndex"] != 0xFFFFFFFF]
    assert len(slots) > 1000 and all(np.isfinite(verts[f][slots, :3]).all() for f in ("v0", "v1", "v2"))
    scene = P.Scene(b.nodes, verts)
    for layout in range(3):
        scene.set_layout(layout)
        for n in (1001, len(rays)):
            hits, vis = device_empty(n, P.RAY_HIT_DTYPE), device_empty(n, np.uint8)
            P.cast_closest(scene, d_rays, hits, n)
            P.cast_any(scene, d_rays, vis, n)
            torch.cuda.synchronize()
            rep = O.compare_closest(from_device(hits, P.RAY_HIT_DTYPE), orc[:n], rays[:n], b.slot_to_tri, verts)
            assert rep["ok"] and rep["near_ties"] <= 2, rep
            assert np.array_equal(from_device(vis, np.uint8), lit[:n])
    assert scene.status() == 0
