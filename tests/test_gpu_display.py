"""The display and TAA kernels at the edges of their blocks and with images aligned to floats only; the filmic
curve on every float."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import oracle as O
from phantasyenginetestbed_gb300 import build as B
from phantasyenginetestbed_gb300.renderer import scale, taa_resolve
from tests.helpers import device_empty, from_device, to_device

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def test_filmic_curve_is_the_divided_one(tmp_path):
    out = tmp_path / "filmic_test"
    subprocess.run([B._nvcc(), *B.ARCH, "-std=c++17", "-fmad=false", f"-I{ROOT / 'include'}", f"-I{B.CSRC / 'device'}",
                    str(ROOT / "tests/cpp/filmic_test.cu"), "-o", str(out)], check=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_linear_axis_of_any_size(tmp_path):
    out = tmp_path / "sampling_test"
    subprocess.run([B._nvcc(), *B.ARCH, "-std=c++17", "-fmad=false", f"-I{ROOT / 'include'}", f"-I{B.CSRC / 'device'}",
                    str(ROOT / "tests/cpp/sampling_test.cu"), "-o", str(out)], check=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def _floats(a, shift):
    """`a` on the device, `shift` floats past an aligned address."""
    import torch
    buf = torch.empty(a.size + shift, dtype=torch.float32, device="cuda")
    buf[shift:] = torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda()
    return buf[shift:]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("src,dst", [((1, 1), (1, 1)), ((5, 3), (33, 65)), ((64, 64), (31, 17)), ((40, 23), (97, 130)),
                                     ((3, 200), (64, 63)), ((200, 2), (31, 129))])
def test_scaling_pass_edges(src, dst, shift):
    import torch
    img = np.random.default_rng(src[0] * 7 + dst[1]).uniform(0, 1.2, (src[1], src[0], 4)).astype(np.float32)
    d_src = _floats(img, shift)
    d_dst = device_empty(dst[0] * dst[1], np.dtype((np.float32, 4)))
    scale(src, d_src, dst, d_dst)
    torch.cuda.synchronize()
    assert np.array_equal(from_device(d_dst, np.float32).reshape(dst[1], dst[0], 4), O.scale(img, dst))


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("res", [(1, 1), (33, 5), (64, 4), (31, 9)])
def test_taa_edges(res, shift):
    import torch
    W, H = res
    rng = np.random.default_rng(W + H)
    cur, hist = (rng.uniform(0, 2, (H, W, 4)).astype(np.float32) for _ in range(2))
    vel, pvel = ((rng.normal(size=(H, W, 2)) * 0.05 + 1e-3).astype(np.float32) for _ in range(2))
    rough = rng.uniform(0, 1, (H, W)).astype(np.float32)
    oc, oh = (device_empty(W * H, np.dtype((np.float32, 4))) for _ in range(2))
    taa_resolve(res, to_device(cur), _floats(hist, shift), oc, oh, _floats(vel, shift), _floats(pvel, shift), to_device(rough))
    torch.cuda.synchronize()
    want_c, want_h = O.taa(cur, hist, rough, vel, pvel)
    assert np.array_equal(from_device(oc, np.float32).reshape(H, W, 4), want_c)
    assert np.array_equal(from_device(oh, np.float32).reshape(H, W, 4), want_h)


@pytest.mark.parametrize("rows", [6079, 6080, 12160, 24319, 24323])   # 1, 2, 4, 4 and 8 rows a warp on 152 SMs
def test_scaling_rows_per_warp(rows):
    import torch
    img = np.random.default_rng(rows).uniform(0, 1.2, (29, 37, 4)).astype(np.float32)
    d_dst = device_empty(31 * rows, np.dtype((np.float32, 4)))
    scale((37, 29), to_device(img), (31, rows), d_dst)
    torch.cuda.synchronize()
    assert np.array_equal(from_device(d_dst, np.float32).reshape(rows, 31, 4), O.scale(img, (31, rows)))


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("res", [(1, 1), (33, 5), (64, 4)])
def test_taa_without_velocities(res, shift):
    import torch
    W, H = res
    rng = np.random.default_rng(W * H)
    cur, hist = (rng.uniform(0, 2, (H, W, 4)).astype(np.float32) for _ in range(2))
    pvel = (rng.normal(size=(H, W, 2)) * 0.05).astype(np.float32)
    rough = rng.uniform(0, 1, (H, W)).astype(np.float32)
    for prev in (None, pvel):
        oc, oh = (device_empty(W * H, np.dtype((np.float32, 4))) for _ in range(2))
        taa_resolve(res, to_device(cur), _floats(hist, shift), oc, oh, None, None if prev is None else _floats(prev, shift),
                    to_device(rough))
        torch.cuda.synchronize()
        zero = np.zeros((H, W, 2), np.float32)
        want_c, want_h = O.taa(cur, hist, rough, zero, zero if prev is None else prev)
        assert np.array_equal(from_device(oc, np.float32).reshape(H, W, 4), want_c)
        assert np.array_equal(from_device(oh, np.float32).reshape(H, W, 4), want_h)


@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("rows", [262140, 262141, 262149, 524280])   # the last of one block per grid row, then two
def test_taa_of_high_images(rows, moving):
    import torch
    W = 2
    rng = np.random.default_rng(rows)
    cur, hist = (rng.uniform(0, 2, (rows, W, 4)).astype(np.float32) for _ in range(2))
    vel = (rng.normal(size=(rows, W, 2)) * 1e-5).astype(np.float32) if moving else None
    rough = rng.uniform(0, 1, (rows, W)).astype(np.float32)
    oc, oh = (device_empty(W * rows, np.dtype((np.float32, 4))) for _ in range(2))
    taa_resolve((W, rows), to_device(cur), to_device(hist), oc, oh, to_device(vel) if moving else None, None, to_device(rough))
    torch.cuda.synchronize()
    want_c, want_h = O.taa(cur, hist, rough, np.zeros((rows, W, 2), np.float32) if vel is None else vel,
                           np.zeros((rows, W, 2), np.float32))
    assert np.array_equal(from_device(oc, np.float32).reshape(rows, W, 4), want_c)
    assert np.array_equal(from_device(oh, np.float32).reshape(rows, W, 4), want_h)
