"""Host code around the device (scene upload, launch sequences) run without one: the library's own objects
linked with a CUDA runtime that keeps device memory on the host and records kernels instead of running them
(tests/cpp/fake_cudart.cpp). Each case runs in a process of its own."""
import ctypes as C
import multiprocessing
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

import phantasyenginetestbed_gb300 as P
from phantasyenginetestbed_gb300 import build as B
from phantasyenginetestbed_gb300 import native

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def fake_library(tmp_path_factory):
    objects = [B.BUILD / f"{s.stem}{s.suffix}.o" for group in B.sources() for s in group]
    B.build(force=not all(o.exists() for o in objects))
    out = tmp_path_factory.mktemp("fake") / "libphe_fake.so"
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-fPIC", "-shared", "-std=c++17", f"-I{B._cuda_include()}",
                    "-Wl,-Bsymbolic", "-Wl,-z,lazy", "-o", str(out), str(ROOT / "tests/cpp/fake_cudart.cpp"), *map(str, objects),
                    "-lpthread", "-ldl"], check=True)
    return str(out)


def _in_child(case, *args):
    p = multiprocessing.get_context("spawn").Process(target=case, args=args)
    p.start()
    p.join(120)
    assert p.exitcode == 0, f"exit code {p.exitcode}"


def _use(library):
    """Makes the package of this process use the library with the recording runtime."""
    lib = C.CDLL(library, mode=os.RTLD_LAZY)
    for name, (res, args) in native.SIGNATURES.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    lib.fake_allocation.restype = C.c_void_p
    lib.fake_launch.restype = C.c_char_p
    lib.fake_launch_scene.restype = C.c_void_p
    lib.fake_fail_new.argtypes = [C.c_long]
    native._lib = lib
    return lib


def _allocation(lib, i):
    size = C.c_size_t()
    address = lib.fake_allocation(i, C.byref(size))
    return np.frombuffer(C.string_at(address, size.value), np.uint8)


def _launches(lib):
    """Every launch so far: kernel, grid, block, dynamic shared memory, whether it may start early."""
    out = []
    for i in range(lib.fake_num_launches()):
        grid, block, smem, early = (C.c_uint32 * 3)(), (C.c_uint32 * 3)(), C.c_size_t(), C.c_int()
        name = lib.fake_launch(i, grid, block, C.byref(smem), C.byref(early)).decode()
        out.append((name, tuple(grid), tuple(block), smem.value, bool(early.value)))
    return out


def _upload(lib, nodes, verts):
    """The bytes of the device nodes and of the rest of the scene's allocation."""
    scene = P.Scene(nodes, verts)
    data = _allocation(lib, lib.fake_num_allocations() - 1)
    scene.close()
    return data[:64 * len(nodes)], data[(64 * len(nodes) + 255) // 256 * 256:]


def _reached(nodes):
    """The tree that the root of device nodes reaches, depth first, without the numbers of its nodes."""
    n = nodes.view(np.int32).reshape(-1, 16)
    out, stack = [], [0]
    while stack:
        node = n[stack.pop()].copy()
        inner = np.nonzero(node[12:14] >= 0)[0] + 12
        stack += list(node[inner])
        node[inner] = 0
        out.append(node)
    return np.array(out)


def _unreached_nodes(library, last):
    lib = _use(library)
    b = P.build_sbvh(P.generate_scene(64, 100, False, 7).tri_verts)
    assert len(b.nodes) > 2048   # some nodes stay behind the ones moved to the front
    stray = np.zeros(3, P.NODE_DTYPE)
    stray["iData"] = [[0x10000000, 0x7FFFFFFF, 0, 0], [len(b.nodes) + 2, len(b.nodes) + 3, 0, 0], [-5, 3, 0, 1 << 30]]
    stray["fData"] = np.nan
    if last:
        nodes = np.concatenate([b.nodes, stray])
    else:   # behind the root: the reached nodes' references move with them
        nodes = np.concatenate([b.nodes[:1], stray, b.nodes[1:]])
        reached = np.r_[0, 4:len(nodes)]
        for c in (0, 1):
            inner = reached[nodes["iData"][reached, 2 + c] == 0]
            nodes["iData"][inner, c] += 3
    want_nodes, want_rest = _upload(lib, b.nodes, b.verts)
    got_nodes, got_rest = _upload(lib, nodes, b.verts)
    assert np.array_equal(got_rest, want_rest)
    assert np.array_equal(_reached(got_nodes), _reached(want_nodes))


@pytest.mark.parametrize("last", [True, False])
def test_upload_ignores_unreached_nodes(fake_library, last):
    """Nodes that the root does not reach are not validated: whatever they refer to, the upload is that of the tree
    without them."""
    _in_child(_unreached_nodes, fake_library, last)


def _taa_heights(library):
    lib = _use(library)
    buf = C.c_void_p(1 << 20)
    for h in (1, 4, 5, 262140, 262141, 262149, 524279, 524280):
        assert lib.phe_taa_resolve(40, h, buf, buf, None, None, None, buf, buf, None) == native.PHE_OK, h
        name, grid, block, _, _ = _launches(lib)[-1]
        assert "taa_kernel" in name and grid[0] * block[0] >= 40 and grid[1] * grid[2] * block[1] >= h
    n = lib.fake_num_launches()
    assert lib.phe_taa_resolve(40, 524281, buf, buf, None, None, None, buf, buf, None) == native.PHE_ERR_CUDA
    assert lib.fake_num_launches() == n


def test_taa_takes_images_up_to_524280_rows(fake_library):
    _in_child(_taa_heights, fake_library)


def _batch_grids(library, graph):
    from phantasyenginetestbed_gb300.batch import Batch
    lib = _use(library)
    b = P.build_sbvh(P.generate_scene(8, 2, False, 7).tri_verts)
    for device, blocks in ((0, 3), (1, 5), (0, 3)):
        lib.fake_set_device(device)
        lib.fake_set_occupancy(device, blocks)
        scene = P.Scene(b.nodes, b.verts)
        batch = Batch([scene], [(0, 0, 1 << 20, 1 << 20, 2 << 20), (0, 1, 1 << 20, 3 << 20, 4 << 20)], use_graph=graph)
        batch.launch()
        name, grid, block, _, _ = _launches(lib)[-1]
        assert "batch_kernel" in name and grid == (152 * blocks, 1, 1) and block[0] == 128, (name, grid)


@pytest.mark.parametrize("graph", [False, True])
def test_batch_grid_follows_the_device(fake_library, graph):
    """The resident blocks that size a batch's grid are those of the device it is launched on."""
    _in_child(_batch_grids, fake_library, graph)


def _frame_launches(library, schedule, timed, want):
    from phantasyenginetestbed_gb300 import renderer as R
    lib = _use(library)
    s = P.generate_scene(8, 2, False, 7)
    b = P.build_sbvh(s.tri_verts)
    r = R.CudaTracerRenderer()
    r.setStaticScene(P.Scene.from_bvh(b, s))
    r.setTargetResolution((64, 64))
    r.set_shadow_schedule(schedule)
    r.set_kernel_timing(timed)
    r.updateCamera((0.5, -0.3, 0.6), (0.0, 0.8, -0.6), (0.0, 0.6, 0.8), 60.0)
    n = lib.fake_num_launches()
    r.render(R.make_lights(np.array([[0.1, 0.1, 0.5]], np.float32), range_=100.0))
    got = [(k, early) for name, _, _, _, early in _launches(lib)[n:]
           for k in ("primary", "any_queue", "bounce", "resolve_taa") if k + "_kernel" in name]
    assert got == want, got


@pytest.mark.parametrize("schedule,timed,want", [
    (2, False, [("primary", False), ("bounce", True), ("any_queue", True), ("resolve_taa", True)]),
    (2, True, [("primary", False), ("bounce", False), ("any_queue", False), ("resolve_taa", False)]),
    (0, False, [("primary", False), ("any_queue", False), ("bounce", True), ("any_queue", False), ("resolve_taa", True)]),
    (1, False, [("primary", False), ("any_queue", False), ("bounce", False), ("any_queue", False), ("resolve_taa", False)])])
def test_stages_start_early_only_behind_a_kernel(fake_library, schedule, timed, want):
    """A frame stage is launched early only where the kernel before it is the stream's last work: not behind the events
    of a timed frame, nor behind the fork and the join of the beside schedule (1)."""
    _in_child(_frame_launches, fake_library, schedule, timed, want)


def _upload_without_memory(library):
    lib = _use(library)
    s = P.generate_scene(8, 2, False, 7)
    b = P.build_sbvh(s.tri_verts)
    P.Scene.from_bvh(b, s).close()   # the device's own allocations are made
    live = lib.fake_live_allocations()
    datas, h = b.slot_datas(s.datas), C.c_void_p()
    for k in range(10000):
        lib.fake_fail_new(k)
        st = lib.phe_scene_create(native.ptr(b.nodes), len(b.nodes), native.ptr(b.verts), native.ptr(datas), len(b.verts),
                                  native.ptr(s.materials), len(s.materials), native.PTR_HOST, C.byref(h))
        lib.fake_fail_new(-1)
        if st == native.PHE_OK:
            break
        assert st == native.PHE_ERR_OUT_OF_MEMORY and not h.value and lib.fake_live_allocations() == live, (k, st)
    assert k > 10 and h.value
    lib.phe_scene_destroy(h)
    assert lib.fake_live_allocations() == live


def test_upload_reports_a_failed_host_allocation(fake_library):
    """Whichever host allocation fails, the upload returns an error and keeps no device memory."""
    _in_child(_upload_without_memory, fake_library)


def _small_casts(library):
    lib = _use(library)
    b = P.build_sbvh(P.generate_scene(64, 100, False, 7).tri_verts)
    scene, buf = P.Scene(b.nodes, b.verts), 1 << 20
    for n in (1, 4096, 8192, 49152, 77824, 77825):
        for cast in (P.cast_closest, P.cast_closest_plain, P.cast_any):
            cast(scene, buf, buf, n)
            name, grid, block, smem, _ = _launches(lib)[-1]
            warps = grid[0] * block[0] // 32
            assert smem == 0 and block[0] <= 128 and warps <= max((n + 127) // 128 * 4, 152 * 7), (name, grid, block, smem, n)


def test_small_casts_leave_room_for_others(fake_library):
    """A cast of few rays holds no SM for itself: launches of other streams run beside it."""
    _in_child(_small_casts, fake_library)


def _direction_limit(library):
    lib = _use(library)
    b = P.build_sbvh(P.generate_scene(8, 2, False, 7).tri_verts * np.float32(1024))   # edges long enough for a finite bound

    def limit(verts):
        scene = P.Scene(b.nodes, verts)
        P.cast_closest(scene, 1 << 20, 1 << 20, 1000)
        s = C.string_at(lib.fake_launch_scene(lib.fake_num_launches() - 1), 128)
        scene.close()
        return np.frombuffer(s, np.float32)[30]

    want = limit(b.verts)
    edge = max(np.abs(b.verts[k][:, :3] - b.verts["v0"][:, :3]).max() for k in ("v1", "v2"))
    assert np.isclose(want, 2.0**124 / (6.0 * np.float64(edge)**2), rtol=1e-6)
    for k, value in (("v0", np.nan), ("v1", np.inf), ("v2", -np.inf)):
        v = b.verts.copy()
        v[k][len(v) // 2, 1] = value
        assert limit(v) == want
    v = b.verts.copy()
    v["v1"][0, 2] = 3e38
    assert 0 < limit(v) < 1


def test_direction_limit_of_a_scene(fake_library):
    """The bound below which rays take the fast triangle test: from the finite edges alone."""
    _in_child(_direction_limit, fake_library)
