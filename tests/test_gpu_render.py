"""Frustum culling and Morton voxelisation on the GPU against the float32 CPU restatement: every mask bit, Morton
code and voxel centre equal (the kernels use single rounded float operations for that reason).  Covers empty input,
sizes that are not a multiple of the four points a thread takes, points behind the camera / outside the planes /
on image borders, negative coordinates, and a multi-million point cloud through properties."""
import concurrent.futures
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from lingbot_map_b200 import render_ops as RO
from oracle import render_oracle as R

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _camera(seed):
    rs = np.random.RandomState(seed)
    q, _ = np.linalg.qr(rs.standard_normal((3, 3)))
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    return q.astype(np.float32), (rs.standard_normal(3) * 0.5).astype(np.float32)


@pytest.mark.parametrize("n", [0, 1, 3, 4, 5, 1023, 100003])
def test_frustum_cull_bit_exact(n):
    rs = np.random.RandomState(n)
    pts = (rs.standard_normal((n, 3)) * 3).astype(np.float32)
    Rm, t = _camera(n + 1)
    args = (300.0, 310.0, 259.0, 189.0, 518, 378, 0.1, 6.0)
    got = RO.frustum_cull(torch.from_numpy(pts).to(DEV), torch.from_numpy(Rm).to(DEV), torch.from_numpy(t).to(DEV), *args)
    want = R.frustum_cull(pts, Rm, t, *args)
    assert got.dtype == torch.bool and got.shape == (n,)
    assert np.array_equal(got.cpu().numpy(), want)
    if n > 1000:
        assert 0.02 < want.mean() < 0.9          # the case exercises both outcomes


@pytest.mark.parametrize("n,voxel", [(0, 0.05), (1, 0.05), (7, 0.5), (4097, 0.05), (250000, 0.02)])
def test_voxelize_frame_bit_exact(n, voxel):
    rs = np.random.RandomState(n + 7)
    xyz = (rs.standard_normal((n, 3)) * 2).astype(np.float32)
    rgb = rs.rand(n, 3).astype(np.float32)
    c, col, codes = RO.voxelize_frame(torch.from_numpy(xyz).to(DEV), torch.from_numpy(rgb).to(DEV), voxel)
    wc, wcol, wcodes = R.voxelize_frame(xyz, rgb, voxel)
    assert np.array_equal(codes.cpu().numpy(), wcodes)
    assert np.array_equal(c.cpu().numpy(), wc)
    assert np.array_equal(col.cpu().numpy(), wcol)
    if n:
        assert np.all(np.diff(wcodes) > 0)       # sorted and unique


def test_large_cloud_properties():
    """8 M points (96 MB of xyz: larger than L2's share): idempotence of voxelisation on its own output centres, and
    the culled set is exactly the set whose projection the oracle accepts on a sample."""
    n = 8_000_000
    g = torch.Generator(device=DEV).manual_seed(1)
    xyz = torch.randn(n, 3, device=DEV, generator=g) * 2
    rgb = torch.rand(n, 3, device=DEV, generator=g)
    c, col, codes = RO.voxelize_frame(xyz, rgb, 0.05)
    assert torch.all(codes[1:] > codes[:-1])
    c2, _, codes2 = RO.voxelize_frame(c, col, 0.05)
    assert torch.equal(codes2, codes) and torch.equal(c2, c)          # centres map to their own voxels
    Rm, t = _camera(3)
    args = (300.0, 310.0, 259.0, 189.0, 518, 378, 0.1, 6.0)
    vis = RO.frustum_cull(xyz, torch.from_numpy(Rm), torch.from_numpy(t), *args)
    idx = torch.arange(0, n, 9973, device=DEV)
    want = R.frustum_cull(xyz[idx].cpu().numpy(), Rm, t, *args)
    assert np.array_equal(vis[idx].cpu().numpy(), want)


@pytest.mark.parametrize("n", [148 * 2048 + 5, 256 * 2048 - 1, 256 * 2048])
def test_voxelize_frame_sort_up_to_its_largest(n):
    """More tiles than SMs, up to the largest cloud the sort takes (256 tiles meet at its barriers), again and again from two threads at
    once, each on its stream."""
    rs = np.random.RandomState(n % 1000)
    xyz = (rs.randint(-300, 301, (n, 3)) + 0.5).astype(np.float32)
    rgb = rs.rand(n, 3).astype(np.float32)
    wc, wcol, wcodes = R.voxelize_frame(xyz, rgb, 1.0)
    dx, dr = torch.from_numpy(xyz).to(DEV), torch.from_numpy(rgb).to(DEV)
    torch.cuda.synchronize()

    def calls(_):
        with torch.cuda.stream(torch.cuda.Stream(DEV)):
            got = [RO.voxelize_frame(dx, dr, 1.0) for _ in range(12)]
            torch.cuda.current_stream().synchronize()
            return got

    with concurrent.futures.ThreadPoolExecutor(2) as pool:
        results = [r for part in pool.map(calls, range(2)) for r in part]
    for c, col, codes in results:
        assert np.array_equal(codes.cpu().numpy(), wcodes) and np.array_equal(c.cpu().numpy(), wc) and np.array_equal(col.cpu().numpy(), wcol)


@pytest.mark.parametrize("sms", [8, 16, 72])
@pytest.mark.parametrize("n", [2048, 40 * 2048 + 1, 256 * 2048])
def test_voxelize_frame_on_part_of_the_gpu(sms, n):
    """A stream that owns a few of the SMs: the sort's tiles do not all run at once there, and a CTA takes several."""
    from torch.cuda import green_contexts
    if not green_contexts.SUPPORTED:
        pytest.skip("PyTorch was built without green contexts")
    rs = np.random.RandomState(sms + n % 1000)
    xyz = (rs.randint(-300, 301, (n, 3)) + 0.5).astype(np.float32)
    rgb = rs.rand(n, 3).astype(np.float32)
    wc, wcol, wcodes = R.voxelize_frame(xyz, rgb, 1.0)
    dx, dr = torch.from_numpy(xyz).to(DEV), torch.from_numpy(rgb).to(DEV)
    torch.cuda.synchronize()
    part = torch.cuda.GreenContext.create(sms, 0)
    part.set_context()
    try:
        got = RO.voxelize_frame(dx, dr, 1.0)
        torch.cuda.synchronize()
    finally:
        part.pop_context()
    for a, b in zip(got, (wc, wcol, wcodes)):
        assert np.array_equal(a.cpu().numpy(), b)


def test_voxelize_frame_waits_as_the_program_chose():
    """The wait for the number of voxels, behind half a second of earlier work on the stream, in a process that has its threads sleep in
    waits for the GPU: the thread spends next to no processor time in it."""
    code = """
import ctypes, time
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0 and cu.cuDevicePrimaryCtxSetFlags_v2(0, 4) == 0           # CU_CTX_SCHED_BLOCKING_SYNC
import torch
from lingbot_map_b200 import render_ops as RO
xyz, rgb = torch.rand(50000, 3, device="cuda:0"), torch.rand(50000, 3, device="cuda:0")
want = RO.voxelize_frame(xyz, rgb, 0.05)
torch.cuda.synchronize()
torch.cuda._sleep(900_000_000)
wall, busy = time.perf_counter(), time.thread_time()
got = RO.voxelize_frame(xyz, rgb, 0.05)
wall, busy = time.perf_counter() - wall, time.thread_time() - busy
assert all(torch.equal(a, b) for a, b in zip(got, want))
assert wall > 0.2, wall
assert busy < 0.25 * wall, (busy, wall)
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 2 * 2048 + 1, 65536])
@pytest.mark.parametrize("extent", [3, 100, 5000, 2 ** 20 - 1])
def test_voxelize_frame_sort_edges(n, extent):
    """The frame-sized sort at the edges of its tiles (2048 points) and for clouds whose voxel indices need from two passes
    (within +-7) over five (below 2^12) to all eight (2^20); every index twice, so that the
    order among equal keys shows in the colours."""
    rs = np.random.RandomState(n + extent)
    idx = rs.randint(-extent, extent + 1, (n, 3))
    idx[n // 2:] = idx[:n - n // 2]
    xyz = (idx + 0.5).astype(np.float32)                   # voxel size 1: exact
    rgb = rs.rand(n, 3).astype(np.float32)
    c, col, codes = RO.voxelize_frame(torch.from_numpy(xyz).to(DEV), torch.from_numpy(rgb).to(DEV), 1.0)
    wc, wcol, wcodes = R.voxelize_frame(xyz, rgb, 1.0)
    assert np.array_equal(codes.cpu().numpy(), wcodes)
    assert np.array_equal(c.cpu().numpy(), wc)
    assert np.array_equal(col.cpu().numpy(), wcol)


@pytest.mark.parametrize("depths", [(0.5, 5.0), (1e-38, 1e-36), (1e36, 3e38)])
@pytest.mark.parametrize("camera_on", ["cpu", "cuda:0"])
def test_frustum_cull_on_image_borders(depths, camera_on):
    """Points whose projections lie within a few rounding steps of the image borders, where the test without divisions must
    hand over to the exact one, and depths whose reciprocal leaves the float range.  Transposed and strided cameras."""
    rs = np.random.RandomState(3)
    n, (fx, fy, cx, cy, W, H) = 40000, (300.0, 310.0, 259.0, 189.0, 518, 378)
    z = np.exp(rs.uniform(np.log(depths[0]), np.log(depths[1]), n)).astype(np.float32)
    u = rs.choice([-1.0, 0.0, W, W - 1, 200.5], n) + rs.randint(-3, 4, n) * rs.choice([0.0, 3e-8, 3e-5, 1e-3, 0.3], n)
    v = rs.choice([-1.0, 0.0, H, H - 1, 100.5], n) + rs.randint(-3, 4, n) * rs.choice([0.0, 3e-8, 3e-5, 1e-3, 0.3], n)
    with np.errstate(over="ignore"):
        cam = np.stack([((u - cx) / fx * z).astype(np.float32), ((v - cy) / fy * z).astype(np.float32), z], axis=1)
    perm = np.array([[0, 1, 0], [0, 0, 1], [1, 0, 0]], np.float32)        # exact in floats; its transpose is not itself
    pts = np.ascontiguousarray(cam @ perm)
    t = np.zeros(3, np.float32)
    args = (fx, fy, cx, cy, W, H, depths[0] * 0.9, min(depths[1] * 1.1, 3.3e38))
    Rm = torch.from_numpy(np.ascontiguousarray(perm.T)).to(camera_on).t()
    tt = torch.zeros(6, device=camera_on)[::2]
    got = RO.frustum_cull(torch.from_numpy(pts).to(DEV), Rm, tt, *args).cpu().numpy()
    with np.errstate(all="ignore"):
        want = R.frustum_cull(pts, perm, t, *args)
    assert np.array_equal(got, want)
    assert 0.02 < want.mean() < 0.98


@pytest.mark.parametrize("W,H", [(0, 378), (518, 0), (0, 0), (-3, 378), (1, 1)])
def test_frustum_cull_of_an_empty_image(W, H):
    """An image without pixels sees nothing, also of the points that project into (-1, 0), which truncation maps to pixel 0; one
    pixel sees those."""
    rs = np.random.RandomState(5)
    n = 4003
    z = rs.uniform(0.5, 5.0, n).astype(np.float32)
    uv = rs.uniform(-2.0, 2.0, (2, n)).astype(np.float32)
    pts = np.ascontiguousarray(np.stack([uv[0] * z / 300, uv[1] * z / 310, z], axis=1).astype(np.float32))
    eye, zero = np.eye(3, dtype=np.float32), np.zeros(3, np.float32)
    args = (300.0, 310.0, 0.0, 0.0, W, H, 0.1, 10.0)
    got = RO.frustum_cull(torch.from_numpy(pts).to(DEV), torch.from_numpy(eye), torch.from_numpy(zero), *args).cpu().numpy()
    assert np.array_equal(got, R.frustum_cull(pts, eye, zero, *args))
    assert got.any() == (W > 0 and H > 0)


@pytest.mark.parametrize("camera_on", ["cpu", "cuda:0"])
@pytest.mark.parametrize("r_shape", [(3, 3), (9,), (1, 9), (9, 1), (1, 3, 3), (3, 3, 1), (3, 1, 3)])
@pytest.mark.parametrize("t_shape", [(3,), (1, 3), (3, 1)])
def test_frustum_cull_takes_a_camera_of_any_shape(camera_on, r_shape, t_shape):
    """Nine and three values in any shape, on the host or on the device, also as every other value of a buffer."""
    rs = np.random.RandomState(8)
    n, args = 5003, (300.0, 310.0, 259.0, 189.0, 518, 378, 0.1, 6.0)
    pts = (3 * rs.standard_normal((n, 3))).astype(np.float32)
    q, _ = np.linalg.qr(rs.standard_normal((3, 3)))
    Rm, t = q.astype(np.float32), (0.5 * rs.standard_normal(3)).astype(np.float32)
    want = R.frustum_cull(pts, Rm, t, *args)
    dense = torch.from_numpy(Rm).to(camera_on).reshape(r_shape)
    apart = torch.stack([dense, 7 + dense], dim=-1)[..., 0]
    for r in (dense, apart):
        got = RO.frustum_cull(torch.from_numpy(pts).to(DEV), r, torch.from_numpy(t).to(camera_on).reshape(t_shape), *args).cpu().numpy()
        assert np.array_equal(got, want)
