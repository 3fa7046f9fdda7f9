"""The correspondence search at the sizes and inputs where its path changes,
bit for bit against the CPU oracle: the largest radius that the merge scans
itself and the next, windows wider than a run of 128 columns and than a slab
of 768, ties everywhere (a plane seen head on: more runs than are kept), the
angle test, a cap inside the windows, and other units (the scale of the
half-precision products)."""
import dataclasses

import numpy as np
import pytest

from cudafusion_b200 import synth
from cudafusion_b200.corr import CorrespondenceSearch, CorrParams, DeviceCorrFrame

pytestmark = pytest.mark.gpu


def frame(w, h, kind, scale=1.0):
    f = synth.corr_frame(w, h, cam_rot_deg=0.8, noise=0.0 if kind == "smooth" else 0.001, seed=w + h)
    if kind == "plane":
        z = np.float32(0.5)
        fx, fy, cx, cy = f.cam
        u, v = np.meshgrid(np.arange(w), np.arange(h))
        ray = np.stack([(u - cx) / fx, (v - cy) / fy, np.ones_like(u)], -1).reshape(-1, 3)
        eye = np.eye(4, dtype=np.float32)
        n = np.tile(np.float32([0, 0, -1]), (w * h, 1))
        f = dataclasses.replace(f, depth=np.full(w * h, z, np.float32), depth_normals=n, live_normals=n.copy(),
                                live_vertices=(ray * 0.502).astype(np.float32), T_cam_world=eye, T_world_cam=eye.copy())
    if scale != 1.0:
        T, Ti = f.T_cam_world.copy(), f.T_world_cam.copy()
        T[:3, 3] *= scale
        Ti[:3, 3] *= scale
        s = np.float32(scale)
        f = dataclasses.replace(f, depth=f.depth * s, live_vertices=f.live_vertices * s, T_cam_world=T, T_world_cam=Ti)
    return f


CASES = [
    (96, 72, "noisy", 1.0, CorrParams(0.1, 0.0, 0.05, 8), 0),
    (96, 72, "noisy", 1.0, CorrParams(0.1, 0.0, 0.05, 9), 0),
    (97, 71, "smooth", 1.0, CorrParams(0.1, 0.0, 0.05, 25), 3),
    (210, 40, "noisy", 1.0, CorrParams(0.1, 0.0, 0.05, 70), 0),
    (840, 16, "noisy", 1.0, CorrParams(0.2, 0.0, 0.05, 400), 2),
    (840, 16, "noisy", 1.0, CorrParams(0.2, 0.3, 0.05, 400), 1),
    (80, 60, "plane", 1.0, CorrParams(0.05, 0.0, 0.05, 20), 2),
    (97, 71, "noisy", 1.0, CorrParams(0.1, 0.4, 0.1, 12), 0),
    (97, 71, "noisy", 1.0, CorrParams(0.004, 0.2, 0.1, 30), 0),
    (97, 71, "noisy", 1.0, CorrParams(0.004, 0.0, 0.0, 30), 0),
    (97, 71, "noisy", 1000.0, CorrParams(100.0, 0.0, 0.05, 12), 0),
    (97, 71, "noisy", 1e-3, CorrParams(0.03, 0.0, 0.05, 12), 0),
]


@pytest.mark.parametrize("w,h,kind,scale,prm,chunks", CASES)
def test_bit_exact(oracle, w, h, kind, scale, prm, chunks):
    f = frame(w, h, kind, scale)
    s = CorrespondenceSearch(w, h)
    s.set_chunks(chunks)
    n = s.find_correspondences(DeviceCorrFrame(f), prm, debug=True)
    recs, st = s.records(w * h), s.stats.cpu().numpy()
    ref, nv, rst = oracle.find_correspondences(f, prm.dist_threshold, prm.angle_threshold, prm.view_threshold,
                                               prm.search_radius_px)
    assert n == nv and np.array_equal(st, rst)
    assert np.array_equal(np.ascontiguousarray(recs).view(np.uint8), np.ascontiguousarray(ref).view(np.uint8))
