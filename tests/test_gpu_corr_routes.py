"""The search's routes on frames large enough for all of them, bit for bit
against the CPU oracle at sampled pixels: the tensor-core search alone, the exact
scan alone (an angle threshold, a cap inside the windows), and chunks that the
search leaves to the exact scan (planes, with whole frames, single tiles or a
few pixels of equal distances); windows wider than a run and a slab, one chunk
of rows and eight, other units."""
import dataclasses

import numpy as np
import pytest

from cudafusion_b200 import synth
from cudafusion_b200.corr import CorrespondenceSearch, CorrParams, DeviceCorrFrame

pytestmark = pytest.mark.gpu


def rays(f):
    fx, fy, cx, cy = f.cam
    u, v = np.meshgrid(np.arange(f.width), np.arange(f.height))
    return np.stack([(u - cx) / fx, (v - cy) / fy, np.ones(u.shape)], -1).reshape(-1, 3), u.reshape(-1), v.reshape(-1)


def surface(f, z, normal, where=None):
    """f with depth z (per pixel) seen along `normal`, and live points 2 mm behind it."""
    ray, _, _ = rays(f)
    where = np.ones(f.num_pixels, bool) if where is None else where
    d, dn, lv, ln = f.depth.copy(), f.depth_normals.copy(), f.live_vertices.copy(), f.live_normals.copy()
    d[where] = z[where].astype(np.float32)
    dn[where] = ln[where] = np.asarray(normal, np.float32) / np.float32(np.linalg.norm(normal))
    lv[where] = (ray * (z + 0.002)[:, None])[where].astype(np.float32)
    eye = np.eye(4, dtype=np.float32)
    return dataclasses.replace(f, depth=d, depth_normals=dn, live_vertices=lv, live_normals=ln, T_cam_world=eye,
                               T_world_cam=eye.copy())


@pytest.fixture(scope="module")
def frames():
    made = {}

    def get(w, h, kind, scale):
        noise = 0.0 if kind == "smooth" else 0.001
        if (w, h, noise) not in made:
            made[w, h, noise] = synth.corr_frame(w, h, noise=noise, seed=w + h, num_nodes=64)
        f = made[w, h, noise]
        ray, u, v = rays(f)
        if kind == "plane":
            f = surface(f, np.full(f.num_pixels, 0.5), (0, 0, -1))
        elif kind == "tilted":
            f = surface(f, 0.5 / (1.0 + 0.2 * ray[:, 0] + 0.1 * ray[:, 1]), (-0.2, -0.1, -1))
        elif kind == "half":  # a plane on the right, the noisy cylinders on the left
            f = surface(f, np.full(f.num_pixels, 0.14), (0, 0, -1), u >= w // 2 + 5)
        elif kind == "patches":  # few pixels of equal distances in each tile
            f = surface(f, np.full(f.num_pixels, 0.14), (0, 0, -1), (u % 32 < 5) & (v % 16 < 5))
        if scale != 1.0:
            T, Ti = f.T_cam_world.copy(), f.T_world_cam.copy()
            T[:3, 3] *= scale
            Ti[:3, 3] *= scale
            s = np.float32(scale)
            f = dataclasses.replace(f, depth=f.depth * s, live_vertices=f.live_vertices * s, T_cam_world=T,
                                    T_world_cam=Ti)
        return f

    return get


CASES = [
    (640, 480, "noisy", 1.0, CorrParams(0.2, 0.0, 0.0, 50), 0),
    (640, 480, "noisy", 1.0, CorrParams(0.2, 0.0, 0.0, 40), 8),
    (640, 480, "noisy", 1.0, CorrParams(0.2, 0.3, 0.0, 30), 0),
    (640, 480, "noisy", 1.0, CorrParams(0.004, 0.0, 0.0, 50), 0),
    (640, 480, "noisy", 1000.0, CorrParams(200.0, 0.0, 0.0, 36), 0),
    (640, 480, "noisy", 1e-3, CorrParams(0.03, 0.0, 0.0, 36), 0),
    (640, 480, "smooth", 1.0, CorrParams(0.2, 0.0, 0.0, 50), 0),
    (640, 480, "smooth", 1.0, CorrParams(0.2, 0.0, 0.0, 20), 0),
    (640, 480, "plane", 1.0, CorrParams(0.2, 0.0, 0.0, 50), 0),
    (640, 480, "plane", 1.0, CorrParams(0.2, 0.0, 0.0, 36), 1),
    (640, 480, "plane", 1.0, CorrParams(0.2, 0.3, 0.0, 20), 0),
    (640, 480, "tilted", 1.0, CorrParams(0.2, 0.0, 0.0, 36), 0),
    (640, 480, "half", 1.0, CorrParams(0.2, 0.0, 0.0, 50), 3),
    (640, 480, "patches", 1.0, CorrParams(0.2, 0.0, 0.0, 40), 0),
    (1201, 49, "noisy", 1.0, CorrParams(0.2, 0.0, 0.0, 400), 0),
    (1201, 49, "plane", 1.0, CorrParams(0.2, 0.0, 0.0, 390), 2),
    (1201, 49, "noisy", 1.0, CorrParams(0.2, 0.3, 0.0, 400), 3),
    # the last radius that the merge scans itself and the next, without and with an angle threshold
    (97, 71, "noisy", 1.0, CorrParams(0.2, 0.0, 0.0, 7), 0),
    (97, 71, "plane", 1.0, CorrParams(0.2, 0.0, 0.0, 8), 0),
    (97, 71, "plane", 1.0, CorrParams(0.2, 0.3, 0.0, 8), 0),
    (97, 71, "noisy", 1.0, CorrParams(0.2, 0.3, 0.0, 9), 0),
    # frames whose merge has at most two CTAs per SM and one that has more
    (320, 236, "noisy", 1.0, CorrParams(0.2, 0.0, 0.0, 20), 0),
    (320, 240, "tilted", 1.0, CorrParams(0.2, 0.0, 0.0, 20), 0),
]


@pytest.mark.parametrize("w,h,kind,scale,prm,chunks", CASES)
def test_bit_exact(oracle, frames, w, h, kind, scale, prm, chunks):
    f = frames(w, h, kind, scale)
    s = CorrespondenceSearch(w, h)
    s.set_chunks(chunks)
    s.find_correspondences(DeviceCorrFrame(f), prm)
    recs = s.records(w * h)
    side = min(2 * prm.search_radius_px + 1, w) * min(2 * prm.search_radius_px + 1, h)
    pix = np.sort(np.random.default_rng(w + prm.search_radius_px).choice(w * h, min(w * h, 2 * 10**7 // side), replace=False))
    ref, _, _ = oracle.find_correspondences(f, prm.dist_threshold, prm.angle_threshold, prm.view_threshold,
                                            prm.search_radius_px, pixels=pix.astype(np.int32))
    assert ref["valid"].any()
    assert np.array_equal(np.ascontiguousarray(recs[pix]).view(np.uint8), np.ascontiguousarray(ref).view(np.uint8))
