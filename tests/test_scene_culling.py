"""The F1 scene's distance with parts left out where they cannot matter (the device
code built for the host) against the oracle's full evaluation, bit for bit: every
variant of every part, ride heights and wing angles beyond the usual range, points
inside the car, around it, far away, and points that are not finite."""
import ctypes

import numpy as np
import pytest

from helpers import shade_host_model
from test_scene_sdf import device_sdf, oracle_sdf


@pytest.fixture(scope="module")
def hm():
    L = shade_host_model()
    if L is None:
        pytest.skip("the CUDA headers are missing")
    return L


def scene_points(rng, b, n):
    lo, hi = np.array([-0.3, -0.1 + b, -1.0]), np.array([5.7, 1.1 + b, 1.0])
    near = rng.uniform(lo, hi, (n, 3))
    around = rng.uniform([-4, -2, -4], [10, 5, 4], (n, 3))
    far = rng.normal(size=(n // 2, 3)) * 10.0 ** rng.uniform(0, 7, (n // 2, 1))
    axes = near[: n // 2].copy()
    axes[:, 2] = rng.choice([0.0, -0.0, 0.17, 0.25, 0.5], len(axes))
    odd = near[: n // 8].copy()
    odd[np.arange(len(odd)), rng.integers(0, 3, len(odd))] = rng.choice([np.nan, np.inf, -np.inf, 1e20, -1e38], len(odd))
    return np.concatenate([near, around, far, axes, odd]).astype(np.float32)


@pytest.mark.parametrize("seed", range(8))
def test_culled_distance_bitexact(hm, oracle_mod, seed):
    from windtunnel import _abi
    rng = np.random.default_rng(seed)
    for k in range(12):
        s = _abi.Shape()
        s.kind = 0
        usual = k % 3 != 0
        s.ride_h = rng.uniform(0.02, 0.12) if usual else rng.uniform(-0.6, 1.2)
        s.rear_ride = s.ride_h + (rng.uniform(-0.02, 0.1) if usual else rng.uniform(-0.5, 0.5))
        w = 1.0 if usual else 4.0
        s.front_flap, s.rear_main, s.rear_flap = (rng.uniform(-0.2, 0.7, 3) * w).tolist()
        s.front_wing, s.rear_wing, s.sidepod, s.cover, s.nose = rng.integers(0, 4, 5).astype(float).tolist()
        pts = scene_points(rng, float(s.ride_h), 12000)
        # and points a few steps along the distance, where a march ends: near the surfaces
        d = oracle_sdf(oracle_mod, s, pts)[:, 0]
        g = rng.normal(size=(len(pts), 3)).astype(np.float32)
        g /= np.linalg.norm(g, axis=1, keepdims=True)
        with np.errstate(all="ignore"):
            pts = np.concatenate([pts, (pts + g * d[:, None]).astype(np.float32)])
        got, ref = device_sdf(hm, s, pts), oracle_sdf(oracle_mod, s, pts)
        same = (got.view(np.uint32) == ref.view(np.uint32)) | (np.isnan(got) & np.isnan(ref))
        bad = np.nonzero(~same.all(1))[0]
        assert len(bad) == 0, (k, len(bad), pts[bad[:3]].tolist(), got[bad[:3]].tolist(), ref[bad[:3]].tolist())
