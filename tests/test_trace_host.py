"""What the traces decide by, on the CPU.  A record that a ray hits nearer than its best
passes the culls, and a pooled head names its view.

Relief moves a tall stone or brick box's hit toward the camera by up to 0.0025 m
per unit of the face's slant, which goes down to 0.08: 0.031 m along a grazing ray,
while the box's entry by its other axis, across which the ray runs steeply, stays
where it is.  The rays here enter such a face within millimetres of its near edge."""
import ctypes as ct
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "stratum_hyperdetail_b200" / "csrc"
GEN = ROOT / "stratum_hyperdetail_b200" / "_build" / "gen"
f32p = np.ctypeslib.ndpointer(np.float32, flags="C_CONTIGUOUS")
i32p = np.ctypeslib.ndpointer(np.int32, flags="C_CONTIGUOUS")


@pytest.fixture(scope="module")
def ht(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    if not (GEN / "trig_table.h").exists():
        from stratum_hyperdetail_b200 import build
        build.gen_tables()
    out = tmp_path_factory.mktemp("ht") / "libht.so"
    subprocess.run([nvcc, "-x", "cu", "-std=c++17", "-O2", "-shared", "--fmad=false", "-Xcompiler", "-fPIC", "-Xcompiler",
                    "-ffp-contract=off", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), "-I", str(GEN),
                    "-I", str(ROOT / "include"), str(ROOT / "tests" / "host_trace.cu"), "-o", str(out)], check=True)
    lib = ct.CDLL(str(out))
    lib.ht_culls.argtypes = [f32p, f32p, ct.c_int, ct.c_float, f32p, i32p]
    lib.ht_relief.argtypes = [f32p, f32p, f32p, f32p, ct.c_int, f32p, f32p]
    lib.ht_heads.argtypes = [i32p, ct.c_int]
    return lib


@pytest.mark.parametrize("steep,along", [(0, 2), (2, 0)])
@pytest.mark.parametrize("far", [0.5, 20.0])
def test_grazed_relief_passes_the_culls(ht, steep, along, far):
    n = 400000
    rng = np.random.default_rng(steep * 2 + int(far))
    half = np.stack([rng.uniform(0.15, 9, n), rng.uniform(1.05, 9, n), rng.uniform(0.15, 9, n)], 1)
    centre = rng.uniform(-12, 12, (n, 3))
    boxes = np.concatenate([centre, half, rng.integers(0, 2, (n, 1))], 1).astype(np.float32)
    b = boxes.astype(np.float64)
    # a unit direction that slants 0.0801..0.1 into the face across axis `steep`
    d = np.zeros((n, 3))
    d[:, steep] = -rng.uniform(0.0801, 0.1, n)
    d[:, 1] = rng.uniform(-0.2, 0.2, n)
    d[:, along] = np.sqrt(1 - d[:, steep]**2 - d[:, 1]**2)
    hit = b[:, :3].copy()  # on the face, 0..6 mm along from its near edge
    hit[:, steep] += b[:, 3 + steep]
    hit[:, along] += -b[:, 3 + along] + rng.uniform(0.0, 0.006, n)
    hit[:, 1] += rng.uniform(-0.9, 0.9, n) * b[:, 4]
    rays = np.concatenate([hit - d * rng.uniform(0.2, far, (n, 1)), d], 1).astype(np.float32)
    t, kept = np.zeros(n, np.float32), np.zeros(n, np.int32)
    ht.ht_culls(boxes, rays, n, ct.c_float(1e-4), t, kept)
    hits = t < 2000
    assert hits.sum() > n // 2
    for bit, name in ((1, "packet"), (2, "ray")):
        lost = hits & ((kept & bit) == 0)
        assert not lost.any(), (name, int(lost.sum()), boxes[lost][0], rays[lost][0], t[lost][0])


def test_pooled_heads_of_every_view(ht):
    """4,095 views are the most that the pooled trace takes."""
    heads = np.array([(v, s, g) for v in (0, 1, 2047, 2048, 4093, 4094) for s in (0, 1, 8191, 16383)
                      for g in (0, 31, 63)], np.int32)
    assert ht.ht_heads(np.ascontiguousarray(heads), len(heads)) == len(heads)


@pytest.mark.parametrize("value", [None, float("nan"), float("inf"), -float("inf"), 1e38])
def test_relief_leaves_out_only_steps_that_come_to_nothing(ht, value):
    """Footprints on both sides of the cut-off, and rays that are not finite: a distance
    that is no number (a miss) stays none."""
    n = 100000
    rng = np.random.default_rng(11)
    half = rng.uniform(1.05, 9, (n, 3))
    boxes = np.concatenate([rng.uniform(-12, 12, (n, 3)), half, rng.integers(0, 2, (n, 1))], 1).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    start = rng.uniform(0.1, 300.0, n)
    face = boxes[:, :3] + np.where(rng.random((n, 3)) < 0.5, -1, 1) * half * rng.choice([1.0, 0.3], (n, 3))
    rays = np.concatenate([face - d * start[:, None], d], 1)
    if value is not None:
        rays[np.arange(n), rng.integers(0, 6, n)] = value
    rays, start = rays.astype(np.float32), start.astype(np.float32)
    cone = np.where(rng.random(n) < 0.5, 0.0275 / start * rng.uniform(0.5, 1.5, n), 0.01).astype(np.float32)
    t, whole = np.zeros(n, np.float32), np.zeros(n, np.float32)
    ht.ht_relief(boxes, rays, start, cone, n, t, whole)
    assert np.array_equal(t, whole, equal_nan=True)
    assert (whole != start).sum() > 1000
