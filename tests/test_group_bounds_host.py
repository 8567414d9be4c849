"""Group bounds from the features that attain them equal the whole grammar's
(CPU only): every lot family and floor count over the dimensions a described
lot has, their extremes included, bit for bit; other rows are not `regular`."""
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
def hb(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    if not (GEN / "trig_table.h").exists():
        from stratum_hyperdetail_b200 import build
        build.gen_tables()
    out = tmp_path_factory.mktemp("hb") / "libhb.so"
    subprocess.run([nvcc, "-x", "cu", "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC", "-Xcompiler",
                    "-ffp-contract=off", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), "-I", str(GEN),
                    str(ROOT / "tests" / "host_bounds.cu"), "-o", str(out)], check=True)
    lib = ct.CDLL(str(out))
    lib.hb_regular.argtypes = [f32p]
    lib.hb_differ.argtypes = [f32p, ct.c_int, i32p]
    return lib


def rows(oracle, n, seed):
    """Described lots, then the same with every family and floor count and with
    dimensions at the ends of their ranges."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        tag = rng.integers(0, 2**32, 4, dtype=np.uint64).astype(np.uint32)
        lot = np.zeros(16, np.float32)
        d = oracle.describe_lot(tag, int(rng.integers(0, 1 << 24)))
        lot[:len(d)] = d
        out.append(lot.copy())
        ty = int(rng.integers(0, 6))
        lot[3], lot[5] = ty, 6 if ty == 2 else int(rng.integers(2, 7))
        ends = rng.random(5) < 0.4
        for k, (lo, hi) in ((0, (9.4, 13.69993)), (1, (9.0, 13.69993)), (7, (3.2, 4.34998)), (8, (0.85, 1.24999))):
            if ends[k % 5]:
                lot[k] = lo if rng.random() < 0.5 else hi
        lot[2] = np.float32(4.2) + np.float32(lot[5]) * np.float32(lot[7])
        out.append(lot)
    return np.ascontiguousarray(np.stack(out), np.float32)


def test_regular_rows_have_the_whole_grammars_bounds(hb, oracle):
    lots = rows(oracle, 20000, 3)
    assert all(hb.hb_regular(np.ascontiguousarray(r)) for r in lots)
    where = np.zeros(192, np.int32)
    bad = hb.hb_differ(lots, len(lots), where)
    assert bad == 0, (bad, where[:30].reshape(-1, 3), lots[where[0]])


@pytest.mark.parametrize("word,value", [(0, 5.0), (0, 20.0), (1, 8.0), (2, 3.0), (3, 7.0), (5, 1.0), (5, 9.0),
                                        (7, 2.0), (8, 0.5), (0, float("nan")), (2, float("inf"))])
def test_other_rows_go_through_the_whole_grammar(hb, oracle, word, value):
    lots = rows(oracle, 4, 5)
    for r in lots:
        r = r.copy()
        r[word] = value
        assert not hb.hb_regular(r)
        assert hb.hb_differ(r, 1, np.zeros(192, np.int32)) == 0
