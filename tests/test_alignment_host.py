"""The connect kernel's bound of the alignment cut, as compiled from alignment.cuh: it passes every triple that the
cut passes, also where both sides round, vanish, overflow or are not numbers, and hardly any other."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from host_fits import NVCC

CSRC = Path(__file__).resolve().parents[1] / "cms-julia_b200" / "csrc"
SOURCE = """
#include "alignment.cuh"
using namespace pxl;
extern "C" void both(const float* a, long n, int barrel, unsigned char* cut, unsigned char* bound) {
  for (long i = 0; i < n; ++i) {
    const float* v = a + 6 * i;
    cut[i] = are_aligned(v[0], v[1], v[2], v[3], v[4], v[5], barrel ? kThetaBarrel : kThetaForward);
    bound[i] = maybe_aligned(v[0], v[1], v[2], v[3], v[4], v[5], barrel != 0);
  }
}
"""


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    d = tmp_path_factory.mktemp("alignment")
    (d / "a.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler",
                    "-fPIC,-ffp-contract=off", "-I", str(CSRC), str(d / "a.cu"), "-o", str(d / "a.so")], check=True)
    lib = ctypes.CDLL(str(d / "a.so"))
    lib.both.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]

    def f(a, barrel):
        a = np.ascontiguousarray(a, np.float32)
        cut, bound = np.zeros(len(a), np.uint8), np.zeros(len(a), np.uint8)
        lib.both(a.ctypes.data, len(a), int(barrel), cut.ctypes.data, bound.ctypes.data)
        return cut.astype(bool), bound.astype(bool)

    return f


@pytest.mark.parametrize("barrel", [True, False])
@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e-18, 1e12, 1e19])
def test_bound_passes_what_the_cut_passes(both, barrel, scale):
    rng = np.random.default_rng(11)
    n, theta = 1_000_000, 0.002 if barrel else 0.003
    r1, z1 = rng.uniform(2, 12, n), rng.uniform(-50, 50, n)
    ri, ro = r1 + rng.uniform(0, 8, n), r1 + rng.uniform(0, 16, n)
    slope = rng.uniform(-5, 5, n)
    zi = z1 + slope * (ri - r1)
    rd, dz = np.abs(ro - r1), slope * (ro - r1)
    # zo off the line by about the cut's limit (some rounding errors to either side), or by anything, or not
    off = theta / 0.9 * np.hypot(rd, dz) * rd / np.maximum(np.abs(ri - r1), 1e-3)
    kind = rng.integers(0, 3, n)
    off *= np.where(kind == 0, 1 + rng.normal(0, 1e-6, n), np.where(kind == 1, rng.uniform(0, 3, n), 0.0))
    a = np.stack([r1, z1, ri, zi, ro, z1 + dz + off * rng.choice([-1, 1], n)], 1) * scale
    a[:1000, 4] = a[:1000, 0]  # equal radii, equal points, and values that are no numbers
    a[:500, 5] = a[:500, 1]
    for k, v in enumerate((np.inf, -np.inf, np.nan)):
        a[1000 + 600 * k:1600 + 600 * k, :][np.arange(600), np.arange(600) % 6] = v
    cut, bound = both(a, barrel)
    assert not (cut & ~bound).any()
    if scale == 1.0:
        assert cut.sum() > n // 4 and (bound & ~cut).sum() < n // 4
        line = (kind == 2) & np.isfinite(a).all(1)  # the cut fails on what is no number, the bound leaves it to the cut
        assert (bound[line] == cut[line]).mean() > 0.999
