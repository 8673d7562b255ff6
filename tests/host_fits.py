"""The fit headers built for the host, so that single tracks can be fitted without a GPU."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = r"""
#include "bl_fit.cuh"
#include "riemann.cuh"
using namespace pxl;

template <int N, class T>
static int riemann(const double* hits, const float* ge, double B, double* out) {
  double h[3][N];
  float g[6][N];
  for (int i = 0; i < N; ++i) {
    for (int a = 0; a < 3; ++a) h[a][i] = hits[3 * i + a];
    for (int q = 0; q < 6; ++q) g[q][i] = ge[6 * i + q];
  }
  rm::RiemannOut o;
  const bool ok = rm::riemann_fit<N, T>(h, g, B, o);
  for (int k = 0; k < 5; ++k) out[k] = o.state[k];
  out[5] = o.chi2_circle; out[6] = o.chi2_line; out[7] = o.pt;
  return ok ? 0 : 1;
}

template <int N, class T>
static int broken_line(const double* hits, const float* ge, double B, double* out) {
  double h[3][N];
  float g[6][N];
  for (int i = 0; i < N; ++i) {
    for (int a = 0; a < 3; ++a) h[a][i] = hits[3 * i + a];
    for (int q = 0; q < 6; ++q) g[q][i] = ge[6 * i + q];
  }
  bl::TrackOut o;
  const bool ok = bl::fit_track<N, T>(h, g, B, o);
  for (int k = 0; k < 5; ++k) out[k] = o.state[k];
  out[5] = o.chi2_circle; out[6] = o.chi2_line; out[7] = o.pt;
  return ok ? 0 : 1;
}

#define BY_N(f, T) (n == 3 ? f<3, T>(hits, ge, B, out) : n == 4 ? f<4, T>(hits, ge, B, out) : f<8, T>(hits, ge, B, out))

extern "C" int fit(int which, int precision, int n, const double* hits, const float* ge, double B, double* out) {
  if (which == 0) return precision ? BY_N(broken_line, bl::f32) : BY_N(broken_line, double);
  return precision ? BY_N(riemann, bl::f32) : BY_N(riemann, double);
}
"""

_lib = None


def _build(directory: Path) -> ctypes.CDLL:
    """With contracted products, as the device code is built."""
    (directory / "host_fits.cu").write_text(SOURCE)
    so = directory / "host_fits.so"
    subprocess.run([NVCC, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler",
                    "-fPIC,-mfma,-ffp-contract=fast", "-I", str(ROOT / "cms-julia_b200" / "csrc"),
                    str(directory / "host_fits.cu"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.fit.argtypes = [ctypes.c_int] * 3 + [ctypes.c_void_p] * 2 + [ctypes.c_double, ctypes.c_void_p]
    return lib


def load(directory: Path):
    global _lib
    if _lib is None:
        _lib = _build(directory)
    return _lib


def fit(lib, which: str, precision: int, hits: np.ndarray, ge: np.ndarray, b_field: float) -> dict:
    """One track of 3, 4 or 8 hits (N, 3) float64 with covariances (N, 6) float32; which: "bl" or "rm"."""
    h, g, out = np.ascontiguousarray(hits, np.float64), np.ascontiguousarray(ge, np.float32), np.zeros(8)
    rc = lib.fit(int(which == "rm"), precision, len(h), h.ctypes.data, g.ctypes.data, b_field, out.ctypes.data)
    return {"status": rc, "state": out[:5], "chi2": out[5:7], "pt": out[7]}
