"""The logarithms, reciprocal and square root of csrc/logtab.cuh and the
conversions of csrc/dfloat.cuh, one by one, against extended precision: at the
table's interval edges, next to 1 and at the limits of their ranges.

Tolerances.  log_tab adds k ln 2, ln c and log1p r, each rounded to 2^-54 of
itself, and the sum may be half the size of its terms: 4 x 2^-53.  The
reciprocal's and square root's last step leaves its own rounding and that of
its correction: 2^-52.  df_log1m is double-float, some ten operations of 2^-47:
2^-45."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deft_gb300",
                    "csrc")
SOURCE = r"""
#include "logtab.cuh"
using namespace deft;
__global__ void k(int which, const double *x, double *out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v = x[i];
  double r = 0;
  if (which == 0) r = log_tab(v);
  if (which == 1) r = rcp_fast(v);
  if (which == 2) r = sqrt_fast(v);
  if (which == 3) {  // 1 - e with e's own digits, as Phi's kernel forms it
    const dfl e = df_from(v);
    const dfl t = df_two_sum(1.0f, -e.hi);
    r = to_double(df_log1m(e, df_fast_two_sum(t.hi, t.lo - e.lo)));
  }
  if (which == 4) r = to_double(df_from(v));
  if (which == 5) r = f2d(d2f_small(v));
  if (which == 6) r = to_double(df_rcp(df_from(v)));
  out[i] = r;
}
extern "C" int run(int which, const double *x, double *out, int n) {
  double *dx, *dy;
  if (cudaMalloc(&dx, 8 * n) || cudaMalloc(&dy, 8 * n)) return 1;
  cudaMemcpy(dx, x, 8 * n, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(which, dx, dy, n);
  const int rc = cudaMemcpy(out, dy, 8 * n, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dy);
  return rc;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("logtab")
    (d / "t.cu").write_text(SOURCE)
    nvcc = "nvcc" if not os.path.exists("/usr/local/cuda/bin/nvcc") else "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", CSRC, "-shared", "-Xcompiler", "-fPIC",
                    str(d / "t.cu"), "-o", str(d / "t.so")], check=True)
    L = ctypes.CDLL(str(d / "t.so"))

    def call(which, x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        out = np.empty_like(x)
        assert L.run(which, ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(out.ctypes.data),
                     x.size) == 0
        return out

    return call


def _positive(lo, hi):
    """Values over the binades 2^lo .. 2^hi, every table edge of one and neighbours, next to 1."""
    rng = np.random.default_rng(1)
    wide = np.ldexp(rng.uniform(1, 2, 40000), rng.integers(lo, hi, 40000))
    edges = 0.75 + np.arange(129) / 128 * 0.75
    edges = np.concatenate([edges, np.float32(edges), 0.75 + np.arange(257) * 2.0 ** -8])
    edges = np.concatenate([edges, np.nextafter(edges, 0), np.nextafter(edges, 9)])
    near = np.concatenate([1 + s * 2.0 ** -rng.uniform(1, 52, 20000) for s in (-1, 1)])
    x = np.concatenate([wide, edges, near, np.ldexp(edges, 5), np.ldexp(edges, -9)])
    return x[(x >= 2.0 ** lo) & (x < 2.0 ** hi)]


def _worst(got, want):
    """Largest error relative to the exact value, which is long double."""
    want = np.asarray(want)
    d = np.abs(got.astype(np.longdouble) - want)
    ok = want != 0
    assert np.all(got[~ok] == 0)
    return float((d[ok] / np.abs(want[ok])).max())


def test_log(run):
    assert np.finfo(np.longdouble).eps < 2.0 ** -60
    x = _positive(-1021, 1023)
    err = _worst(run(0, x), np.log(x.astype(np.longdouble)))
    near = x[(x > 1) & (x < 1 + 2.0 ** -6)]
    print(f"log_tab: {err * 2 ** 53:.2f} x 2^-53, just above 1 "
          f"{_worst(run(0, near), np.log(near.astype(np.longdouble))) * 2 ** 53:.2f}")
    assert err <= 4 * 2.0 ** -53
    s = np.array([0.0, -0.0, np.inf, np.nan, -1.0, -np.inf, 5e-324, 2.0 ** -1030, 1.0])
    with np.errstate(divide="ignore"):
        got, want = run(0, s), np.log(np.abs(s))
    assert np.isneginf(got[0]) and np.isneginf(got[1]) and np.isposinf(got[2])
    assert np.all(np.isnan(got[3:6])) and got[8] == 0
    assert np.all(np.abs(got[6:8] / want[6:8] - 1) <= 4 * 2.0 ** -53)


def test_reciprocal_and_root(run):
    x = np.concatenate([_positive(-300, 300), 2.0 ** np.array([-75.0, -74, -73, 105, 106, 107, 127])])
    xl = x.astype(np.longdouble)
    signed = np.concatenate([x, -x])
    e1, e2 = _worst(run(1, signed), 1 / signed.astype(np.longdouble)), _worst(run(2, x), np.sqrt(xl))
    print(f"rcp_fast {e1 * 2 ** 53:.2f} x 2^-53, sqrt_fast {e2 * 2 ** 53:.2f}")
    assert e1 <= 2.0 ** -52 and e2 <= 2.0 ** -52
    s = np.array([0.0, -0.0, np.inf, -np.inf, np.nan])
    assert np.array_equal(run(1, s), [np.inf, -np.inf, 0, -0.0, np.nan], equal_nan=True)
    assert np.array_equal(run(2, np.array([0.0, np.inf, -1.0, np.nan])), [0, np.inf, np.nan, np.nan],
                          equal_nan=True)


def test_log1m(run):
    rng = np.random.default_rng(2)
    tiny = np.concatenate([s * 2.0 ** -rng.uniform(1, 60, 20000) for s in (-1, 1)])
    e = np.concatenate([tiny, 1 - _positive(-19, 19), rng.uniform(-0.5, 0.5, 20000)])
    e = run(4, e)  # double-floats
    e = e[(1 - e > 2.0 ** -19) & (e != 0)]
    err = _worst(run(3, e), np.log1p(-e.astype(np.longdouble)))
    print(f"df_log1m: {err * 2 ** 46:.2f} x 2^-46")
    assert err <= 2.0 ** -45
    assert run(3, np.zeros(1))[0] == 0


def test_conversions(run):
    rng = np.random.default_rng(3)
    x = np.ldexp(rng.uniform(1, 2, 100000), rng.integers(-74, 126, 100000))
    x = np.concatenate([x, -x, np.float64(np.float32(x))])
    assert _worst(run(4, x), x.astype(np.longdouble)) <= 2.0 ** -48
    assert _worst(run(5, x), x.astype(np.longdouble)) <= 2.0 ** -24
    f = np.float64(np.float32(np.ldexp(rng.uniform(1, 2, 10000), rng.integers(-149, 127, 10000))))
    f = np.concatenate([f, [0.0, -0.0, np.inf, -np.inf, np.nan]])
    assert np.array_equal(run(5, f), f, equal_nan=True)
    r = x[(np.abs(x) < 2.0 ** 60) & (np.abs(x) > 2.0 ** -60)]
    d = run(4, r)
    err = _worst(run(6, r), 1 / d.astype(np.longdouble))
    print(f"df_rcp: {err * 2 ** 46:.2f} x 2^-46")
    assert err <= 2.0 ** -45
