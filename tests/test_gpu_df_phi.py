"""Phi and its partials at single points (csrc/df_phi.cuh) against extended
precision, for every hard-sphere kind: dilute to overdense, on both sides of the
series and of the limits beyond which a point takes the FP64 formulas.

Tolerances, relative to a partial's terms taken with their signs off.
Double-float: 2^-46 an operation chain, of which the closed forms just above
n3 = 1/32 and 1/16 cancel up to eight bits: 2^-38.  FP64 (points outside): the
same bits of 2^-53, and ln(1 - n3)'s argument is rounded: 2^-45 + 4 x 2^-53 / |n3|."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deft_gb300",
                    "csrc")
SOURCE = r"""
#include "df_phi.cuh"
using namespace deft;
__global__ void k(WbRadius r, DfPhiConst dk, double c, const double *x, double *out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  dfl w[5], d[5];
  for (int a = 0; a < 5; a++) w[a] = df_from(x[5 * i + a]);
  const dfl v2 = w[2] * w[2] + w[3] * w[3] + w[4] * w[4];
  double acc[6] = {0, 0, 0, 0, 0, 0};
  df_phi_point(r, dk, c, w, true, acc, d);
  double *o = out + 14 * i;
  for (int a = 0; a < 5; a++) o[a] = to_double(d[a]);
  o[5] = acc[0] * dk.s0;
  o[6] = acc[1] * dk.s1;
  o[7] = acc[2] * dk.s2;
  o[8] = df_point_ok(df_one_minus(w[0]), w[1], v2, true);
  for (int a = 0; a < 5; a++) o[9 + a] = to_double(w[a]);
}
extern "C" int run(int kind, double R, double c, const double *x, double *out, int n) {
  WbRadius r;
  wb_radius(r, R, kind);
  double *dx, *dy;
  if (cudaMalloc(&dx, 40 * n) || cudaMalloc(&dy, 112 * n)) return 1;
  cudaMemcpy(dx, x, 40 * n, cudaMemcpyHostToDevice);
  k<<<(n + 127) / 128, 128>>>(r, df_phi_const(r, c), c, dx, dy, n);
  const int rc = cudaMemcpy(out, dy, 112 * n, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dy);
  return rc;
}
"""
LD = np.longdouble


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("phi")
    (d / "t.cu").write_text(SOURCE)
    nvcc = "nvcc" if not os.path.exists("/usr/local/cuda/bin/nvcc") else "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", CSRC, "-shared", "-Xcompiler", "-fPIC",
                    str(d / "t.cu"), "-o", str(d / "t.so")], check=True)
    L = ctypes.CDLL(str(d / "t.so"))
    L.run.argtypes = [ctypes.c_int, ctypes.c_double, ctypes.c_double, ctypes.c_void_p,
                      ctypes.c_void_p, ctypes.c_int]
    return L


def _coeffs(kind, e):
    """f2, f2', f3, f3' of the kind, by series where the closed forms cancel."""
    pi = LD("3.14159265358979323846264338327950288")
    u, l = 1 / (1 - e), np.log1p(-e)
    small = np.abs(e) < LD(0.25)
    x, y = np.where(small, LD(0.5), e), np.where(small, e, LD(0))
    lx = np.log1p(-x)
    f2, df2 = u, u * u
    if kind == 1:
        return f2, df2, u * u / (24 * pi), 2 * u ** 3 / (24 * pi), l
    if kind == 0:
        S = (x + (1 - x) ** 2 * lx) / x ** 2
        dS = (x - 2 * (1 - x) * lx - 2 * (x + (1 - x) ** 2 * lx) / x) / x ** 2
        s, d = np.zeros_like(e), np.zeros_like(e)
        for j in range(70, 0, -1):
            c = LD(2) / (j * (j + 1) * (j + 2))
            s, d = (s + c) * y, d * y + j * c
        S, dS = np.where(small, LD(1.5) - s, S), np.where(small, -d, dS)
        k = 36 * pi
        return f2, df2, S * u * u / k, (dS + 2 * S * u) * u * u / k, l
    B = (1 - x) * lx / x
    dB = -(lx + 1) / x - (1 - x) * lx / x ** 2
    P2, dP2 = 1 + (6 - 3 * x + 6 * B) / 9, (-3 + 6 * dB) / 9
    N = 6 - 9 * x + 6 * x * x + 6 * (1 - x) * B
    dN = -9 + 12 * x + 6 * ((1 - x) * dB - B)
    P3, dP3 = 1 - N / (9 * x), -(dN / x - N / x ** 2) / 9
    A, D, C, G = (np.zeros_like(e) for _ in range(4))
    for k in range(80, 1, -1):
        A, D = A * y + LD(1) / (k * (k + 1)), D * y + LD(1) / (k + 1)
        if k > 2:
            C = C * y + LD(1) / ((k - 1) * k * (k + 1))
    P2 = np.where(small, 1 + LD(2) / 3 * y * y * A, P2)
    dP2 = np.where(small, LD(2) / 3 * y * D, dP2)
    P3 = np.where(small, 1 - LD(4) / 9 * y + LD(4) / 3 * y * y * C, P3)
    dP3 = np.where(small, LD(4) / 3 * A - LD(2) / 3, dP3)
    f3k = u * u / (24 * pi)
    return P2 * u, (dP2 + P2 * u) * u, P3 * f3k, (dP3 + 2 * P3 * u) * f3k, l


def _exact(kind, R, c, w):
    """The eight outputs and the sizes of their terms."""
    n3, n2, v = w[:, 0], w[:, 1], w[:, 2:]
    pi = LD("3.14159265358979323846264338327950288")
    a2 = 1 / (4 * pi * LD(R))
    a1 = a2 / LD(R)
    f2, df2, f3, df3, l = _coeffs(kind, n3)
    u = 1 / (1 - n3)
    v2 = (v * v).sum(1)
    q, qa = n2 * n2 - v2, n2 * n2 + v2
    t, ta = n2 * (n2 * n2 - 3 * v2), np.abs(n2) * (n2 * n2 + 3 * v2)
    ab = np.abs
    cv, ca = -2 * a2 * f2 - 6 * f3 * n2, 2 * a2 * ab(f2) + 6 * ab(f3 * n2)
    val = [c * (a1 * n2 * u + a2 * q * df2 + df3 * t), c * (-a1 * l + 2 * a2 * n2 * f2 + 3 * f3 * q),
           c * cv * v[:, 0], c * cv * v[:, 1], c * cv * v[:, 2], f3 * t, -a1 * n2 * l, a2 * q * f2]
    size = [c * (ab(a1 * n2 * u) + a2 * qa * ab(df2) + ab(df3) * ta),
            c * (ab(a1 * l) + 2 * a2 * ab(n2 * f2) + 3 * ab(f3) * qa), c * ca * ab(v[:, 0]),
            c * ca * ab(v[:, 1]), c * ca * ab(v[:, 2]), ab(f3) * ta, ab(a1 * n2 * l), a2 * qa * ab(f2)]
    return np.array(val), np.array(size)


def _points(R):
    rng = np.random.default_rng(7)
    inside = [np.exp(rng.uniform(np.log(1e-8), np.log(0.95), 20000)),
              rng.uniform(0.05, 0.6, 8000), -np.exp(rng.uniform(np.log(1e-8), np.log(9e5), 4000)),
              1 - 2.0 ** -rng.uniform(1, 19.9, 4000)]
    for t in (1 / 32, 1 / 16):  # the series' ends
        inside += [s * t * (1 + d) for s in (-1, 1) for d in (rng.uniform(-1e-3, 1e-3, 300),)]
        inside += [np.array([t, -t, np.nextafter(t, 0), np.nextafter(np.float32(t), 0)])]
    outside = [1 - 2.0 ** -rng.uniform(20.1, 30, 300), 1 - 2.0 ** rng.uniform(20.1, 24, 300),
               np.exp(rng.uniform(np.log(1e-14), np.log(2e-10), 300))]
    n3 = np.concatenate(inside + outside)
    n2 = 3 * np.abs(n3).clip(None, 1) / R * rng.uniform(0.5, 1.5, n3.size)
    v = rng.uniform(-0.57, 0.57, (n3.size, 3)) * n2[:, None]
    w = np.concatenate([n3[:, None], n2[:, None], v], 1)
    big = w[:200].copy()
    big[:, 0] = 0.3
    big[:, 1:] = big[:, 1:] / big[:, 1:2] * 2e9  # weighted densities beyond FP32's powers
    return np.concatenate([w, big])


@pytest.mark.parametrize("kind,R,c", [(0, 1.0, 0.008), (1, 0.8, 1.7e-3), (2, 2.87, 0.02)])
def test_points(lib, kind, R, c):
    x = np.ascontiguousarray(_points(R))
    out = np.empty((x.shape[0], 14))
    assert lib.run(kind, R, c, x.ctypes.data, out.ctypes.data, x.shape[0]) == 0
    ok, w = out[:, 8] != 0, out[:, 9:].astype(LD)
    val, size = _exact(kind, R, LD(c), w)
    err = (np.abs(out[:, :8].T - val) / size).astype(np.float64)
    n3 = np.abs(w[:, 0]).astype(np.float64)
    assert ok.sum() > 35000 and (~ok).sum() > 1000
    print(f"kind {kind}: double-float {err[:, ok].max() * 2 ** 46:.1f} x 2^-46 "
          f"(n3 {float(w[ok, 0][err[:, ok].max(0).argmax()]):.3g}), "
          f"dilute {err[:, ok & (n3 < 1e-4)].max() * 2 ** 46:.1f}, FP64 "
          f"{(err / (2.0 ** -45 + 4 * 2.0 ** -53 / n3))[:, ~ok].max():.2f} of its allowance")
    assert err[:, ok].max() <= 2.0 ** -38
    assert np.all(err[:, ~ok] <= 2.0 ** -45 + 4 * 2.0 ** -53 / n3[~ok])
