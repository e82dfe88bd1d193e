"""recip and root of the flux functions, and Roe's flux, on values that no sound
state has: a root is what the square root gives, a reciprocal without a value is
not finite, so that a run which went wrong is still reported."""
import os
import subprocess

import numpy as np
import pytest

import flurrypp_b200 as fb
from conftest import ROOT
from flurrypp_b200.decks import write_deck

pytestmark = pytest.mark.gpu

SOURCE = r'''
#include <cmath>
#include <cstdio>
#include "fr_physics.cuh"
__global__ void k(const double *x, int n, double *out, const double *st, int m, double *flux, float *rest) {
  for (int i = 0; i < n; i++) {
    out[4 * i] = frk::recip(x[i]);
    out[4 * i + 1] = frk::root(x[i]);
    out[4 * i + 2] = frk::recip((float)x[i]);
    out[4 * i + 3] = frk::root((float)x[i]);
  }
  const double nrm[2] = {0.6, 0.8};
  for (int i = 0; i < m; i++) frk::roe2d<double>(st + 8 * i, st + 8 * i + 4, nrm, 1.4, flux + 4 * i);
  const float a[4] = {1, 1e-40f, 0, 2.5f}, b[4] = {1, -2e-40f, 0, 2.5f}, nf[2] = {0.6f, 0.8f};
  frk::roe2d<float>(a, b, nf, 1.4f, rest);
}
// Roe's flux with plain divisions and square roots
static void roe(const double *UL, const double *UR, const double *n, double g, double *F) {
  double vL[2], vR[2], um[2], du[4], usq = 0, unm = 0, qL = 0, qR = 0;
  for (int i = 0; i < 2; i++) vL[i] = UL[i + 1] / UL[0], vR[i] = UR[i + 1] / UR[0];
  const double pL = (g - 1) * (UL[3] - 0.5 * UL[0] * (vL[0] * vL[0] + vL[1] * vL[1]));
  const double pR = (g - 1) * (UR[3] - 0.5 * UR[0] * (vR[0] * vR[0] + vR[1] * vR[1]));
  const double hL = (UL[3] + pL) / UL[0], hR = (UR[3] + pR) / UR[0], sq = sqrt(UR[0] / UL[0]), rr = 1 / (sq + 1);
  for (int i = 0; i < 2; i++) {
    um[i] = rr * (vL[i] + sq * vR[i]);
    usq += 0.5 * um[i] * um[i];
    unm += um[i] * n[i];
    qL += UL[i + 1] * n[i];
    qR += UR[i + 1] * n[i];
  }
  const double hm = rr * (hL + sq * hR), am2 = (g - 1) * (hm - usq), am = sqrt(am2);
  for (int i = 0; i < 4; i++) du[i] = UR[i] - UL[i];
  double l0 = fabs(unm), lP = fabs(unm + am), lM = fabs(unm - am);
  const double eps = 0.5 * (fabs(qL / UL[0] - qR / UR[0]) + fabs(sqrt(g * pL / UL[0]) - sqrt(g * pR / UR[0])));
  if (l0 < 2 * eps) l0 = 0.25 * l0 * l0 / eps + eps;
  if (lP < 2 * eps) lP = 0.25 * lP * lP / eps + eps;
  if (lM < 2 * eps) lM = 0.25 * lM * lM / eps + eps;
  const double a2 = 0.5 * (lP + lM) - l0, a3 = 0.5 * (lP - lM) / am, a1 = a2 * (g - 1) / am2, a4 = a3 * (g - 1);
  const double a5 = usq * du[0] - um[0] * du[1] - um[1] * du[2] + du[3];
  const double a6 = unm * du[0] - n[0] * du[1] - n[1] * du[2], aL1 = a1 * a5 - a3 * a6, bL1 = a4 * a5 - a2 * a6;
  F[0] = 0.5 * (qL + qR) - 0.5 * (l0 * du[0] + aL1);
  for (int i = 0; i < 2; i++)
    F[i + 1] = 0.5 * (UL[i + 1] * qL / UL[0] + UR[i + 1] * qR / UR[0] + (pL + pR) * n[i]) -
               0.5 * (l0 * du[i + 1] + aL1 * um[i] + bL1 * n[i]);
  F[3] = 0.5 * (hL * qL + hR * qR) - 0.5 * (l0 * du[3] + aL1 * hm + bL1 * unm);
}
int main() {
  const double inf = INFINITY;
  const double x[] = {0.0, -0.0, 1.0, 2.0, -3.0, inf, -inf, NAN, 1e-300, -1e-300};
  // sound states; negative pressure left; negative density right, left
  const double st[] = {1, 0.2, 0.1, 2.0, 0.9, 0.5, -0.1, 2.2,  1, 0.9, 0.1, 0.2, 0.9, 0.95, -0.1, 2.2,
                       1, 0.2, 0.1, 2.0, -0.9, 0.5, -0.1, 2.2, -1, 0.2, 0.1, 2.0, 0.9, 0.5, -0.1, 2.2,
                       // at rest but for a subnormal velocity, which the entropy fix scales by
                       1, 1e-310, 0, 2.5, 1, -2e-310, 0, 2.5};
  const int n = sizeof x / 8, m = sizeof st / 64;
  double *dx, *dout, *ds, *df, out[4 * n], f[4 * m], r[4];
  float *dr, rest[4];
  cudaMalloc(&dx, sizeof x), cudaMalloc(&dout, sizeof out), cudaMalloc(&ds, sizeof st), cudaMalloc(&df, sizeof f), cudaMalloc(&dr, 16);
  cudaMemcpy(dx, x, sizeof x, cudaMemcpyHostToDevice), cudaMemcpy(ds, st, sizeof st, cudaMemcpyHostToDevice);
  k<<<1, 1>>>(dx, n, dout, ds, m, df, dr);
  cudaMemcpy(out, dout, sizeof out, cudaMemcpyDeviceToHost), cudaMemcpy(f, df, sizeof f, cudaMemcpyDeviceToHost);
  cudaMemcpy(rest, dr, 16, cudaMemcpyDeviceToHost);
  int bad = 0;
  for (int q = 0; q < 4; q++)  // the pressure alone
    if (!(fabs(rest[q] - (q == 1 ? 0.6 : q == 2 ? 0.8 : 0.0)) < 1e-6)) printf("at rest %d got %g\n", q, rest[q]), bad++;
  const auto same = [](double a, double b) { return a == b || (a != a && b != b); };
  for (int i = 0; i < n; i++) {
    const bool tiny = x[i] != 0 && fabs(x[i]) < 1e-200;  // a root that small gives its argument back; FP32: zero
    const float xf = (float)x[i];
    const double want[4] = {1 / x[i], tiny && x[i] > 0 ? x[i] : sqrt(x[i]), 1 / xf, sqrtf(xf)};
    for (int q = 0; q < 4; q++)
      if (q % 2 == 0 && (x[i] == 0 || x[i] != x[i] || fabs(x[i]) == inf || (tiny && q == 2)))  // a reciprocal there: not finite
        bad += std::isfinite(out[4 * i + q]);
      else if (!same(out[4 * i + q], want[q]) && !(tiny && q == 0)) printf("x %g op %d got %g want %g\n", x[i], q, out[4 * i + q], want[q]), bad++;
  }
  const double nrm[2] = {0.6, 0.8};
  for (int i = 0; i < m; i++) {
    roe(st + 8 * i, st + 8 * i + 4, nrm, 1.4, r);
    for (int q = 0; q < 4; q++) {
      const bool nan = r[q] != r[q];
      if (nan != (f[4 * i + q] != f[4 * i + q]) || (!nan && fabs(f[4 * i + q] - r[q]) > 1e-14 * (1 + fabs(r[q]))))
        printf("flux %d.%d got %g want %g\n", i, q, f[4 * i + q], r[q]), bad++;
    }
  }
  return bad || cudaGetLastError() != cudaSuccess;
}
'''


def test_special_values(tmp_path):
    """About 60 roundings of terms below 4 in a flux: 60 * 2^-53 * 4 = 3e-14 at most, 1e-14 of 1 + |F| allowed."""
    src = tmp_path / "t.cu"
    src.write_text(SOURCE)
    inc = os.path.join(ROOT, "flurrypp_b200", "csrc", "kernels")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", inc, str(src), "-o", str(tmp_path / "t")], check=True, timeout=300)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("prec", [fb.FR_PREC_FP64, fb.FR_PREC_MIXED])
def test_roe_run_with_a_negative_density_is_reported(tmp_path, prec):
    d = write_deck(str(tmp_path / "r.deck"), nDims=2, order=2, meshType=1, riemannType=1, nx=6, ny=5, xmin=0, ymin=0,
                   xmax=1, ymax=1, dt=0.001)
    s = fb.Solver(d, precision=prec)
    U = np.broadcast_to(np.array([1.0, 0.3, 0.1, 2.0]), s.shape).copy()
    U[:, -1, 0] = -1.0  # the last element: the right side of its faces
    s.set_state(U)
    s.calc_residual(0)
    with pytest.raises(fb.FrError) as e:
        s.residual_norm(2)
    assert e.value.code == fb.FR_ERR_NONFINITE
