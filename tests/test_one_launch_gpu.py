"""The one-launch RK stage against the two-kernel form (faces, then elements).

Both forms evaluate the same operations up to the order of the sums over
directions, so FP64 arrays agree to a few tens of ulps of the largest value
per stage and FP32 ones likewise: with at most 50 roundings a stage and 16
stages, 50 * 16 * 2^-53 = 9e-14 (FP64) and 50 * 16 * 2^-24 = 5e-5 (FP32).
Residuals are differences of flux terms, which the operators scale by up to
(P + 1)^2; they are compared on the scale of that."""
import os
import subprocess

import numpy as np
import pytest

import flurrypp_b200 as fb
from conftest import ROOT
from flurrypp_b200.decks import write_deck

pytestmark = pytest.mark.gpu
TOL = {fb.FR_PREC_FP64: 9e-14, fb.FR_PREC_MIXED: 5e-5}

WALLS = dict(create_bcBottom="slip_wall", create_bcTop="slip_wall", create_bcLeft="char", create_bcRight="char")


def deck(tmp_path, nd, order, size, **kw):
    o = dict(nDims=nd, order=order, meshType=1, dt=0.002, CFL=0.3, uBound=0.35, pBound=0.7142857143)
    for name, n in zip("xyz", size):
        o.update({"n" + name: n, name + "min": 0, name + "max": 1.0})
    o.update(kw)
    return write_deck(str(tmp_path / "case.deck"), **o)


def start(s):
    """Free stream with a 1 % seeded disturbance of every value."""
    v = np.array([0.35, 0.1, 0.05])[:s.nDims]
    u = np.concatenate([[1.0], v, [0.7142857143 / 0.4 + 0.5 * (v @ v)]])
    r = np.random.default_rng(7).uniform(-0.01, 0.01, s.shape)
    return u * (1 + r)


def snapshot(s):
    names = ["U_spts", "U0", "U_fpts", "Fn_fpts", "waveSp_fpts", "divF_0"]
    return {n: s.get_array(n) for n in names}


def compare(d, prec, tmp_order, **opts):
    one = fb.Solver(d, precision=prec, **opts)
    two = fb.Solver(d, precision=prec, tile_variant=0, **opts)
    U = start(one)
    kernels = []
    for s in (one, two):
        s.set_state(U)
        s.update()
        n0 = s.info().launches
        s.run(3)
        kernels.append(s.info().launches - n0)
    assert kernels[0] < kernels[1]  # the forms really differ
    flux = None
    for stage in ("run", "residual"):
        a, b = snapshot(one), snapshot(two)
        flux = max(float(np.max(np.abs(b["Fn_fpts"]))), float(np.max(np.abs(b["U_spts"]))))
        for n in a:
            scale = flux * (tmp_order + 1) ** 2 if n == "divF_0" else float(np.max(np.abs(b[n]))) or 1.0
            if n == "Fn_fpts":
                scale = flux
            assert np.max(np.abs(a[n] - b[n])) <= TOL[prec] * scale, (stage, n)
        if prec == fb.FR_PREC_FP64:  # FP32: a CFL step follows the wave speeds, compared above
            assert abs(one.info().time - two.info().time) <= 1e-12 * two.info().time
        one.calc_residual(0)
        two.calc_residual(0)


@pytest.mark.parametrize("prec", [fb.FR_PREC_FP64, fb.FR_PREC_MIXED])
@pytest.mark.parametrize("order", range(6))
@pytest.mark.parametrize("size", [(5, 3), (4, 4), (11, 3), (7, 5, 3), (4, 3, 3), (3, 3, 3)])
def test_orders_and_block_remainders(tmp_path, prec, order, size):
    """Every order on element counts around the block sizes (15, 16, 33 in
    2-D; 105 and 27, which rule out TMA rows, and 36 in 3-D), walls and far
    field on the first size of each dimension."""
    nd = len(size)
    d = deck(tmp_path, nd, order, size, **(WALLS if size in ((5, 3), (7, 5, 3)) else {}))
    compare(d, prec, order)


@pytest.mark.parametrize("prec", [fb.FR_PREC_FP64, fb.FR_PREC_MIXED])
@pytest.mark.parametrize("kw", [dict(timeType=2), dict(timeType=5), dict(timeType=6), dict(dtType=1), dict(dtType=2),
                                dict(dtType=2, timeType=5), dict(spts_type_quad="Lobatto", vcjhSchemeQuad=2)])
@pytest.mark.parametrize("size", [(9, 4), (4, 3, 3)])
def test_time_schemes_and_steps(tmp_path, prec, kw, size):
    compare(deck(tmp_path, len(size), 3, size, **WALLS, **kw), prec, 3)


@pytest.mark.parametrize("prec", [fb.FR_PREC_FP64, fb.FR_PREC_MIXED])
@pytest.mark.parametrize("order", [1, 4])
def test_roe(tmp_path, prec, order):
    compare(deck(tmp_path, 2, order, (9, 5), riemannType=1, **WALLS), prec, order)


@pytest.mark.parametrize("prec", [fb.FR_PREC_FP64, fb.FR_PREC_MIXED])
def test_common_flux_behind_a_kept_pointer(tmp_path, prec):
    """Fn_fpts is formed on demand; a caller that took its device pointer
    sees it refreshed by every call, and a new state leaves the last
    evaluation's values in place."""
    import torch

    s = fb.Solver(deck(tmp_path, 2, 3, (6, 5), **WALLS), precision=prec)
    s.set_state(start(s))
    s.update()
    ptr, size = s.device_ptr("Fn_fpts")

    class View:
        __cuda_array_interface__ = {"shape": (size // (4 if prec else 8),), "typestr": "<f4" if prec else "<f8",
                                    "data": (ptr, False), "version": 2}

    view = torch.as_tensor(View(), device="cuda")
    for call in (lambda: s.run(2), s.update, lambda: s.calc_residual(0)):
        call()
        s.synchronize()
        got = view.cpu().numpy().astype(np.float64)
        assert np.array_equal(got, s.get_array("Fn_fpts"))
    ref = fb.Solver(deck(tmp_path, 2, 3, (6, 5), **WALLS), precision=prec)
    ref.set_state(start(ref))
    ref.calc_residual(0)
    before = ref.get_array("Fn_fpts")
    ref.calc_residual(0)
    ref.set_state(1.1 * start(ref))
    assert np.array_equal(ref.get_array("Fn_fpts"), before)


def test_reciprocal_and_root_within_one_ulp(tmp_path):
    """recip and root of the flux functions against CUDA's correctly rounded
    division and square root, over 60 decades (FP32: 24)."""
    src = tmp_path / "t.cu"
    src.write_text(r'''
#include <cstdio>
#include <cmath>
#include "fr_physics.cuh"
__global__ void k(unsigned long long *out) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long h = (i + 1) * 0x9E3779B97F4A7C15ull;
  h ^= h >> 29; h *= 0xBF58476D1CE4E5B9ull; h ^= h >> 32;
  const double m = 1.0 + (double)(h >> 12) * 0x1p-52;
  const double x = ldexp(m, (int)(i % 200) - 100);
  const float xf = ldexpf((float)m, (int)(i % 80) - 40);
  const double r[2] = {frk::recip(x), frk::root(x)}, e[2] = {1.0 / x, sqrt(x)};
  const float rf[2] = {frk::recip(xf), frk::root(xf)}, ef[2] = {1.0f / xf, sqrtf(xf)};
  for (int q = 0; q < 2; q++) {
    const long long d = llabs(__double_as_longlong(r[q]) - __double_as_longlong(e[q]));
    const int f = abs(__float_as_int(rf[q]) - __float_as_int(ef[q]));
    atomicMax(&out[q], (unsigned long long)d);
    atomicMax(&out[2 + q], (unsigned long long)f);
  }
  if (i == 0 && (frk::root(0.0) != 0.0 || frk::root(0.0f) != 0.0f)) out[4] = 1;
}
int main() {
  unsigned long long *d, h[5];
  cudaMalloc(&d, sizeof h);
  cudaMemset(d, 0, sizeof h);
  k<<<4096, 256>>>(d);
  cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost);
  printf("%llu %llu %llu %llu %llu\n", h[0], h[1], h[2], h[3], h[4]);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
''')
    exe = tmp_path / "t"
    inc = os.path.join(ROOT, "flurrypp_b200", "csrc", "kernels")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", inc, str(src), "-o", str(exe)], check=True, timeout=300)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=60).stdout.split()
    ulps = [int(v) for v in out]
    assert max(ulps[:4]) <= 1 and ulps[4] == 0, ulps
