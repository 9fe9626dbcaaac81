"""The FAST-PT grid cell (fpt_cell.cuh) in both forms against extended
precision: which pairs (multipole, node) lie on the grid, their cell and their
weight, on either side of every edge.  The FP64 form rounds the coordinate to
3e-13 of a cell (three roundings at 1100 cells), the two-float form to 5e-12,
and its weight to FP32 (2^-24); pairs within 1e-9 of an edge of the grid are left
out.  A weight that rounds to 1 is the next cell's 0."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cocoa-cosmolike-core_gb300", "csrc")

SRC = r"""
#include "fpt_cell.cuh"
using namespace cl2pt;
template <typename T>
__global__ void k(Params P, int m, const double* a, const double* b, int* in, int* cell, double* w)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m) return;
  const FptCell<T> c = fpt_cell(P, FptPart<T>::of_l(P, a[t]), FptPart<T>::of_p(P, b[t]));
  in[t] = c.in;
  cell[t] = c.i;
  w[t] = (double)c.w;
}
extern "C" int run(int f64, int n, double lim0, double lim1, int m, const double* a, const double* b, int* in, int* cell,
                   double* w)
{
  static Params P;
  P.fpt_n = n;
  P.fpt_lim0 = lim0;
  P.fpt_lim1 = lim1;
  P.fpt_lim2 = (lim1 - lim0) / n;
  double *da, *db, *dw;
  int *di, *dc;
  if (cudaMalloc(&da, 8 * m) || cudaMalloc(&db, 8 * m) || cudaMalloc(&dw, 8 * m) || cudaMalloc(&di, 4 * m) ||
      cudaMalloc(&dc, 4 * m))
    return 1;
  cudaMemcpy(da, a, 8 * m, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, 8 * m, cudaMemcpyHostToDevice);
  if (f64) k<double><<<(m + 127) / 128, 128>>>(P, m, da, db, di, dc, dw);
  else k<float><<<(m + 127) / 128, 128>>>(P, m, da, db, di, dc, dw);
  cudaMemcpy(in, di, 4 * m, cudaMemcpyDeviceToHost);
  cudaMemcpy(cell, dc, 4 * m, cudaMemcpyDeviceToHost);
  cudaMemcpy(w, dw, 8 * m, cudaMemcpyDeviceToHost);
  const int e = (int)cudaGetLastError();
  cudaFree(da);
  cudaFree(db);
  cudaFree(dw);
  cudaFree(di);
  cudaFree(dc);
  return e;
}
"""


@pytest.fixture(scope="module")
def cell(tmp_path_factory):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d = tmp_path_factory.mktemp("cell")
    src, so = str(d / "cell.cu"), str(d / "cell.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"), src, "-o", so], check=True)
    return ctypes.CDLL(so).run


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64, 1100, 5000])
@pytest.mark.parametrize("f64", [0, 1])
def test_cell(cell, n, f64):
    lim0, lim1 = np.log(0.05), np.log(1e6)
    h = (lim1 - lim0) / n
    rng = np.random.default_rng(n)
    off = np.array([s * 10.0 ** -e for e in range(1, 9) for s in (1, -1)])
    r = np.concatenate([rng.uniform(-2, n + 2, 20000)] + [e + off for e in (0, 1, n // 2, n - 1, n)])
    b = rng.uniform(np.log(1e-3), np.log(3.0), r.size)
    a = lim0 + r * h + b
    L = np.longdouble
    exact = (L(1) * a - b - L(lim0)) / L((lim1 - lim0) / n)
    m = r.size
    inn, cel, w = np.zeros(m, np.int32), np.zeros(m, np.int32), np.zeros(m)
    ptr = lambda x: x.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    assert cell(f64, n, ctypes.c_double(lim0), ctypes.c_double(lim1), m, ptr(a), ptr(b), ptr(inn), ptr(cel), ptr(w)) == 0
    top = (L(lim1) - L(lim0)) / L((lim1 - lim0) / n)
    clear = (np.abs(exact) > 1e-9) & (np.abs(exact - top) > 1e-9)
    on = (exact > 0) & (exact < top)
    assert np.array_equal(inn[clear] != 0, on[clear])
    g = clear & on
    tol = 1e-9 if f64 else 2.0 ** -24 + 1e-9
    last = g & (cel + 1 >= n)
    assert (exact[last] > n - 1 - tol).all() and (w[last] == 0).all()
    g &= cel + 1 < n
    assert np.abs(cel[g] + w[g] - exact[g].astype(float)).max() <= tol
    assert (w[g] >= 0).all() and (w[g] <= 1).all()
