"""GMRES + ILU on levels either side of the one-CTA kernels' limits (needs a B200): 18,755 rows
for the triangular solves, 25,600 for the Arnoldi steps, dependency levels too wide for one
CTA, rows too long for the one-CTA factorisation.  ILUPrecond bit for bit against a
restatement of LASPACK's ILUFactor / MulInv_QV compiled here (every operation in its order,
contrib/laspack/factor.c:25-320, operats.c:1049-1290; no fused multiply-add), smoother calls
against GMRESIter restated on host arrays."""
import shutil
import subprocess

import numpy as np
import pytest

import exfemus_b200 as ex
from exfemus_b200 import _lib, workloads

from test_gpu_ilu_cta import gmres
from test_gpu_upload import permuted_arrays, structured_arrays

pytestmark = pytest.mark.gpu

ORACLE = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
int main(int argc, char **argv) {
  FILE *in = fopen(argv[1], "rb"), *out = fopen(argv[2], "wb");
  int hd[2];
  if (!in || !out || fread(hd, 4, 2, in) != 2) return 1;
  const int n = hd[0], nnz = hd[1];
  std::vector<int> rp(n + 1), col(nnz), at(n, -1), dp(n);
  std::vector<double> f(nnz), c(n), inv(n), w(n), y(n);
  if (fread(rp.data(), 4, n + 1, in) != (size_t)n + 1 || fread(col.data(), 4, nnz, in) != (size_t)nnz ||
      fread(f.data(), 8, nnz, in) != (size_t)nnz || fread(c.data(), 8, n, in) != (size_t)n) return 1;
  for (int i = 0; i < n; i++) {
    int m = 0;  // S = the columns <= i, ascending
    while (col[rp[i] + m] < i) m++;
    dp[i] = rp[i] + m;
    const int *S = &col[rp[i]];
    const int M = m + 1;
    std::vector<double> B(M * M, 0.);
    std::vector<int> pl(M, -1);
    for (int b = 0; b < M; b++) at[S[b]] = b;
    for (int a = 0; a < M; a++)
      for (int k = rp[S[a]]; k < rp[S[a] + 1]; k++)
        if (at[col[k]] >= 0) {
          B[a * M + at[col[k]]] = f[k];
          if (col[k] == i) pl[a] = k;
        }
    for (int b = 0; b < M; b++) at[S[b]] = -1;
    for (int j = 0; j < m; j++)
      for (int k = j + 1; k < m; k++) {
        B[m * M + k] = B[m * M + k] - (B[m * M + j] * B[j * M + k]) / B[j * M + j];
        B[k * M + m] = B[k * M + m] - (B[j * M + m] * B[k * M + j]) / B[j * M + j];
      }
    double d = B[m * M + m];
    for (int j = 0; j < m; j++) d = d - (B[j * M + m] * B[m * M + j]) / B[j * M + j];
    for (int j = 0; j < m; j++) {
      f[rp[i] + j] = B[m * M + j];
      f[pl[j]] = B[j * M + m];
    }
    f[dp[i]] = d;
    inv[i] = 1. / d;
  }
  for (int i = 0; i < n; i++) {
    double s = 0.;
    for (int k = rp[i]; k < dp[i]; k++) s = s - f[k] * w[col[k]];
    w[i] = (s + c[i]) * inv[i];
  }
  for (int i = n - 1; i >= 0; i--) {
    double s = 0.;
    for (int k = rp[i + 1] - 1; k > dp[i]; k--) s = s - f[k] * y[col[k]];
    y[i] = (s + (0. + f[dp[i]] * w[i])) * inv[i];
  }
  return fwrite(y.data(), 8, n, out) == (size_t)n && fclose(out) == 0 ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def ilu_oracle(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("ilu")
    (d / "o.cpp").write_text(ORACLE)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", str(d / "o.cpp"), "-o", str(d / "o")], check=True)

    def run(rp, col, val, c):
        with open(d / "in", "wb") as f:
            f.write(np.array([c.size, col.size], np.int32).tobytes() + np.asarray(rp, np.int32).tobytes() +
                    np.asarray(col, np.int32).tobytes() + np.asarray(val, np.float64).tobytes() + c.tobytes())
        subprocess.run([str(d / "o"), str(d / "in"), str(d / "out")], check=True)
        return np.fromfile(d / "out", np.float64)

    return run


def system(dim, nlev, n0, permuted):
    m = ex.Mesh(dim, nlev, n0, (0, 2, 0, 1, 0, 1)[:2 * dim])
    if permuted:
        m = ex.Mesh.upload(**permuted_arrays(structured_arrays(m, n0), 3)[0])
    t = ex.MGSolT(m)
    t.GenBc(_lib.BC_HEAT_DIRICHLET)
    t.phys = ex.phys(inv_dt=1000.0)
    t.set_source(workloads.heat_source(m.nel(nlev - 1)))
    t.assemble_all()
    return t


LEVELS = [
    (2, 1, (64, 72), False, 18705),   # the last that the one-CTA solves hold
    (2, 1, (68, 68), False, 18769),   # ... and the first that they do not
    (2, 1, (79, 80), False, 25599),   # the last that the one-CTA Arnoldi step holds
    (2, 1, (80, 80), False, 25921),   # ... and the first that it does not
    (2, 2, (32, 32), True, 16641),    # random numbering: few wide levels, 15 entries up to the diagonal
    (3, 2, (4, 4, 4), True, 4913),    # rows of 75 entries up to the diagonal
    (3, 1, (13, 13, 13), False, 19683),
]


@pytest.mark.parametrize("dim,nlev,n0,permuted,rows", LEVELS)
def test_ilu_apply_bitwise(gpu_lib, ilu_oracle, dim, nlev, n0, permuted, rows):
    t = system(dim, nlev, n0, permuted)
    lev = nlev - 1
    assert t.ndof(lev) == rows
    rp, col, val = t.csr(lev)
    for seed in range(2):
        c = np.random.default_rng(seed).standard_normal(rows)
        assert np.array_equal(t.ilu_apply(lev, c), ilu_oracle(rp, col, val, c)), seed


@pytest.mark.parametrize("dim,nlev,n0,permuted,rows", [lev for lev in LEVELS if lev[-1] != 18705])
@pytest.mark.parametrize("m", [1, 4, 33])
def test_smoother_call(gpu_lib, dim, nlev, n0, permuted, rows, m):
    t = system(dim, nlev, n0, permuted)
    lev = nlev - 1
    p = ex.mg_params(smoother=_lib.SMOOTH_GMRES_ILU, eps=1e-30)
    rng = np.random.default_rng(m)
    x, b = rng.standard_normal(rows), rng.standard_normal(rows)
    got = t.smooth(lev, p, m, x, b)
    want = gmres(lambda u: t.spmv(lev, u), lambda u: t.ilu_apply(lev, u), x, b, m)
    # least squares here, rotations there: rounding of m <= 33 steps of a system whose
    # preconditioned condition number is below 1e3 (the mass term of 1000 bounds it)
    assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)


def test_factorisation_memory(gpu_lib):
    """A 257 x 257 level: factor 8.4 MB, 63 places of 4 bytes a row 16.7 MB, entries above the
    diagonal 4.2 MB, rows, orders and flags 2.5 MB: less than 40 MB in 2 MB pages (a fixed
    1 KB of places a row would take 86 MB)."""
    import torch
    t = system(2, 7, (2, 2), False)
    c = np.ones(t.ndof(6))
    t.coarse_solve(np.ones(t.ndof(0)))
    free = torch.cuda.mem_get_info()[0]
    t.ilu_apply(6, c)
    assert c.size == 257 * 257 and free - torch.cuda.mem_get_info()[0] < 40e6
