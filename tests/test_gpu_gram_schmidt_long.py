"""The Gram-Schmidt kernels over long Krylov spaces and many rows: 31, 32, 33
and 37 vectors around the 32 columns that a block's warps take at once, 29 to 31
(the most) for independent problems, and more tiles of 128 rows than blocks.

The residual after m iterations from zero is the least over the Krylov space,
which the CPU builds in float64: ILU(0) by the oracle, Arnoldi with two passes,
least squares.  Off-diagonal entries of c / sqrt(row length) in size with random
signs keep the iterations from ending before: the least residual after the last
one is 5e-6 to 0.1 of b.  In FP64 any order of the sums moves it by less than
1e-6 of itself and 1e-9 of b (m N eps < 1e-9 with a factor of 10 for the
preconditioner).  FP32 vectors and factors move it by their rounding, 6e-8 an
entry, times the coefficients' sum and the preconditioner's norm, both below 30:
1e-4 of b, and 1e-2 of itself; they are checked where it is 0.05 or more."""
import os
import re
import shutil
import subprocess

import ctypes
import numpy as np
import pytest

import oracle
from goma_gb300 import problem as pb
from goma_gb300.newton import msr_pattern_host
from tests.test_gpu_gram_schmidt import matrix
from tests.test_gpu_line_sweeps import cavity, cube, union

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CASES = {  # problem, c, independent problems
    "cavity 9x4": (lambda: cavity(9, 4), 1.0, 1),
    "cavity 20x17": (lambda: cavity(20, 17), 0.93, 1),
    "cube 4x2x3": (lambda: cube(4, 2, 3), 1.0, 1),
    "reacting 2x2x2": (lambda: pb.reacting_channel_3d(2, 2, 2), 1.02, 1),
    "3 cavities 20x17": (lambda: union(cavity(20, 17), 3), 0.93, 3),
    "cavity 180x90": (lambda: cavity(180, 90), 0.8, 1),
}


def system(prob, c):
    ija = msr_pattern_host(prob).astype(np.int64)
    N = int(ija[0]) - 1
    rng = np.random.default_rng(8)
    a = np.zeros(len(ija))
    a[:N] = 1.0
    rows = np.repeat(np.arange(N), np.diff(ija[:N + 1]))
    a[N + 1:] = c * rng.choice([-1.0, 1.0], len(rows)) / np.sqrt(np.bincount(rows, minlength=N))[rows]
    return ija, N, a, rng.uniform(-1, 1, N)


def least_residuals(A, F, b, m):
    """|b - A M^-1 V y| / |b| over the Krylov spaces of up to m vectors."""
    from scipy.sparse import identity, tril, triu
    from scipy.sparse.linalg import splu
    N = len(b)
    opts = dict(permc_spec="NATURAL", diag_pivot_thresh=0)
    lower = splu((tril(F, -1) + identity(N)).tocsc(), **opts)
    upper = splu(triu(F).tocsc(), **opts)
    V, W, best = [b / np.linalg.norm(b)], [], []
    for j in range(m):
        w = A @ upper.solve(lower.solve(V[j]))
        W.append(w.copy())
        for _ in range(2):
            for v in V:
                w -= (v @ w) * v
        V.append(w / np.linalg.norm(w))
        B = np.stack(W, 1)
        best.append(np.linalg.norm(V[0] - B @ np.linalg.lstsq(B, V[0], rcond=None)[0]))
    return best


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
def test_the_residual_is_the_least_over_a_long_space(name):
    from goma_gb300.newton import GomaNewton
    make, c, nseg = CASES[name]
    prob = make()
    ija, N, a, b = system(prob, c)
    big = name == "cavity 180x90"
    assert not big or (N > 128 * 1216 and N % 128)  # blocks take a second tile
    ms = (2, 5) if big else ((29, 30, 31) if nseg > 1 else (31, 32, 33, 37))
    A = matrix(ija, N, a).tocsr()
    F = matrix(ija, N, oracle.Oracle(prob).ilu0(a)).tocsr()
    parts = np.split(np.arange(N), nseg)
    best = [least_residuals(A[s][:, s], F[s][:, s], b[s], max(ms)) for s in parts]
    gn = GomaNewton(prob)
    for m in ms:
        for fp32 in (False, True):
            opts = dict(krylov_dim=m, max_linear_its=m, linear_tol=1e-30)
            if fp32:
                opts.update(fp32_inner=True, inner_tol=1e-30, max_refinements=1)
            x, its, _ = gn.linear_solve(a, b, **opts)
            assert its == m
            for s, e in zip(parts, best):
                got = np.linalg.norm(b[s] - A[s][:, s] @ x[s]) / np.linalg.norm(b[s])
                want = e[m - 1]
                assert want > 1e-6
                if not fp32:
                    assert abs(got - want) <= 1e-6 * want + 1e-9, (m, got, want)
                elif want >= 0.05:
                    assert abs(got - want) <= 1e-2 * want + 1e-4, (m, got, want)
    gn.close()


DOT = """
#include <cuda_runtime.h>
%s
__global__ void dot(int n, const float *a, const float *b, double *out) {
  SumF32 s;
  for (int i = 0; i < n; i++) s.add(a[i], b[i]);
  *out = s.get();
}
extern "C" int run(int n, const float *a, const float *b, double *out) {
  dot<<<1, 1>>>(n, a, b, out);
  return cudaDeviceSynchronize();
}
"""


@pytest.mark.gpu
def test_fp32_dots(tmp_path):
    """The running sum of the FP32 dots: infinite where the products' sum is,
    and otherwise the sum of the n rounded products with the error of Knuth's
    two-sum, (n 2^-24)^2 of the sum of their sizes."""
    import torch
    text = open(os.path.join(ROOT, "goma_gb300", "csrc", "gb_solve.cu")).read()
    src, so = os.path.join(tmp_path, "dot.cu"), os.path.join(tmp_path, "dot.so")
    with open(src, "w") as f:
        f.write(DOT % re.search(r"struct SumF32 \{.*?\n\};", text, re.S).group(0))
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-gencode",
                    "arch=compute_103a,code=sm_103a", "-shared", "-Xcompiler", "-fPIC", src, "-o",
                    so], check=True, capture_output=True)
    L = ctypes.CDLL(so)
    out = torch.zeros(1, dtype=torch.float64, device="cuda")

    def dot(a, b):
        a, b = (torch.tensor(np.asarray(v, np.float32), device="cuda") for v in (a, b))
        torch.cuda.synchronize()
        assert L.run(len(a), ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()),
                     ctypes.c_void_p(out.data_ptr())) == 0
        return out.item()

    big = np.full(4, 3e38)
    assert dot([1.0, 1e20, 2.0], [1.0, 1e20, 1.0]) == np.inf   # an infinite product
    assert dot([1.0, 1e20, 2.0], [1.0, -1e20, 1.0]) == -np.inf
    assert dot(big, np.ones(4)) == np.inf                      # an infinite sum
    assert np.isnan(dot([np.inf, 1.0], [0.0, 1.0]))
    rng = np.random.default_rng(1)
    for n in (1, 2, 7, 1000):
        a, b = (rng.standard_normal(n).astype(np.float32) for _ in range(2))
        p = (a * b).astype(np.float64)
        assert abs(dot(a, b) - p.sum()) <= (n * 2.0 ** -24) ** 2 * np.abs(p).sum()
