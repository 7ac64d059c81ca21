"""GPU: the dense steps of ALS (Gram, inverse, row solve) over every tile count
and both sides of each kernel's rank limit, against FP64."""
import numpy as np
import pytest

from conftest import rel_err
from hiparti_b200 import COOTensor, DeviceTensor, ffi, synth
from hiparti_b200.api import _MatrixSet

pytestmark = pytest.mark.gpu


def _solve(lib, grams, rhs, R):
    S = _MatrixSet([g.copy() for g in grams] + [np.zeros_like(grams[0])], R)
    T = _MatrixSet([rhs], R)
    assert lib.ptiMatrixSolveNormals(0, len(grams), S.ptrs, T.ptrs[0]) == 0


@pytest.mark.parametrize("R,stride", [(1, 8), (7, 8), (8, 8), (9, 9), (17, 24), (31, 33), (32, 32), (33, 40), (56, 64),
                                      (64, 64), (65, 70), (100, 104), (121, 128), (128, 136)])
@pytest.mark.parametrize("I", [1, 9, 1003])
def test_solve_normals(lib, cuda, R, stride, I):
    """Pad columns that are NaN must not be read as data.  The rows are FP32
    results of an FP64 solve: 1e-6 with condition numbers below 1e4."""
    rng = np.random.default_rng(R * 7 + I)
    grams = []
    for _ in range(3):
        a = rng.standard_normal((4 * R + 20, R))
        g = np.full((R, stride), np.nan, np.float32)
        g[:, :R] = a.T @ a
        grams.append(g)
    rhs0 = rng.standard_normal((I, R)).astype(np.float32)
    rhs = np.full((I, stride), np.nan, np.float32)
    rhs[:, :R] = rhs0
    _solve(lib, grams, rhs, R)
    V = grams[1][:, :R].astype(np.float64) * grams[2][:, :R]
    V = np.triu(V) + np.triu(V, 1).T
    assert rel_err(rhs[:, :R], np.linalg.solve(V, rhs0.astype(np.float64).T).T) < 1e-6
    assert not rhs[:, R:].any()


@pytest.mark.parametrize("R", [5, 40, 100])
def test_not_positive_definite(lib, cuda, R):
    """An indefinite matrix is solved by the pivoting fallback, a singular one
    leaves the rows as they are."""
    rng = np.random.default_rng(R)
    stride = (R + 7) // 8 * 8
    a = rng.standard_normal((3 * R, R))
    one = np.ones((R, stride), np.float32)
    g = np.zeros((R, stride), np.float32)
    g[:, :R] = a.T @ a
    g[R // 2, R // 2] *= -1
    rhs = np.zeros((50, stride), np.float32)
    rhs[:, :R] = rng.standard_normal((50, R))
    want = np.linalg.solve(g[:, :R].astype(np.float64), rhs[:, :R].astype(np.float64).T).T
    got = rhs.copy()
    _solve(lib, [one, g, one], got, R)
    assert rel_err(got[:, :R], want) < 1e-5
    g[R // 2, :] = 0
    g[:, R // 2] = 0
    got = rhs.copy()
    _solve(lib, [one, g, one], got, R)
    np.testing.assert_array_equal(got, rhs)


@pytest.mark.parametrize("R", [1, 8, 20, 33, 48, 64, 65, 80, 128])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_als_iterations(lib, cuda, orc, R, precision):
    """Three iterations against the FP64 oracle, rows with a pad, mode sizes
    around the row tiles (8 and 32).  BF16: one iteration from factors that are
    BF16 values, where only the gathers of later modes see rounded factors."""
    import torch
    dims = (65, 257, 31)
    inds, vals = synth.uniform_tensor(dims, 60_000, seed=R)
    rng = np.random.default_rng(R)
    init = [torch.from_numpy(rng.standard_normal((d, R)).astype(np.float32)).bfloat16().float().numpy() for d in dims]
    iters = 3 if precision == "fp32" else 1
    o = orc.cpd_als(dims, inds, vals, R, iters, init)
    dt = DeviceTensor.from_coo(COOTensor(dims, inds, vals))
    stride = (R + 7) // 8 * 8 + 8
    fac = []
    for a in init:
        f = torch.full((a.shape[0], stride), 3.0, device=cuda)
        f[:, :R] = torch.from_numpy(a).to(cuda)
        fac.append(f)
    lam, fits = dt.cpd_als(fac, iters, rank=R, precision=precision, fp32_sweeps=0)
    tol = 2e-4 if precision == "fp32" else 2e-2
    for f, w in zip(fac, o["factors"]):
        assert rel_err(f[:, :R].cpu().numpy(), w) < tol
    assert rel_err(lam.cpu().numpy(), o["lambda_"]) < tol
    assert abs(fits[-1] - o["fit"]) < tol
    dt.free()
