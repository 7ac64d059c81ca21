"""GPU: tensors of few tiles, and the CP model's tiles cut for them.  Sizes around
one tile, a part and a wave, with rows that continue across parts; MTTKRP and
the CP model against FP64 (all terms positive: the FP32 summation bound of an
element is (modes + nonzeros of its row) * eps times the element)."""
import numpy as np
import pytest

from hiparti_b200 import COOTensor, DeviceTensor, synth

pytestmark = pytest.mark.gpu


# a turn of the GPU is 592 tiles of 2048: within one, just over one, three even turns, more than five
@pytest.mark.parametrize("nnz", [1_211_111, 1_212_417, 3_100_003, 6_100_001])
@pytest.mark.parametrize("R", [16, 40])
def test_even_turns(lib, cuda, orc, nnz, R):
    import torch
    dims = (300, 250, 200)
    inds, vals = synth.uniform_tensor(dims, nnz, seed=nnz)
    mats = synth.factor_matrices(dims, R, seed=R)
    dmats = [torch.from_numpy(m).to(cuda) for m in mats]
    eps = np.finfo(np.float32).eps
    coo = DeviceTensor.from_coo(COOTensor(dims, inds, vals))
    want = orc.mttkrp_coo_f64(inds, vals, mats, R, 1)[: dims[1]]
    rows = np.bincount(inds[1], minlength=dims[1])[:, None]
    got = coo.mttkrp(dmats, 1, rank=R).cpu().numpy()
    assert np.all(np.abs(got - want) <= (3 + rows) * eps * want + 1e-30)
    model = coo.kruskal_values(dmats, rank=R).cpu().numpy()
    p = mats[0][inds[0][::97], :R].astype(np.float64) * mats[1][inds[1][::97], :R] * mats[2][inds[2][::97], :R]
    assert np.all(np.abs(model[::97] - p.sum(1)) <= (3 + R) * eps * p.sum(1))
    coo.free()


@pytest.mark.parametrize("nnz", [1, 63, 257, 2047, 2049, 4099, 40_000])
@pytest.mark.parametrize("R", [4, 10, 32, 128])
@pytest.mark.parametrize("N", [3, 4])
def test_parts(lib, cuda, orc, nnz, R, N):
    import torch
    dims = (60, 50, 40) if N == 3 else (40, 30, 20, 10)
    inds, vals = synth.zipf_tensor(dims, nnz, s=1.1, seed=nnz + R)
    mats = synth.factor_matrices(dims, R, seed=R)
    dmats = [torch.from_numpy(m).to(cuda) for m in mats]
    eps = np.finfo(np.float32).eps
    coo = DeviceTensor.from_coo(COOTensor(dims, inds, vals))
    hic = coo.to_hicoo(4, 6, 8)
    for m in range(N):
        want = orc.mttkrp_coo_f64(inds, vals, mats, R, m)[: dims[m]]
        rows = np.bincount(inds[m], minlength=dims[m])[:, None]
        for dt in (coo, hic):
            got = dt.mttkrp(dmats, m, rank=R).cpu().numpy()
            assert np.all(np.abs(got - want) <= (N + rows) * eps * want + 1e-30), (nnz, R, m)
    model = coo.kruskal_values(dmats, rank=R).cpu().numpy()
    p = np.ones((nnz, R))
    for a, ix in zip(mats, inds):
        p *= a[ix, :R].astype(np.float64)
    assert np.all(np.abs(model - p.sum(1)) <= (N + R) * eps * p.sum(1))
    for dt in (coo, hic):
        dt.check()
        dt.free()
