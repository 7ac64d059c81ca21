"""GPU: the scheduled MTTKRP above 128 columns (column panels over one
schedule) and above 4 modes (COO records of 5 to 8 modes), against the FP64
oracle: every element within the FP32 summation bound of the exact sum,
(modes + nonzeros of the row) * eps * sum of absolute products."""
import numpy as np
import pytest

from hiparti_b200 import COOTensor, DeviceTensor, synth

pytestmark = pytest.mark.gpu


def _dims(N):
    return (70, 40, 30, 9, 6, 5, 4, 3)[:N]


@pytest.mark.parametrize("N,R", [(3, 129), (3, 256), (4, 132), (4, 300), (5, 3), (5, 32), (5, 128), (6, 8), (6, 257),
                                 (7, 33), (8, 16), (8, 150)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_coo_panels_and_orders(lib, cuda, orc, N, R, dtype):
    import torch
    dims = _dims(N)
    # from where ranks above 128 take panels and orders above 4 schedules; the
    # last tile holds one nonzero
    nnz = 262_145 if N > 4 else 16_385
    inds, vals = synth.zipf_tensor(dims, nnz, s=1.1, seed=N * 1000 + R)
    mats = synth.factor_matrices(dims, R, seed=R + 1)
    dmats = [torch.from_numpy(m).to(cuda).to(getattr(torch, dtype)) for m in mats]
    fm = [d.float().cpu().numpy() for d in dmats]
    dt = DeviceTensor.from_coo(COOTensor(dims, inds, vals))
    eps = np.finfo(np.float32).eps
    for m in range(N):
        got = dt.mttkrp(dmats, m, rank=R).cpu().numpy()
        exact = orc.mttkrp_coo_f64(inds, vals, fm, R, m)[: dims[m]]  # all terms are positive: also the bound's sum
        rows = np.bincount(inds[m], minlength=dims[m])[:, None]
        assert np.all(np.abs(got - exact)[:, :R] <= ((N + rows) * eps * exact)[:, :R] + 1e-30), (N, R, m)
        assert not got[:, R:].any()
    dt.check()
    dt.free()


@pytest.mark.parametrize("N,R", [(3, 200), (5, 16)])
def test_first_use_under_capture_and_on_two_streams(lib, cuda, orc, N, R):
    """A first call inside a stream capture keeps to the kernels without a
    schedule; a first call on one stream followed by one on another waits for
    the build."""
    import torch
    dims = _dims(N)
    inds, vals = synth.uniform_tensor(dims, 20_000 if N == 3 else 270_000, seed=N)
    mats = synth.factor_matrices(dims, R, seed=R)
    dmats = [torch.from_numpy(m).to(cuda) for m in mats]
    want = orc.mttkrp_coo_f64(inds, vals, mats, R, 1)[: dims[1]]
    dt = DeviceTensor.from_coo(COOTensor(dims, inds, vals))
    out = torch.empty((dims[1], mats[0].shape[1]), device=cuda)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        dt.mttkrp(dmats, 1, rank=R, out=out)
    for _ in range(2):
        out.fill_(7.0)
        g.replay()
        torch.cuda.synchronize()
        assert np.abs(out.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()
    del g
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        x = dt.mttkrp(dmats, 1, rank=R)
    with torch.cuda.stream(b):
        y = dt.mttkrp(dmats, 1, rank=R)
    torch.cuda.synchronize()
    for o in (x, y):
        assert np.abs(o.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()
    dt.check()
    dt.free()


def test_prepare_of_five_modes(lib, cuda, orc):
    """HiCOO tensors of five modes have no schedule to build and say so by
    succeeding; COO ones are refused."""
    import torch
    from hiparti_b200 import HiCOOTensor
    dims, n = (4, 5, 6, 7, 8), 300
    rng = np.random.default_rng(5)
    inds = [rng.integers(0, d, n).astype(np.uint32) for d in dims]
    vals = rng.random(n).astype(np.float32)
    h = HiCOOTensor(dims, 4, 6, 8, [0, n], [[0]] * 5, inds, vals)
    mats = synth.factor_matrices(dims, 8, seed=1)
    dmats = [torch.from_numpy(m).to(cuda) for m in mats]
    dt = DeviceTensor.from_hicoo(h)
    dt.prepare()
    want = orc.mttkrp_coo_f64(inds, vals, mats, 8, 2)[: dims[2]]
    got = dt.mttkrp(dmats, 2, rank=8).cpu().numpy()
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    dt.free()
    dc = DeviceTensor.from_coo(COOTensor(dims, inds, vals))
    with pytest.raises(Exception):
        dc.prepare()
    dc.free()
