"""GPU: lane groups whose size is no power of two (6, 9 and 10 lanes leave 2, 5
and 2 lanes of a warp without a group): both sides of the ranks that take them,
COO and HiCOO, 3- and 4-D, FP32 and BF16 rows, tiles with a remainder and rows
that fill many groups, against FP64 within the FP32 summation bound."""
import numpy as np
import pytest

from hiparti_b200 import COOTensor, DeviceTensor, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [3, 4])
@pytest.mark.parametrize("dtype,ranks", [("float32", (20, 21, 24, 33, 36, 37, 40, 41)),
                                         ("bfloat16", (40, 41, 48, 65, 72, 73, 80, 81))])
@pytest.mark.parametrize("nnz", [7, 5_001])
def test_lane_groups(lib, cuda, orc, N, dtype, ranks, nnz):
    import torch
    dims = (30, 40, 50) if N == 3 else (20, 30, 15, 10)
    inds, vals = synth.zipf_tensor(dims, nnz, s=1.1, seed=nnz)
    coo = DeviceTensor.from_coo(COOTensor(dims, inds, vals))
    hic = coo.to_hicoo(4, 6, 8)
    eps = np.finfo(np.float32).eps
    for R in ranks:
        mats = synth.factor_matrices(dims, R, seed=R)
        dmats = [torch.from_numpy(m).to(cuda).to(getattr(torch, dtype)) for m in mats]
        fm = [d.float().cpu().numpy() for d in dmats]
        for m in range(N):
            want = orc.mttkrp_coo_f64(inds, vals, fm, R, m)[: dims[m]]
            rows = np.bincount(inds[m], minlength=dims[m])[:, None]
            for dt in (coo, hic):
                got = dt.mttkrp(dmats, m, rank=R).cpu().numpy()
                assert np.all(np.abs(got - want) <= (N + rows) * eps * want + 1e-30), (R, m)
                assert not got[:, R:].any()
    for dt in (coo, hic):
        dt.check()
        dt.free()
