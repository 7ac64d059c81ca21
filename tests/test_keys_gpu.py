"""GPU: COO -> HiCOO around the limits of its one-word sort keys (3-D: Morton
bits up to 21 a mode, 4-D: up to 16, 64 bits in all; wider keys take two words),
on the host path and on the device, against the oracle's conversion; schedules
built from the result, and from blocks whose element offsets pass the block
edge, against FP64."""
import numpy as np
import pytest

from hiparti_b200 import COOTensor, DeviceTensor, HiCOOTensor, ffi, synth

pytestmark = pytest.mark.gpu

CASES = [
    ((300, 200, 100), 5000, 3, 5, 6),
    ((300, 200, 100), 1, 2, 2, 2),
    ((300, 2, 1), 200, 4, 12, 20),
    ((5000, 4000, 3000), 4097, 8, 10, 14),
    ((1 << 21, 1 << 20, 3000), 20000, 7, 21, 21),            # 63 Morton bits
    (((1 << 21) + 5, 1 << 20, 3000), 20000, 7, 21, 21),      # and one kernel bit: 64
    (((1 << 21) + 5, (1 << 21) + 9, 3000), 20000, 7, 21, 21),  # 65
    ((1 << 22, 1 << 20, 3000), 20000, 7, 22, 22),            # 22 bits a mode
    ((1 << 25, 1 << 25, 40), 20000, 1, 20, 20),              # 60 Morton bits and 10 kernel bits
    ((1 << 25, 1 << 20, 40), 20000, 5, 25, 25),              # above the reference's 24 bits
    ((90, 80, 70, 60), 30000, 3, 4, 5),
    ((1 << 16, 3000, 2000, 50), 30000, 7, 16, 16),           # 64 Morton bits
    (((1 << 16) + 1, 3000, 2000, 50), 30000, 7, 16, 16),     # 65
    ((1 << 17, 3000, 2000, 50), 30000, 7, 17, 17),
    ((40000, 30000, 20000, 500), 30000, 7, 10, 14),
]


def _download(lib, h, N, nnz):
    nb = h.nb
    bptr, vals = np.empty(nb + 1, np.uint64), np.empty(nnz, np.float32)
    binds, einds = [np.empty(nb, np.uint32) for _ in range(N)], [np.empty(nnz, np.uint8) for _ in range(N)]
    bp = ffi.new("void *[]", [ffi.cast("void *", b.ctypes.data) for b in binds])
    ep = ffi.new("void *[]", [ffi.cast("void *", e.ctypes.data) for e in einds])
    assert lib.ptiB200DownloadHiCOO(h._h, ffi.cast("ptiNnzIndex *", bptr.ctypes.data), bp, ep,
                                    ffi.cast("ptiValue *", vals.ctypes.data)) == 0
    return bptr, binds, einds, vals


@pytest.mark.parametrize("dims,nnz,sb,sk,sc", CASES)
def test_conversion(lib, cuda, orc, dims, nnz, sb, sk, sc):
    N = len(dims)
    inds, vals = synth.uniform_tensor(dims, nnz, seed=nnz + sb)
    o = orc.hicoo_build(dims, inds, vals, sb, sk, sc)
    dev = DeviceTensor.from_coo(COOTensor(dims, inds, vals)).to_hicoo(sb, sk, sc)
    host = COOTensor(dims, [i.copy() for i in inds], vals.copy())
    h = host.to_hicoo(sb, sk, sc)
    for key in ("bptr", "kptr", "cptr", "vals"):
        np.testing.assert_array_equal(getattr(h, key), o[key])
    bptr, binds, einds, dv = _download(lib, dev, N, nnz)
    np.testing.assert_array_equal(bptr, o["bptr"])
    np.testing.assert_array_equal(dv, o["vals"])
    assert dev.max_nnzb == h.max_nnzb == int(np.diff(o["bptr"].astype(np.int64)).max())
    blk = np.repeat(np.arange(h.nb), np.diff(o["bptr"].astype(np.int64)))
    for m in range(N):
        np.testing.assert_array_equal(h.binds[m], o["binds"][m])
        np.testing.assert_array_equal(h.einds[m], o["einds"][m])
        np.testing.assert_array_equal(binds[m], o["binds"][m])
        np.testing.assert_array_equal(einds[m], o["einds"][m])
        # the caller's COO is left in HiCOO order
        np.testing.assert_array_equal(host.inds[m], (o["binds"][m][blk] << sb) + o["einds"][m])
    np.testing.assert_array_equal(host.vals, o["vals"])
    small = [m for m in range(N) if dims[m] <= 5000]
    if len(small) == N:
        _check_mttkrp(orc, dev, dims, inds, vals)
    dev.free()


def _check_mttkrp(orc, dt, dims, inds, vals, R=12):
    import torch
    mats = synth.factor_matrices(dims, R, seed=3)
    dmats = [torch.from_numpy(m).cuda() for m in mats]
    eps = np.finfo(np.float32).eps
    for m in range(len(dims)):
        for dtype in (torch.float32, torch.bfloat16):  # the decoding kernel (3-D) and the records
            fm = [d.to(dtype) for d in dmats]
            got = dt.mttkrp(fm, m, rank=R).cpu().numpy()
            want = orc.mttkrp_coo_f64(inds, vals, [f.float().cpu().numpy() for f in fm], R, m)[: dims[m]]
            rows = np.bincount(inds[m], minlength=dims[m])[:, None]
            assert np.all(np.abs(got - want) <= (len(dims) + rows) * eps * want + 1e-30), m
    dt.check()


@pytest.mark.parametrize("dims,nnz", [((700, 40, 30), 3000), ((700, 600, 500), 2048), ((60, 50, 40, 30), 9000)])
def test_offsets_past_the_block_edge(lib, cuda, orc, dims, nnz):
    """Element offsets of 8 bits in blocks of 4: rows of neighbouring blocks
    interleave, and a tile's rows still have to come out in order."""
    N, sb = len(dims), 2
    inds, vals = synth.zipf_tensor(dims, nnz, s=1.1, seed=nnz)
    rng = np.random.default_rng(1)
    back = [np.minimum(i, rng.integers(0, 250, nnz)).astype(np.uint32) for i in inds]  # offset to aim for
    bl = [((i - b) >> sb).astype(np.int64) for i, b in zip(inds, back)]
    order = np.lexsort(tuple(bl[::-1]))
    key = np.stack([b[order] for b in bl], 1)
    start = np.flatnonzero(np.append(True, np.any(key[1:] != key[:-1], axis=1)))
    bptr = np.append(start, nnz).astype(np.uint64)
    einds = [(i[order] - (b[order].astype(np.uint32) << sb)).astype(np.uint8) for i, b in zip(inds, bl)]
    dt = DeviceTensor.from_hicoo(HiCOOTensor(dims, sb, 4, 5, bptr, [k[start].astype(np.uint32) for k in key.T], einds,
                                             vals[order]))
    _check_mttkrp(orc, dt, dims, inds, vals)
    dt.free()
