"""The reference memory image to and from the device layout: gauge fields by
blocks of 32 sites, and the general path (other multiplicities, image
addresses that are only 8-byte aligned), exactly, in both precisions."""

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("ts", [(1, 1, 1, 1), (31, 1, 1, 1), (4, 4, 2, 1), (3, 11, 1, 1), (5, 4, 3, 7), (8, 8, 8, 9)])
@pytest.mark.parametrize("single", [False, True])
def test_round_trip(q, ts, single):
    import torch
    geo, V = q.Geometry(ts), int(np.prod(ts))
    rng = np.random.default_rng(V)
    for m in (4, 1, 3):
        a = rng.standard_normal((V, m, 3, 3)) + 1j * rng.standard_normal((V, m, 3, 3))
        want = a.astype(np.complex64).astype(np.complex128) if single else a
        f = q.FieldColorMatrix(geo, m, precision=q.F32 if single else q.F64)
        f.from_numpy(a)
        assert np.array_equal(f.to_numpy(), want)
        assert np.isclose(f.qnorm(), (np.abs(want) ** 2).sum(), rtol=1e-12)  # the padding stays zero
        # a device image at a 16-byte boundary and 8 bytes past one; the words around it stay
        flat = torch.from_numpy(np.ascontiguousarray(a).view(np.float64).ravel()).cuda()
        for shift in (0, 1):
            src = torch.zeros(flat.numel() + 4, dtype=torch.float64, device="cuda")
            src[shift:shift + flat.numel()] = flat
            dst = torch.full_like(src, 7.0)
            torch.cuda.synchronize()
            g = q.FieldColorMatrix(geo, m, precision=f.precision)
            g.upload_device(src[shift:].data_ptr())
            g.download_device(dst[shift:].data_ptr())
            q.synchronize()
            out = dst.cpu().numpy()
            assert np.array_equal(out[shift:shift + flat.numel()].view(np.complex128).reshape(a.shape), want)
            assert (out[:shift] == 7.0).all() and (out[shift + flat.numel():] == 7.0).all()


@pytest.mark.gpu
def test_chains_of_a_batch_start_anywhere(q):
    shapes = [(3, 3, 3, 3), (4, 4, 4, 4), (6, 6, 6, 6), (2, 2, 2, 2)]
    b = q.ChainBatch(shapes, [5.5] * 4)
    rng = np.random.default_rng(0)
    a = [rng.standard_normal((int(np.prod(s)), 4, 3, 3)) + 0j for s in shapes]
    for c in (2, 0, 3, 1):
        b.chain_from_numpy(c, a[c])
    for c in range(4):
        assert np.array_equal(b.chain_to_numpy(c), a[c])
