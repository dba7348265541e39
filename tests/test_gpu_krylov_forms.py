"""Krylov kernels at the forms where they choose another path: conversions on
the integer pipe, vectors that are not 16-byte aligned, ragged row counts."""
import numpy as np
import pytest
import torch

from ucfd_sparse_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_fp32_conversions_round_as_the_type_does(ucfd):
    """FP32 values and products of a diagonal matrix: ties to even either way,
    subnormal, overflowing, infinite, NaN and signed zero entries, and random
    bit patterns, equal the conversions of numpy."""
    from ucfd_sparse_gb300.krylov import SpMat
    rng = np.random.default_rng(3)
    e = np.array([1 + 2.0 ** -24, 1 + 3 * 2.0 ** -24, 1 + 2.0 ** -24 + 2.0 ** -52, 2 - 2.0 ** -24, 2 - 2.0 ** -25,
                  2.0 ** -126, 2.0 ** -126 * (1 - 2.0 ** -25), 2.0 ** -149, 2.0 ** -150, 1.5 * 2.0 ** -150, 1e-300,
                  5e-324, float(np.finfo(np.float32).max), float(np.finfo(np.float32).max) * (1 + 2.0 ** -25), 1e39,
                  np.inf, np.nan, 0.0])
    bits = rng.integers(0, 1 << 63, 200000, dtype=np.uint64) | (rng.integers(0, 2, 200000, dtype=np.uint64) << np.uint64(63))
    near = ((bits & np.uint64(0x800fffffffffffff)) |
            (rng.integers(1023 - 160, 1023 + 140, 200000).astype(np.uint64) << np.uint64(52)))
    x = np.concatenate([e, -e, bits.view(np.float64), near.view(np.float64)])
    n = x.size
    idx = np.arange(n, dtype=np.int32)
    one, rp = dev(np.ones(n)), dev(np.arange(n + 1, dtype=np.int32))
    y = torch.zeros(n, dtype=torch.float64, device="cuda")
    with np.errstate(over="ignore", invalid="ignore"):
        want = x.astype(np.float32).astype(np.float64)
    # as matrix values (their FP32 copy), then as the multiplied vector
    for values, vec in ((dev(x), one), (one, dev(x))):
        torch.cuda.synchronize()
        SpMat(n, 1, rp, dev(idx), values).mult(1.0, vec, 0.0, y, fp32=True)
        np.testing.assert_array_equal(y.cpu().numpy(), want)


# one warp's worth of rows less one, exactly, and one more; several blocks
@pytest.mark.parametrize("bn", [31, 32, 33, 1000])
@pytest.mark.parametrize("blk", [1, 5, 7])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_matvec_and_apply_of_unaligned_vectors(bn, blk, prec, port, ucfd):
    """The same product and preconditioner apply from vectors 8 bytes off a
    16-byte boundary and from aligned ones, at ragged row counts; the product
    in FP64 against the oracle bit for bit."""
    from ucfd_sparse_gb300.krylov import Precon, SpMat
    rng = np.random.default_rng(bn + blk)
    nei = np.stack([np.where(np.arange(bn) >= d, np.arange(bn) - d, -1) for d in (1, 3)] +
                   [np.where(np.arange(bn) < bn - d, np.arange(bn) + d, -1) for d in (1, 3)]).astype(np.int32)
    s = mg.bsr_from_table(nei, blk, seed=bn)
    rp, ci, ds, va = (dev(s[k]) for k in ("rowptr", "colidx", "diagslots", "values"))
    A = SpMat(bn, blk, rp, ci, va)
    pc = Precon(rp, ci, ds, va)
    pc.set_blusgs(bn, blk)
    pc.set_precision(prec)
    pc.prepare()
    x = rng.standard_normal(bn * blk)
    out = []
    for off in (0, 1):
        store = torch.zeros(bn * blk + 2, dtype=torch.float64, device="cuda")
        xv, y = store[off:off + bn * blk], torch.zeros(bn * blk + 2, dtype=torch.float64, device="cuda")[off:off + bn * blk]
        xv.copy_(dev(x))
        torch.cuda.synchronize()
        A.mult(1.0, xv, 0.0, y, precision=prec)
        pc.apply(xv)
        out.append((y.cpu().numpy(), xv.cpu().numpy()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    if prec == 0:
        np.testing.assert_array_equal(out[0][0], port.bsr_spmv(s, x))
