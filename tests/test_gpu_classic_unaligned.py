"""GPU: classic jobs whose shard pointers are not 16-byte aligned against the
oracle, byte for byte: shards packed back to back at odd lengths (every
alignment occurs), lengths from one byte over the first whole word to several
tiles, one to nine outputs, encode, verify, rebuild and the accumulating
incremental calls, on few columns (byte kernel) and on many (word kernel);
bytes around the shards must stay."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 1), (2, 1, 3), (3, 2, 7), (4, 2, 11), (4, 4, 12), (5, 3, 13), (6, 3, 21), (9, 4, 127), (10, 4, 1029),
         (12, 4, 4095), (12, 4, 4107), (16, 4, 8211), (21, 5, 4099), (30, 9, 301), (7, 8, 12305), (12, 4, 100003)]


@pytest.mark.parametrize("k,m,length", CASES)
@pytest.mark.parametrize("shift,columns", [(0, 0), (5, 0), (1, 260 << 10), (10, 260 << 10)])
def test_packed_odd_shards(k, m, length, shift, columns):
    import torch

    import rsgpu

    rng = np.random.default_rng(k * 1000 + m + length)
    total, stripes = k + m, max(3, min(24000, columns // length + 1))
    check = np.unique(np.r_[0:3, rng.integers(0, stripes, 9), stripes - 1])  # stripes the oracle computes
    codec = rsgpu.ReedSolomon(k, m)
    rc, mat = O.build_matrix(k, m)
    assert rc == 0
    size = stripes * total * length
    raw = rng.integers(0, 256, size + 64, dtype=np.uint8)
    lo = 16 + shift

    def block(a):
        return a[lo:lo + size].reshape(stripes, total, length)

    def device(a):
        t = torch.from_numpy(a.copy()).cuda()
        return t, rsgpu.device_pointer_table(t.data_ptr() + lo, np.arange(stripes * total, dtype=np.uint64) * np.uint64(length))

    want = raw.copy()
    for i in check:
        ref = [np.ascontiguousarray(block(raw)[i, j]) for j in range(total)]
        O.classic_encode(mat, ref)
        block(want)[i] = np.stack(ref)
    buf, ptrs = device(raw)
    codec.prepare_batch("encode", ptrs, length).launch()
    torch.cuda.synchronize()
    got = buf.cpu().numpy()
    rest = np.setdiff1d(np.arange(stripes), check)
    assert np.array_equal(block(got)[rest, :k], block(raw)[rest, :k])
    block(want)[rest] = block(got)[rest]
    assert np.array_equal(got, want)

    bad = want.copy()
    block(bad)[1, total - 1, length - 1] ^= 1
    block(bad)[2, 0, 0] ^= 128
    buf, ptrs = device(bad)
    batch = codec.prepare_batch("verify", ptrs, length)
    batch.launch()
    assert list(np.flatnonzero(~batch.verify_result())) == [1, 2]

    pres = np.ones((stripes, total), np.uint8)
    for i in range(stripes):
        pres[i, rng.choice(total, size=min(m, i % m + 1), replace=False)] = 0
    erased = want.copy()
    for i, j in np.argwhere(pres == 0):
        block(erased)[i, j] = 0
    buf, ptrs = device(erased)
    codec.prepare_batch("reconstruct", ptrs, length, present=pres).launch()
    torch.cuda.synchronize()
    assert np.array_equal(buf.cpu().numpy(), want)

    # encode_single accumulates shard by shard; verify_with_buffer stores.
    buf, _ = device(raw)
    views = [buf[lo + j * length:lo + (j + 1) * length] for j in range(total)]
    for j in range(k):
        codec.encode_single(j, views)
    torch.cuda.synchronize()
    first = raw.copy()
    block(first)[0] = block(want)[0]
    assert np.array_equal(buf.cpu().numpy(), first)
    out = torch.zeros(m * length + 32, dtype=torch.uint8, device="cuda")
    parity = [out[3 + j * length:3 + (j + 1) * length] for j in range(m)]
    assert codec.verify_with_buffer(views, parity)
    got = out.cpu().numpy()
    assert np.array_equal(got[3:3 + m * length].reshape(m, length), block(want)[0, k:])
    assert not got[:3].any() and not got[3 + m * length:].any()
