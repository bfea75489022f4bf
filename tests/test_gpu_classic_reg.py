"""GPU: the classic kernel with its tables in registers against the oracle,
byte for byte: every input count it is built for and the first one past it
(1 to 21), shard lengths around its tiles (2, 4 and 8 KiB) and its 16-byte
tails, one table for all stripes and one per stripe."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = (16, 2032, 2064, 4111, 8208, 16399)


@pytest.mark.parametrize("k", list(range(1, 22)))
def test_tables_in_registers(k):
    import torch

    import rsgpu

    rng = np.random.default_rng(k)
    m = 1 + (k - 1) % 4
    total, stripes = k + m, 5
    codec = rsgpu.ReedSolomon(k, m)
    rc, mat = O.build_matrix(k, m)
    assert rc == 0
    for length in (LENGTHS[k % 6], LENGTHS[(k + 3) % 6]):
        pitch = (length + 15) // 16 * 16
        host = rng.integers(0, 256, (stripes, total, pitch), dtype=np.uint8)
        host[:, :, length:] = 0x5A  # padding: must stay
        ptrs = None

        def upload(a):
            nonlocal ptrs
            t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
            ptrs = rsgpu.device_pointer_table(t.data_ptr(),
                                              np.arange(stripes * total, dtype=np.uint64) * np.uint64(pitch))
            return t

        want = host.copy()
        for i in range(stripes):
            ref = [np.ascontiguousarray(want[i, j, :length]) for j in range(total)]
            O.classic_encode(mat, ref)
            for j in range(total):
                want[i, j, :length] = ref[j]
        buf = upload(host)
        codec.prepare_batch("encode", ptrs, length).launch()
        torch.cuda.synchronize()
        assert np.array_equal(buf.cpu().numpy(), want), (length, "encode")

        bad = want.copy()
        bad[2, total - 1, length - 1] ^= 8
        bad[4, 0, 0] ^= 1
        buf = upload(bad)
        batch = codec.prepare_batch("verify", ptrs, length)
        batch.launch()
        assert list(batch.verify_result()) == [True, True, False, True, False], (length, "verify")

        pres = np.ones((stripes, total), np.uint8)
        for i in range(stripes):  # a pattern of its own per stripe, one stripe complete
            if i != 3:
                pres[i, rng.choice(total, size=min(m, 1 + i % m), replace=False)] = 0
        erased = want.copy()
        for i, j in np.argwhere(pres == 0):
            erased[i, j, :length] = 0
        buf = upload(erased)
        codec.prepare_batch("reconstruct", ptrs, length, present=pres).launch()
        torch.cuda.synchronize()
        assert np.array_equal(buf.cpu().numpy(), want), (length, "reconstruct")
