"""GPU: verifies of one to five inputs against the oracle on either side of the
line between the two K1 tiles (classic_rules.hpp), shards of several tiles and a
remainder: good stripes, and single bytes damaged in the first and the last
column of a data and of a parity shard."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,m", [(1, 1), (1, 4), (2, 1), (2, 2), (3, 1), (4, 1), (4, 4), (5, 2)])
@pytest.mark.parametrize("length,stripes", [(16384, 256), (16368, 257), (16400, 256), (16384, 255), (1 << 20, 5),
                                            (4112, 3)])
def test_damaged_stripes_are_found(k, m, length, stripes):
    import torch

    import rsgpu

    rng = np.random.default_rng(100 * k + m)
    total, distinct = k + m, 2
    codec = rsgpu.ReedSolomon(k, m)
    rc, mat = O.build_matrix(k, m)
    assert rc == 0
    words = rng.integers(0, 256, (distinct, total, length), dtype=np.uint8)
    for word in words:
        shards = [np.ascontiguousarray(s) for s in word]
        O.classic_encode(mat, shards)
        word[:] = np.stack(shards)
    buf = torch.from_numpy(words).cuda()[torch.arange(stripes, device="cuda") % distinct].contiguous()
    ptrs = rsgpu.device_pointer_table(buf.data_ptr(), np.arange(stripes * total, dtype=np.uint64) * np.uint64(length))
    batch = codec.prepare_batch("verify", ptrs, length)
    batch.launch()
    assert batch.verify_result().all()
    hits = [(0, 0, 0), (1, k - 1, length - 1), (stripes // 2 + 1, k, 0), (stripes - 1, total - 1, length - 1)]
    for stripe, shard, byte in hits:
        buf[stripe, shard, byte] ^= 16
    batch.launch()
    assert list(np.flatnonzero(~batch.verify_result())) == sorted({h[0] for h in hits})
