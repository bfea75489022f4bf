"""GPU: classic operations of few inputs in mixed batches against the oracle, byte
for byte: each remainder of the lookup groups (fives, three, one more), jobs of
one and two inputs on pairs of tiles, shards that end before, on and after a tile
and a pair, more than four outputs, a damaged verify."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [0, 1, 2])
@pytest.mark.parametrize("k,m", [(1, 1), (1, 5), (2, 1), (2, 6), (3, 2), (4, 4), (6, 3), (7, 2), (9, 4), (12, 5)])
def test_every_remainder(k, m, tile):
    import torch

    import rsgpu

    rng = np.random.default_rng(10 * k + m)
    codec = rsgpu.ReedSolomon(k, m)
    rc, mat = O.build_matrix(k, m)
    assert rc == 0
    total, ops, bufs, want, flags = k + m, [], [], [], []
    for length in (16, 4080, 4096, 4112, 8176, 8192, 8208, 12304, 40963):
        word = [np.ascontiguousarray(s) for s in rng.integers(0, 256, (total, length), dtype=np.uint8)]
        O.classic_encode(mat, word)
        word = np.stack(word)
        pitch = (length + 15) // 16 * 16
        for op in ("encode", "verify", "damaged", "reconstruct"):
            src, present = np.zeros((total, pitch), np.uint8), np.ones(total, np.uint8)
            src[:, :length] = word
            out = src.copy()
            if op == "encode":
                src[k:, :length] = 0xA5
            elif op == "damaged":
                src[total - 1, length - 1] ^= 2
                out = src.copy()
            elif op == "reconstruct":
                present[rng.choice(total, size=m, replace=False)] = 0
                src[present == 0, :length] = 0xA5
            buf = torch.from_numpy(src).cuda()
            ops.append(dict(codec=codec, op="verify" if op == "damaged" else op, shard_len=length, present=present,
                            shards=[buf.data_ptr() + j * pitch for j in range(total)]))
            bufs.append(buf)
            want.append(out)
            flags.append(op != "damaged")
    batch = rsgpu.MixedBatch(ops, plans=[(0, tile)] * len(ops))
    batch.launch()
    assert list(batch.results()) == flags
    for i, (b, w) in enumerate(zip(bufs, want)):
        assert np.array_equal(b.cpu().numpy(), w), (ops[i]["op"], ops[i]["shard_len"])
