"""GPU: misaligned classic jobs on enough columns for the word kernel
(classic_rules.hpp), with the checks of test_gpu_classic_unaligned.py: lengths
from the shortest it takes to several tiles, every remainder of a word and of a
tile's last row of threads, one to twenty outputs; and the launch that is just too
small for it."""
import pytest

import test_gpu_classic_unaligned as unaligned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,m,length", [(1, 1, 1645), (3, 2, 1649), (4, 4, 2051), (5, 3, 3079), (10, 4, 4103),
                                        (12, 4, 4107), (16, 4, 8203), (21, 4, 8211), (10, 4, 100003)])
@pytest.mark.parametrize("shift", [0, 5])
def test_up_to_four_outputs(k, m, length, shift):
    unaligned.test_packed_odd_shards(k, m, length, shift, 704 << 10)


@pytest.mark.parametrize("k,m,length", [(7, 8, 2573), (9, 5, 4101), (30, 9, 12305), (50, 20, 100003)])
def test_more_outputs(k, m, length):
    unaligned.test_packed_odd_shards(k, m, length, 3, 1 << 20)


@pytest.mark.parametrize("k,m,length,stripes", [(10, 4, 4103, 175), (6, 3, 720897 - 2, 1), (9, 5, 4101, 255)])
def test_one_stripe_less(k, m, length, stripes):
    unaligned.test_packed_odd_shards(k, m, length, 1, (stripes - 1) * length)


@pytest.mark.parametrize("k,m", [(4, 2), (10, 4), (7, 8)])
def test_one_long_stripe(k, m):
    """The storing verify by words, the adding calls of one shard by bytes."""
    unaligned.test_packed_odd_shards(k, m, 1100003, 2, 0)


@pytest.mark.parametrize("k,m,changed,length", [(10, 4, 10, 3355451), (10, 4, 5, 3355451), (12, 4, 5, 6710891),
                                                (9, 5, 7, 4793499), (9, 5, 4, 8388611)])
@pytest.mark.parametrize("shift", [1, 6])
def test_update(k, m, changed, length, shift):
    """Adding calls on either side of their line: the new parity is the encode of
    the new data, and nothing around the shards is written."""
    import numpy as np
    import torch

    import oracle as O
    import rsgpu

    rng = np.random.default_rng(k + changed)
    rc, mat = O.build_matrix(k, m)
    assert rc == 0
    pitch = length + 13
    host = rng.integers(0, 256, (k + m) * pitch + 64, dtype=np.uint8)
    words = [np.ascontiguousarray(host[shift + j * pitch:][:length]) for j in range(k + m)]
    O.classic_encode(mat, words)
    for j in range(k, k + m):
        host[shift + j * pitch:][:length] = words[j]
    new = [rng.integers(0, 256, length, dtype=np.uint8) for _ in range(changed)]
    fresh = [torch.from_numpy(np.concatenate([np.zeros(3, np.uint8), x])).cuda()[3:] for x in new]
    buf = torch.from_numpy(host).cuda()
    views = [buf[shift + j * pitch:][:length] for j in range(k + m)]
    rsgpu.ReedSolomon(k, m).update(views[:k], fresh + [None] * (k - changed), views[k:])
    torch.cuda.synchronize()
    words[:changed] = new
    O.classic_encode(mat, words)
    want = host.copy()
    for j in range(k, k + m):
        want[shift + j * pitch:][:length] = words[j]
    assert np.array_equal(buf.cpu().numpy(), want)
