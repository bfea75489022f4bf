"""GPU: the bit-sliced Leopard GF(2^8) kernels against the oracle, byte for
byte, at the edges of their tiles and dispatch: one radix-2 layer up to 256
lanes (28-thread rows), odd and even log2 sizes, a single and several data
groups, shard lengths of one 64-byte block, one tile, one tile and a block, and
16-byte-misaligned pointers (which take the register-stage kernels)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rs():
    import rsgpu

    return rsgpu


def _run(rs, k, m, length, stripes, seed, shift=0):
    import torch

    rng = np.random.default_rng(seed)
    codec = rs.ReedSolomon(k, m, rs.CodecOptions(codec_family="leopard_gf8"))
    total = k + m
    pitch = (length + 63) // 64 * 64 + 64
    buf = torch.zeros(stripes * total * pitch + 64, dtype=torch.uint8, device="cuda")
    base = buf.data_ptr() + shift
    ptrs = np.uint64(base) + np.arange(stripes * total, dtype=np.uint64) * np.uint64(pitch)
    host = rng.integers(0, 256, (stripes, total, length), dtype=np.uint8)  # not codewords

    def upload(a):
        h = np.zeros(buf.numel(), np.uint8)
        for i in range(stripes):
            for j in range(total):
                o = shift + (i * total + j) * pitch
                h[o:o + length] = a[i, j]
        buf.copy_(torch.from_numpy(h))

    def download():
        h = buf.cpu().numpy()
        return np.stack([np.stack([h[shift + (i * total + j) * pitch:][:length] for j in range(total)])
                         for i in range(stripes)]), h

    # encode
    upload(host)
    codec.prepare_batch("encode", ptrs, length).launch()
    torch.cuda.synchronize()
    got, raw = download()
    want = host.copy()
    for i in range(stripes):
        rc, par = O.leopard_encode(8, k, m, [host[i, j] for j in range(k)])
        assert rc == 0
        want[i, k:] = np.stack(par)
    assert np.array_equal(got, want)
    # verify: one stripe damaged in its last byte
    batch = codec.prepare_batch("verify", ptrs, length)
    batch.launch()
    assert batch.verify_result().all()
    bad = want.copy()
    bad[-1, -1, -1] ^= 1
    upload(bad)
    batch.launch()
    assert list(batch.verify_result()) == [True] * (stripes - 1) + [False]
    # reconstruct from arbitrary shards, a pattern of its own per stripe
    pres = np.ones((stripes, total), np.uint8)
    for i in range(stripes):
        pres[i, rng.choice(total, size=min(m, 1 + i % m), replace=False)] = 0
    upload(host)
    codec.prepare_batch("reconstruct", ptrs, length, present=pres).launch()
    torch.cuda.synchronize()
    got, raw = download()
    for i in range(stripes):
        ref = [host[i, j].copy() if pres[i, j] else np.zeros(length, np.uint8) for j in range(total)]
        assert O.leopard_reconstruct(8, k, m, ref, pres[i].tolist()) == 0
        assert np.array_equal(got[i], np.stack(ref)), (i, np.flatnonzero(pres[i] == 0))
    # nothing outside the shards was written
    mask = np.ones(raw.size, bool)
    for i in range(stripes * total):
        mask[shift + i * pitch:shift + i * pitch + length] = False
    assert not raw[mask].any()


@pytest.mark.parametrize("k,m,length,stripes", [
    (16, 16, 64, 3),        # one block; one data group, decode of 32 lanes
    (32, 16, 1024, 2),      # exactly one tile
    (33, 16, 1088, 2),      # a tile and a block; a data group of one shard
    (20, 17, 960, 2),       # m = 32: odd log2 size
    (100, 30, 2048, 2),     # four data groups, 256-lane decode (28-thread rows)
    (128, 64, 896, 2),      # exactly one 28-thread tile
    (128, 64, 960, 1),
    (5, 128, 1984, 1),      # 128-lane encode of one group, 256-lane decode
    (200, 32, 128, 2),      # seven data groups
    (128, 128, 64, 1),      # the widest code
    (9, 3, 4096, 9),        # 16-lane decode
])
def test_slice_kernels_match_oracle(rs, k, m, length, stripes):
    _run(rs, k, m, length, stripes, seed=k * 1000 + m)


@pytest.mark.parametrize("k,m,length,stripes", [
    (1, 1, 64 * 8192, 1), (3, 1, 64 * 8192, 1),    # no layer; radix-2 decode
    (2, 2, 1 << 20, 2), (4, 2, 1 << 20, 2),        # one radix-2 layer
    (6, 3, 1 << 20, 2), (8, 8, 1 << 20, 2),
])
def test_slice_kernels_small_codes_on_long_shards(rs, k, m, length, stripes):
    _run(rs, k, m, length, max(stripes, (2 << 20) // length), seed=k * 1000 + m)


def test_misaligned_shards_keep_their_bytes(rs):
    _run(rs, 32, 16, 1088, 2, seed=5, shift=4)
