"""GPU: Leopard encodes and verifies on either side of the lines of leo_rules.hpp
against the oracle, byte for byte: the least work that the bit-sliced kernels
take, and one 64-byte block or one stripe less."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _encode_and_verify(bits, k, m, length, stripes):
    import torch

    import rsgpu

    rng = np.random.default_rng(1000 * k + m)
    codec = rsgpu.ReedSolomon(k, m, rsgpu.CodecOptions(codec_family="leopard_gf%d" % bits))
    total, distinct = k + m, min(stripes, 3)
    words = rng.integers(0, 256, (distinct, total, length), dtype=np.uint8)
    for word in words:
        rc, par = O.leopard_encode(bits, k, m, [word[j] for j in range(k)])
        assert rc == 0
        word[k:] = np.stack(par)
    want = torch.from_numpy(words).cuda()[torch.arange(stripes, device="cuda") % distinct].contiguous()
    buf = want.clone()
    buf[:, k:] = 0xA5
    ptrs = rsgpu.device_pointer_table(buf.data_ptr(), np.arange(stripes * total, dtype=np.uint64) * np.uint64(length))
    encode = codec.prepare_batch("encode", ptrs, length)
    encode.launch()
    torch.cuda.synchronize()
    assert torch.equal(buf, want)
    verify = codec.prepare_batch("verify", ptrs, length)
    verify.launch()
    assert verify.verify_result().all()
    buf[stripes - 1, total - 1, length - 1] ^= 1
    buf[0, 0, 0] ^= 128
    verify.launch()
    assert list(np.flatnonzero(~verify.verify_result())) == sorted({0, stripes - 1})
    return encode


@pytest.mark.parametrize("k,m,length,stripes", [
    (16, 16, 524288, 1), (9, 9, 2048, 256), (60, 16, 1024, 511), (64, 9, 524288 - 64, 1),  # 16 lanes: 512 KiB
    (65, 16, 524288, 1),                                                                  # too many data groups
    (32, 16, 64, 2), (33, 16, 1088, 2),                                                   # verify from two groups
    (40, 20, 512, 3), (40, 20, 448, 3), (32, 17, 64, 2), (224, 32, 576, 2),               # 32 lanes: 512-byte shards
    (128, 64, 512, 112), (128, 64, 960, 60), (128, 64, 57344 - 64, 1), (60, 64, 512, 2),  # 64 lanes: 56 KiB
    (100, 100, 57344, 1), (128, 128, 960, 60), (5, 128, 57344 - 64, 1), (100, 70, 448, 150),  # 128 lanes
])
def test_gf8(k, m, length, stripes):
    _encode_and_verify(8, k, m, length, stripes)


@pytest.mark.parametrize("k,m,length,stripes,sliced", [
    (30, 33, 2048, 75, True), (64, 64, 2048, 74, False),      # 64 lanes, one data group: 148 KiB
    (120, 64, 4096, 19, True), (190, 64, 2048, 37, False),    # two and three: 74 KiB
    (200, 60, 2048, 3, True), (193, 50, 4160, 2, True),       # four; the last tile of three a block
    (200, 60, 2112, 2, False), (200, 60, 1984, 2, False),     # half-filled tiles, short shards
    (100, 100, 4096, 19, True), (128, 70, 2048, 37, False),   # 128 lanes: 74 KiB
    (200, 100, 3072, 13, True), (200, 100, 2048, 18, False),  # two groups: 37 KiB, tiles filled to three quarters
    (512, 128, 2048, 1, True), (300, 128, 2048, 18, False),
    (256, 256, 1088, 18, True), (60, 200, 1024, 18, False),   # 256 lanes: 18.5 KiB
    (300, 256, 1024, 8, True), (300, 256, 1024, 9, False),    # two groups: up to 8 tiles too
    (100, 500, 1024, 8, True), (600, 500, 1088, 9, False), (600, 300, 1088, 18, True),  # 512 lanes
    (100, 1000, 1024, 9, True),
])
def test_gf16(k, m, length, stripes, sliced):
    batch = _encode_and_verify(16, k, m, length, stripes)
    assert batch.kernel_count() == (3 if sliced else 1)
