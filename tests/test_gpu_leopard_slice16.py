"""GPU: the bit-sliced Leopard GF(2^16) kernels against the oracle, byte for
byte, at the edges of their split and dispatch: the fewest lanes they take and
the first code past the most, odd and even level sizes, one and several data
groups, shards of half a tile, one tile, a tile and a block, patterns of their
own per stripe, and launches under stream capture (which run the register-stage
kernels)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _setup(k, m, length, stripes, seed):
    import torch

    import rsgpu

    rng = np.random.default_rng(seed)
    codec = rsgpu.ReedSolomon(k, m, rsgpu.CodecOptions(codec_family="leopard_gf16"))
    total = k + m
    host = rng.integers(0, 256, (stripes, total, length), dtype=np.uint8)  # not codewords
    buf = torch.from_numpy(host.copy()).cuda()
    ptrs = rsgpu.device_pointer_table(buf.data_ptr(), np.arange(stripes * total, dtype=np.uint64) * np.uint64(length))
    return torch, codec, rng, host, buf, ptrs


@pytest.mark.parametrize("k,m,length,stripes", [
    (300, 256, 1024, 2),     # encode from 256 lanes; half a tile
    (256, 256, 2048, 1),     # one data group, exactly one tile
    (700, 300, 2112, 2),     # 512-lane encode, two groups, the second partial
    (1100, 512, 4096, 1),    # three groups
    (2048, 1024, 1088, 1),   # 4096-lane decode
    (600, 1024, 1024, 1),    # fewer data than parity lanes
    (200, 60, 2112, 2),      # 64 lanes, four groups
    (30, 33, 2048, 2),       # 64 lanes, one partial group
    (200, 100, 4096, 1),     # 128 lanes
    (250, 100, 1024, 2),     # 128 lanes, shards too short: register-stage kernels
    (300, 20, 2048, 2),      # 32 lanes: register-stage kernels
])
def test_encode_and_verify(k, m, length, stripes):
    torch, codec, rng, host, buf, ptrs = _setup(k, m, length, stripes, k + m)
    want = host.copy()
    for i in range(stripes):
        rc, par = O.leopard_encode(16, k, m, [host[i, j] for j in range(k)])
        assert rc == 0
        want[i, k:] = np.stack(par)
    codec.prepare_batch("encode", ptrs, length).launch()
    torch.cuda.synchronize()
    assert np.array_equal(buf.cpu().numpy(), want)
    batch = codec.prepare_batch("verify", ptrs, length)
    batch.launch()
    assert batch.verify_result().all()
    buf[stripes - 1, k + m - 1, length - 1] ^= 1
    batch.launch()
    assert list(batch.verify_result()) == [True] * (stripes - 1) + [False]


@pytest.mark.parametrize("k,m,length,stripes", [
    (64, 32, 1024, 3),       # 128 lanes
    (100, 60, 2112, 3),      # 256 lanes: even levels
    (65, 33, 3136, 2),       # padding lanes between parity and data
    (300, 100, 2048, 2),     # 512 lanes
    (900, 90, 1024, 1),      # 1024 lanes
    (1024, 512, 4160, 1),    # 2048 lanes
    (2048, 1024, 1088, 1),   # 4096 lanes: 64-row levels
    (40, 16, 2048, 2),       # 64 lanes: 4-row low levels
    (20, 33, 1088, 2),       # the fewest lanes, more parity than data
    (20, 12, 2048, 2),       # 32 lanes: register-stage kernels
    (3500, 600, 1024, 1),    # 8192 lanes: register-stage kernels
])
def test_reconstruct(k, m, length, stripes):
    torch, codec, rng, host, buf, ptrs = _setup(k, m, length, stripes, 7 * k + m)
    total = k + m
    pres = np.ones((stripes, total), np.uint8)
    for i in range(stripes):
        lost = m if i == 0 else 1 + i
        pres[i, rng.choice(total, size=lost, replace=False)] = 0
    codec.prepare_batch("reconstruct", ptrs, length, present=pres).launch()
    torch.cuda.synchronize()
    got = buf.cpu().numpy()
    for i in range(stripes):
        ref = [host[i, j].copy() if pres[i, j] else np.zeros(length, np.uint8) for j in range(total)]
        assert O.leopard_reconstruct(16, k, m, ref, pres[i].tolist()) == 0
        assert np.array_equal(got[i], np.stack(ref)), i


def test_launch_under_capture_gives_the_same_bytes():
    k, m, length, stripes = 300, 256, 2048, 2
    torch, codec, rng, host, buf, ptrs = _setup(k, m, length, stripes, 3)
    batch = codec.prepare_batch("encode", ptrs, length)
    batch.launch()
    torch.cuda.synchronize()
    want = buf.clone()
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        batch.launch()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            batch.launch()
    buf[:, k:] = 0
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(buf, want)
