"""GPU: Leopard GF(2^16) work whose bit-sliced rows do not all fit their scratch
buffer, so that it runs in chunks of tiles, and rebuilds in a request server's own
buffer, byte for byte against the oracle: three and more chunks with borders
inside stripes and a shorter last one; a server batch in which a wider code
replaces the buffer after a narrower one's launch was built."""
import numpy as np
import pytest

import oracle as O
import test_gpu_server as server_tests

pytestmark = pytest.mark.gpu

K, M, LENGTH, STRIPES = 1024, 512, 39936, 11  # 19 and a half tiles a stripe: 220 in all


@pytest.fixture(scope="module")
def words():
    """Two codewords of the oracle, taken by the stripes in turn."""
    import torch

    rng = np.random.default_rng(1)
    out = rng.integers(0, 256, (2, K + M, LENGTH), dtype=np.uint8)
    for word in out:
        rc, par = O.leopard_encode(16, K, M, [word[j] for j in range(K)])
        assert rc == 0
        word[K:] = np.stack(par)
    return torch.from_numpy(out).cuda()[torch.arange(STRIPES, device="cuda") % 2].contiguous()


def _batch(op, buf, present=None):
    import rsgpu

    codec = rsgpu.ReedSolomon(K, M, rsgpu.CodecOptions(codec_family="leopard_gf16"))
    ptrs = rsgpu.device_pointer_table(buf.data_ptr(),
                                      np.arange(STRIPES * (K + M), dtype=np.uint64) * np.uint64(LENGTH))
    return codec.prepare_batch(op, ptrs, LENGTH, present=present)


def test_encode_and_verify_in_three_chunks(words):
    import torch

    buf = words.clone()
    buf[:, K:] = 0xA5
    batch = _batch("encode", buf)
    assert batch.kernel_count() == 3 * 3  # 74, 74 and 72 tiles
    for _ in range(2):  # the second launch works in the rows the first one left
        batch.launch()
        torch.cuda.synchronize()
        assert torch.equal(buf, words)
    batch = _batch("verify", buf)
    batch.launch()
    assert batch.verify_result().all()
    hits = [(3, K + M - 1, 14 * 2048 - 1), (3, K, 14 * 2048), (7, 5, 8 * 2048), (STRIPES - 1, K + M - 1, LENGTH - 1)]
    for stripe, shard, byte in hits:  # either side of a border, and the very end
        batch = _batch("verify", buf)
        buf[stripe, shard, byte] ^= 64
        batch.launch()
        assert list(np.flatnonzero(~batch.verify_result())) == [stripe]
        buf[stripe, shard, byte] ^= 64


def test_rebuild_in_six_chunks(words):
    import torch

    rng = np.random.default_rng(2)
    present = np.ones((STRIPES, K + M), np.uint8)
    for i, row in enumerate(present):
        row[rng.choice(K + M, size=M if i % 2 else 1 + i, replace=False)] = 0
    buf = words.clone()
    buf[torch.from_numpy(present == 0).cuda()] = 0xA5
    batch = _batch("reconstruct", buf, present)
    assert batch.kernel_count() == 6 * 3  # 37 tiles, the last 35
    batch.launch()
    torch.cuda.synchronize()
    assert torch.equal(buf, words)


def test_server_rebuilds_in_a_buffer_that_moves():
    import torch

    import rsgpu

    geoms = [("leopard_gf16", 512, 256 + i) for i in range(-3, 1)] + [("leopard_gf16", 300, 400), ("leopard_gf16", 3500, 600)]
    codecs = {g: rsgpu.ReedSolomon(g[1], g[2], rsgpu.CodecOptions(codec_family=g[0])) for g in geoms}
    rng = np.random.default_rng(8)
    reqs = []
    for i, g in enumerate(geoms + geoms[:3]):
        k, m = g[1:]
        present = np.ones(k + m, np.uint8)
        present[rng.choice(k + m, size=m if i % 2 else 7, replace=False)] = 0
        length = (1024, 2112, 4096)[i % 3]
        reqs.append(dict(geom=g, op="reconstruct", data=rng.integers(0, 256, (k + m, length), dtype=np.uint8),
                         present=present, goal="data" if i % 4 == 3 else "all", len=length))
    server = rsgpu.Server(streams=1, max_batch=16)
    got, _, _ = server_tests.run(rsgpu, server, codecs, reqs, one_at_a_time=False, device=torch)
    again, _, _ = server_tests.run(rsgpu, server, codecs, reqs, one_at_a_time=False, device=torch)
    server.close()
    for i, r in enumerate(reqs):
        want, _ = server_tests.oracle_apply(r["geom"], codecs[r["geom"]], r["op"], r["data"], r["present"], r["goal"])
        assert np.array_equal(got[i], want), (i, r["geom"])
        assert np.array_equal(again[i], want), (i, r["geom"])
