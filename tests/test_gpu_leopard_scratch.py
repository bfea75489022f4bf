"""GPU: the device memory that Leopard GF(2^16) launches of one codec work in.

A rebuild of 2048 lanes and more that is launched under stream capture keeps
its work rows in a buffer of the codec, whose address stays in the graph; its
replays may run while the same codec encodes on another stream."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _codec(k, m):
    import rsgpu

    return rsgpu.ReedSolomon(k, m, rsgpu.CodecOptions(codec_family="leopard_gf16"))


def _pointers(buf):
    import rsgpu

    stripes, total, length = buf.shape
    return rsgpu.device_pointer_table(buf.data_ptr(), np.arange(stripes * total, dtype=np.uint64) * np.uint64(length))


def _codewords(k, m, length, distinct, seed):
    """`distinct` codewords of the oracle, shape (distinct, k + m, length)."""
    rng = np.random.default_rng(seed)
    out = rng.integers(0, 256, (distinct, k + m, length), dtype=np.uint8)
    for word in out:
        rc, par = O.leopard_encode(16, k, m, [word[j] for j in range(k)])
        assert rc == 0
        word[k:] = np.stack(par)
    return out


def test_replayed_rebuild_beside_encodes_of_the_same_codec():
    import torch

    k, m, length, stripes = 1024, 512, 4096, 16
    codec = _codec(k, m)
    words = torch.from_numpy(_codewords(k, m, length, 2, 5)).cuda()
    want = words.repeat(stripes // 2, 1, 1).contiguous()
    rebuilt, encoded = want.clone(), want.clone()
    rng = np.random.default_rng(6)
    pres = np.ones((stripes, k + m), np.uint8)
    for row in pres:
        row[rng.choice(k + m, size=m, replace=False)] = 0
    lost = torch.from_numpy(pres == 0).cuda()
    rebuild = codec.prepare_batch("reconstruct", _pointers(rebuilt), length, present=pres)
    encode = codec.prepare_batch("encode", _pointers(encoded), length)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    rebuild.launch()
    encode.launch()
    torch.cuda.synchronize()
    with torch.cuda.stream(first):
        with torch.cuda.graph(graph, stream=first):
            rebuild.launch()
    for _ in range(20):
        rebuilt[lost] = 0xA5
        encoded[:, k:] = 0
        torch.cuda.synchronize()
        with torch.cuda.stream(first):
            graph.replay()
        for _ in range(4):
            encode.launch(stream=second.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(rebuilt, want)
        assert torch.equal(encoded, want)


@pytest.mark.parametrize("k,m", [(1024, 512), (300, 100)])  # work rows in the codec's buffer, in shared memory
def test_rebuild_captured_after_one_plain_launch(k, m):
    """The captured kernels are not the ones the plain launch ran."""
    import torch

    length = 2048
    codec = _codec(k, m)
    want = torch.from_numpy(_codewords(k, m, length, 2, k)).cuda()
    buf = want.clone()
    pres = np.ones((2, k + m), np.uint8)
    pres[0, ::3] = 0
    pres[0, :m // 2] = 1
    pres[0, np.flatnonzero(pres[0] == 0)[m:]] = 1
    pres[1, k:] = 0
    buf[torch.from_numpy(pres == 0).cuda()] = 0
    batch = codec.prepare_batch("reconstruct", _pointers(buf), length, present=pres)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        batch.launch()
        torch.cuda.synchronize()
        assert torch.equal(buf, want)
        with torch.cuda.graph(graph, stream=stream):
            batch.launch()
    buf[torch.from_numpy(pres == 0).cuda()] = 0
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(buf, want)
