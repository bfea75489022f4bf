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


@pytest.mark.parametrize("shift,step,count,bound", [
    (0, 2048, 41, 3 << 30),    # bit-sliced rows: 6 MiB more a step; the library's pool keeps 2 GiB of freed memory
    (4, 128, 148, 512 << 20),  # shards off 16 bytes: work rows of one more CTA a step
])
def test_rebuilds_of_rising_sizes_hold_a_bounded_amount(shift, step, count, bound):
    import torch

    import rsgpu

    k, m = 1024, 512
    codec = _codec(k, m)
    buf = torch.zeros((k + m) * step * (count + 1) + 16, dtype=torch.uint8, device="cuda")
    pres = np.ones((1, k + m), np.uint8)
    pres[0, :8] = 0
    free = None
    for i in range(count):
        length = step * (i + 1)
        ptrs = rsgpu.device_pointer_table(buf.data_ptr() + shift,
                                          np.arange(k + m, dtype=np.uint64) * np.uint64(length))
        codec.prepare_batch("reconstruct", ptrs, length, present=pres).launch()
        torch.cuda.synchronize()
        if free is None:
            free = torch.cuda.mem_get_info()[0]
    assert free - torch.cuda.mem_get_info()[0] < bound


_NO_ROOM = """
import numpy as np, torch, rsgpu
k, m, length, stripes = 512, 256, 16384, 16
codec = rsgpu.ReedSolomon(k, m, rsgpu.CodecOptions(codec_family="leopard_gf16"))
want = torch.randint(0, 256, (stripes, k + m, length), dtype=torch.uint8, device="cuda")
for stripe in range(stripes):  # one by one, in little scratch
    codec.encode_batch(want[stripe:stripe + 1])
buf = want.clone()
offsets = np.arange(stripes * (k + m), dtype=np.uint64) * np.uint64(length)
pres = np.ones((stripes, k + m), np.uint8)
pres[:, :m] = 0
def rebuild(n):
    batch = codec.prepare_batch("reconstruct", rsgpu.device_pointer_table(buf.data_ptr(), offsets[:n * (k + m)]), length,
                                present=pres[:n])
    buf[:n, :m] = 0
    batch.launch()
    torch.cuda.synchronize()
    assert torch.equal(buf, want)
    return batch
# Every kernel of the path loads while there is memory for its code.
odd = torch.zeros((k + m) * 64 + 16, dtype=torch.uint8, device="cuda")
codec.prepare_batch("reconstruct", rsgpu.device_pointer_table(odd.data_ptr() + 4, np.arange(k + m, dtype=np.uint64) *
                    np.uint64(64)), 64, present=pres[:1]).launch()
small = rebuild(2)
assert small.kernel_count() == 3
torch.cuda.synchronize()
full = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
for n in (stripes, 2, stripes):
    assert rebuild(n).kernel_count() == (3 if n == 2 else 1), n
buf[:2, :m] = 0
small.launch()
torch.cuda.synchronize()
assert torch.equal(buf, want)
print("done")
"""


def test_no_room_for_larger_rows_leaves_the_smaller_ones_in_use():
    """In a process of its own: the library's pool holds nothing else there."""
    import os
    import subprocess
    import sys

    import rsgpu

    env = dict(os.environ, PYTHONPATH=os.path.dirname(os.path.dirname(rsgpu.__file__)))
    done = subprocess.run([sys.executable, "-c", _NO_ROOM], env=env, capture_output=True, text=True, timeout=300)
    assert done.stdout.strip().endswith("done"), done.stderr[-2000:]


@pytest.mark.parametrize("op,prepared", [("encode", True), ("verify", True), ("reconstruct", True),
                                         ("encode", False), ("reconstruct", False)])
def test_launches_of_one_codec_do_not_wait_for_another_stream(op, prepared):
    """A small launch finishes while one of the same codec is held up behind
    other work on its own stream (at most 1 second of it)."""
    import torch

    k, m, length, stripes = 200, 60, 4096, 2
    codec = _codec(k, m)
    want = torch.from_numpy(_codewords(k, m, length, stripes, 9)).cuda()
    pres = np.ones((stripes, k + m), np.uint8)
    pres[:, 3:3 + m] = 0
    streams = [torch.cuda.Stream() for _ in range(2)]
    bufs = [want.clone() for _ in streams]
    batches = [codec.prepare_batch(op, _pointers(b), length, present=pres if op == "reconstruct" else None) for b in bufs]

    def wipe(buf):
        if op == "encode":
            buf[:, k:] = 0
        elif op == "reconstruct":
            buf[:, 3:3 + m] = 0

    def launch(i):
        with torch.cuda.stream(streams[i]):
            if prepared:
                batches[i].launch()
            elif op == "encode":
                codec.encode_batch(bufs[i])
            else:
                codec.reconstruct_batch(bufs[i], pres)

    for i in range(2):  # every kernel is loaded
        launch(i)
    torch.cuda.synchronize()
    for b in bufs:
        wipe(b)
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(500_000_000)  # a quarter of a second
        held = torch.cuda.Event()
        launch(0)
        held.record()
    launch(1)
    streams[1].synchronize()
    assert not held.query()
    assert torch.equal(bufs[1], want)
    torch.cuda.synchronize()
    assert torch.equal(bufs[0], want)
    if op == "verify":
        for i in range(2):
            with torch.cuda.stream(streams[i]):
                assert batches[i].verify_result().all()


def test_codec_destroyed_while_another_device_is_current():
    """Its buffers go back only behind its last kernels."""
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices")
    k, m, length, stripes = 512, 256, 16384, 8
    want = torch.from_numpy(_codewords(k, m, length, 2, 3)).cuda().repeat(stripes // 2, 1, 1).contiguous()
    pres = np.ones((stripes, k + m), np.uint8)
    pres[:, :m] = 0
    bufs = [want.clone() for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    for b in bufs:
        b[:, :m] = 0
    torch.cuda.synchronize()
    for i, b in enumerate(bufs):  # the second would work in the first one's rows
        codec = _codec(k, m)
        with torch.cuda.stream(streams[i]):
            if i == 0:
                torch.cuda._sleep(500_000_000)
            codec.reconstruct_batch(b, pres)
        with torch.cuda.device(1):
            del codec
    torch.cuda.synchronize()
    for b in bufs:
        assert torch.equal(b, want)
