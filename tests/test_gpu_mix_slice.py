"""GPU: mixed batches whose Leopard GF(2^8) operations go in bit-sliced launches
beside the persistent kernel (planners "table" and "model"), byte for byte
against the oracle: a codec with enough columns and one without, both rebuild
goals, few and many lost shards, a damaged verify, a shard that is not 16-byte
aligned (stays in the persistent kernel), as a graph and as plain launches."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("planner", ["table", "model"])
def test_sliced_ops_match_oracle(planner, graph):
    import torch

    import rsgpu

    rng = np.random.default_rng(7)
    codecs = {g: rsgpu.ReedSolomon(*g, rsgpu.CodecOptions(codec_family="leopard_gf8")) for g in [(32, 16), (10, 5)]}
    # (geometry, op, length, lost, goal, address offset)
    specs = [((32, 16), "encode", 131072, 0, "all", 0), ((32, 16), "encode", 65600, 0, "all", 0),
             ((32, 16), "encode", 65536, 0, "all", 0), ((32, 16), "encode", 64, 0, "all", 0),
             ((32, 16), "encode", 16384, 0, "all", 8),
             ((32, 16), "reconstruct", 131072, 16, "all", 0), ((32, 16), "reconstruct", 131136, 12, "data", 0),
             ((32, 16), "reconstruct", 65536, 1, "all", 0), ((32, 16), "reconstruct", 65536, 0, "all", 0),
             ((32, 16), "verify", 131072, 0, "all", 0), ((32, 16), "verify", 131136, 0, "bad", 0),
             ((32, 16), "verify", 64, 0, "bad", 0),
             ((10, 5), "encode", 4096, 0, "all", 0), ((10, 5), "reconstruct", 4096, 5, "all", 0)]
    ops, bufs, want, flags = [], [], [], []
    for (k, m), op, length, lost, goal, shift in specs:
        total = k + m
        data = rng.integers(0, 256, (total, length), dtype=np.uint8)
        rc, par = O.leopard_encode(8, k, m, [data[j] for j in range(k)])
        assert rc == 0
        code = np.concatenate([data[:k], np.stack(par)])
        present = np.ones(total, np.uint8)
        if op == "encode":
            src, out = data, code
        else:
            src = code.copy()
            present[rng.choice(total, size=lost, replace=False)] = 0
            if goal == "bad":
                src[total - 1, length - 1] ^= 128
            src[present == 0] = 0xA5
            out = src.copy()
            rebuilt = (present == 0) & ((np.arange(total) < k) | (goal == "all"))
            out[rebuilt] = code[rebuilt]
        buf = torch.empty(total * length + 16, dtype=torch.uint8, device="cuda")
        assert buf.data_ptr() % 16 == 0
        buf[shift:shift + total * length] = torch.from_numpy(src.reshape(-1)).cuda()
        ops.append(dict(codec=codecs[(k, m)], op=op, shard_len=length, present=present,
                        goal="data" if goal == "data" else "all",
                        shards=[buf.data_ptr() + shift + j * length for j in range(total)]))
        bufs.append(buf[shift:shift + total * length])
        want.append(out)
        flags.append(goal != "bad")
    batch = rsgpu.MixedBatch(ops, planner=planner, graph=graph)
    for again in range(2):  # the verify flags are cleared for each launch
        batch.launch()
        assert list(batch.results()) == flags
        for i, (b, w) in enumerate(zip(bufs, want)):
            assert np.array_equal(b.cpu().numpy().reshape(w.shape), w), (again, specs[i])
