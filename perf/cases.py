"""Performance cases of the erasure-coding path: what a user of this library
has it do, through its public Python API, over the range of sizes it is used at.

``listed()`` names the standing cases, ``draw(rng)`` gives more of the same
ranges, ``prepare`` makes what a program has in hand before the call, ``run``
makes one pass and ``work`` says what bytes that pass cannot do without.  All
outputs are bytes (or flags), so they have no rounding and no ``exact`` value.

A case is a plain dict:
  via      "call"      one call per stripe on separate device buffers
           "batch"     one call over a (stripes, k + m, shard_len) device block
           "prepared"  a prepared batch over such a block, launched again
           "host"      one call over such a block in pinned host memory
           "mixed"     a prepared mixed batch (many codecs, lengths, operations)
  family   "classic", "leopard_gf8" or "leopard_gf16"
  op       "encode", "reconstruct" or "verify"
  lost     shards missing per stripe (reconstruct)
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(os.getcwd(), "rustfs-erasure-codec_b200")
if not os.path.isdir(_PKG):
    _PKG = os.path.join(ROOT, "rustfs-erasure-codec_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import rsgpu  # noqa: E402
from rsgpu import workload  # noqa: E402

KIB, MIB = 1 << 10, 1 << 20


def _case(name, via, family, op, k, m, shard_len, stripes, lost=0):
    return dict(name=name, via=via, family=family, op=op, k=k, m=m, shard_len=shard_len, stripes=stripes, lost=lost)


def listed():
    return [
        # The smallest call a storage node makes: one small object, latency counts.
        _case("call_encode_4x2_4k", "call", "classic", "encode", 4, 2, 4 * KIB, 1),
        # A degraded read: two lost disks, one 64 KiB-shard stripe, one call.
        _case("call_rebuild_10x4_64k", "call", "classic", "reconstruct", 10, 4, 64 * KIB, 1, lost=2),
        # Bulk ingest: many 1 MiB-shard stripes resident on the device.
        _case("encode_10x4_1m", "prepared", "classic", "encode", 10, 4, MIB, 512),
        # Healing after disk loss: every stripe has its own erasure pattern.
        _case("rebuild_16x4_1m", "prepared", "classic", "reconstruct", 16, 4, MIB, 256, lost=3),
        # A scrub over objects whose shard length is odd, packed back to back.
        _case("verify_12x4_odd", "batch", "classic", "verify", 12, 4, 100003, 128),
        # A wide classic code: more parity than one pass of four outputs.
        _case("encode_50x20_256k", "prepared", "classic", "encode", 50, 20, 256 * KIB, 32),
        # Leopard GF(2^8), the usual 32+16 layout, bulk encode.
        _case("leo8_encode_32x16_1m", "prepared", "leopard_gf8", "encode", 32, 16, MIB, 32),
        # Leopard GF(2^8), wide layout, rebuild of a quarter of a rack.
        _case("leo8_rebuild_128x64_512k", "prepared", "leopard_gf8", "reconstruct", 128, 64, 512 * KIB, 16, lost=32),
        # Leopard GF(2^16), the widest standing layout, both directions.
        _case("leo16_encode_1024x512_16k", "prepared", "leopard_gf16", "encode", 1024, 512, 16 * KIB, 16),
        _case("leo16_rebuild_1024x512_16k", "prepared", "leopard_gf16", "reconstruct", 1024, 512, 16 * KIB, 16,
              lost=512),
        # A storage node's mixed queue: seven codecs, 4 KiB to 4 MiB shards.
        dict(name="mixed_96", via="mixed", ops=96, workload_seed=7, lo=4 * KIB, hi=4 * MIB),
        # Host memory in, host memory out (pinned), the drop-in use.
        _case("host_encode_10x4_1m", "host", "classic", "encode", 10, 4, MIB, 16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _stripes(rng, k, m, shard_len, budget):
    """Stripes for about `budget` bytes or (log-uniformly) down to 1/16 of it."""
    return max(1, int(_log(rng, budget // 16, budget) // ((k + m) * shard_len)))


def draw(rng):
    kind = rng.choice(["call", "call", "classic", "classic", "ragged", "wide", "leo8", "leo8", "leo16", "leo16",
                       "mixed", "host"])
    op = rng.choice(["encode", "encode", "reconstruct", "reconstruct", "verify"])
    if kind == "mixed":
        return dict(via="mixed", ops=rng.randint(16, 96), workload_seed=rng.randint(1, 1 << 20), lo=4 * KIB,
                    hi=_log(rng, 256 * KIB, 4 * MIB))
    if kind == "call":
        k = _log(rng, 2, 24)
        m = rng.randint(1, min(k, 8))
        c = _case("", "call", "classic", op, k, m, _log(rng, KIB, MIB), 1)
    elif kind == "classic":
        k, m = rng.randint(2, 24), rng.randint(1, 4)
        shard_len = max(1, _log(rng, 16 * KIB, 2 * MIB) // 16) * 16
        c = _case("", rng.choice(["prepared", "batch"]), "classic", op, k, m, shard_len,
                  _stripes(rng, k, m, shard_len, 2 << 30))
    elif kind == "ragged":
        k, m = rng.randint(2, 24), rng.randint(1, 4)
        shard_len = _log(rng, 4 * KIB, 512 * KIB) | 1
        c = _case("", rng.choice(["prepared", "batch"]), "classic", op, k, m, shard_len,
                  _stripes(rng, k, m, shard_len, 256 << 20))
    elif kind == "wide":
        k, m = _log(rng, 17, 128), _log(rng, 5, 64)
        shard_len = max(1, _log(rng, 16 * KIB, 512 * KIB) // 16) * 16
        c = _case("", "prepared", "classic", op, k, m, shard_len, _stripes(rng, k, m, shard_len, 256 << 20))
    elif kind == "leo8":
        k, m = _log(rng, 8, 128), _log(rng, 3, 64)
        shard_len = max(1, _log(rng, 4 * KIB, MIB) // 64) * 64
        c = _case("", "prepared", "leopard_gf8", op, k, m, shard_len, _stripes(rng, k, m, shard_len, 512 << 20))
    elif kind == "leo16":
        k, m = _log(rng, 48, 2048), _log(rng, 16, 1024)
        shard_len = max(1, _log(rng, 2 * KIB, 64 * KIB) // 64) * 64
        c = _case("", "prepared", "leopard_gf16", op, k, m, shard_len, _stripes(rng, k, m, shard_len, 96 << 20))
    else:
        k, m = rng.randint(4, 16), rng.randint(2, 4)
        c = _case("", "host", "classic", op, k, m, _log(rng, 64 * KIB, 2 * MIB), 1)
        c["stripes"] = _stripes(rng, k, m, c["shard_len"], 128 << 20)
    if op == "reconstruct":
        c["lost"] = rng.randint(1, min(c["m"], c["k"]))
    elif op == "verify" and c["via"] != "call" and c["stripes"] < 16:
        c["op"] = "encode"  # a scrub goes over many stripes
    del c["name"]
    return c


# ------------------------------------------------------------------ set-up
class _State:
    """What a program keeps: the codec, its buffers and (prepared) its batch."""


def _codec(case):
    opts = None if case["family"] == "classic" else rsgpu.CodecOptions(codec_family=case["family"])
    return rsgpu.ReedSolomon(case["k"], case["m"], opts)


def _present(case, rng):
    """Presence flags, a random erasure pattern of its own for every stripe."""
    total = case["k"] + case["m"]
    pres = np.ones((case["stripes"], total), np.uint8)
    for row in pres:
        row[rng.sample(range(total), case["lost"])] = 0
    return pres


def _random_block(shape, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = math.prod(shape)
    words = torch.randint(-(1 << 63), (1 << 63) - 1, ((n + 7) // 8,), dtype=torch.int64, device="cuda", generator=gen)
    return words.view(torch.uint8)[:n].view(shape)


def _plan_table():
    if rsgpu.Tuner.table_size() == 0:
        rsgpu.Tuner.load(os.path.join(_PKG, "tuning", "plans_b200.txt"))


def _prepare_mixed(case, seed):
    _plan_table()
    specs = workload.mixed_specs(case["ops"], case["workload_seed"], lo=case["lo"], hi=case["hi"])
    idx = list(range(len(specs)))
    off, size = workload.layout(specs, idx)
    st = _State()
    st.arena = _random_block((size,), seed)
    st.codecs = {}
    ops = []
    for i in idx:
        s = specs[i]
        if s.geom not in st.codecs:
            fam, k, m = s.geom
            st.codecs[s.geom] = rsgpu.ReedSolomon(
                k, m, None if fam == "classic" else rsgpu.CodecOptions(codec_family=fam))
        codec = st.codecs[s.geom]
        block = st.arena[off[i]:off[i] + s.stripe_bytes].view(s.total, s.shard_len)
        if s.op != "encode":
            codec.encode(list(block))  # a codeword, as a node's stored stripes are
        op = dict(codec=codec, op=s.op, shards=[block[j].data_ptr() for j in range(s.total)], shard_len=s.shard_len)
        if s.op == "reconstruct":
            op["present"] = s.present
            for j in np.flatnonzero(s.present == 0):
                block[int(j)].fill_(0xA5)
        ops.append(op)
    st.batch = rsgpu.MixedBatch(ops, planner="table")
    st.run = lambda: _run_mixed(st)
    return st


def _run_mixed(st):
    st.batch.launch()
    return [st.arena, st.batch.results().astype(np.uint8)]


def prepare(case, seed):
    if case["via"] == "mixed":
        return _prepare_mixed(case, seed)
    rng = random.Random(seed)
    k, m, op, via = case["k"], case["m"], case["op"], case["via"]
    total, n = k + m, case["stripes"]
    st = _State()
    st.codec = codec = _codec(case)
    block = _random_block((n, total, case["shard_len"]), seed)
    pres = _present(case, rng) if op == "reconstruct" else None
    if op == "encode":
        block[:, k:] = 0
    else:
        codec.encode_batch(block)
    if op == "reconstruct":
        for i, row in enumerate(pres):
            block[i, torch.from_numpy(np.flatnonzero(row == 0)).cuda()] = 0xA5
    elif op == "verify":  # about one stripe in eight is damaged, anywhere
        for i in rng.sample(range(n), max(1, n // 8)):
            block[i, rng.randrange(total), rng.randrange(case["shard_len"])] ^= 0x40
    if via == "call":
        shards = [block[0, i].clone() for i in range(total)]
        if op == "encode":
            st.run = lambda: _call_encode(codec, shards, k)
        elif op == "verify":
            buffer = [torch.zeros_like(shards[0]) for _ in range(m)]
            st.run = lambda: _call_verify(codec, shards, buffer)
        else:
            lost = [int(i) for i in np.flatnonzero(pres[0] == 0)]
            st.run = lambda: _call_rebuild(codec, shards, lost)
    elif via == "prepared":
        ptrs = rsgpu.device_pointer_table(block.data_ptr(),
                                          np.arange(n * total, dtype=np.uint64) * np.uint64(case["shard_len"]))
        batch = codec.prepare_batch(op, ptrs, case["shard_len"], present=pres)
        st.batch = batch
        st.run = lambda: _launch(batch, block, op)
    else:
        if via == "host":
            host = torch.empty(block.shape, dtype=torch.uint8, pin_memory=True)
            host.copy_(block)
            block = host.numpy()
            st.host = host
        st.run = lambda: _batch_call(codec, block, op, pres)
    st.block = block
    torch.cuda.synchronize()
    return st


def _call_encode(codec, shards, k):
    codec.encode(shards)
    return shards[k:]


def _call_verify(codec, shards, buffer):
    ok = codec.verify_with_buffer(shards, buffer)
    return [int(ok)] + buffer


def _call_rebuild(codec, shards, lost):
    work = list(shards)
    for i in lost:
        work[i] = None
    codec.reconstruct(work)
    return [work[i] for i in lost]


def _launch(batch, block, op):
    batch.launch()
    return batch.verify_result().astype(np.uint8) if op == "verify" else block


def _batch_call(codec, block, op, pres):
    if op == "encode":
        codec.encode_batch(block)
        return block
    if op == "reconstruct":
        codec.reconstruct_batch(block, pres)
        return block
    return np.array(codec.verify_batch(block), np.uint8)


def run(state):
    return state.run()


# ------------------------------------------------------------------ bytes
def work(case):
    if case["via"] == "mixed":
        specs = workload.mixed_specs(case["ops"], case["workload_seed"], lo=case["lo"], hi=case["hi"])
        return {"bytes": sum(s.algorithmic_bytes() for s in specs), "flops": 0}
    k, m = case["k"], case["m"]
    shards = k + m  # encode and verify; Leopard rebuilds read every present shard
    if case["op"] == "reconstruct" and case["family"] == "classic":
        shards = k + case["lost"]
    return {"bytes": shards * case["shard_len"] * case["stripes"], "flops": 0}
