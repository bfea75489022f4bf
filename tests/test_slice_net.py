"""CPU: the generated XOR networks (slice_net.cuh) are what gen_slice_net.py
writes, and each is multiplication by its constant."""
import pathlib
import re
import subprocess
import sys

CSRC = pathlib.Path(__file__).resolve().parents[1] / "rustfs-erasure-codec_b200" / "csrc"


def test_generated_file_is_current():
    out = subprocess.run([sys.executable, str(CSRC / "gen_slice_net.py")], capture_output=True, text=True, check=True)
    assert out.stdout == (CSRC / "slice_net.cuh").read_text()


def _gen():
    sys.path.insert(0, str(CSRC))
    try:
        import gen_slice_net
    finally:
        sys.path.pop(0)
    return gen_slice_net


def test_networks_multiply():
    gen = _gen()
    text = (CSRC / "slice_net.cuh").read_text()
    tables = re.findall(r"void (mac2?|sub2?)_nibble<(?:(\d+), )?(\d+)>(.*?)\n}\n", text, re.S)
    assert len(tables) == 2 * (2 + 4 + 2)
    for name, bits, shift, body in tables:
        # "sub": the subfield GF(256) of GF(2^16), on half the planes.
        mul = gen.field(int(bits or 16))
        bits, shift, pairs = int(bits or 8), int(shift), 2 if name.endswith("2") else 1
        nx = bits * pairs
        code = "".join(re.findall(r'"(.*)"\n', body)).replace("\\n", "\n").replace("\\t", "")
        nets = re.findall(r"^N(\d+):\n(.*?)bra\.uni N0;", code, re.S | re.M)
        assert [int(n) for n, _ in nets] == list(range(1, 16))
        for n, ops in nets:
            # Registers as sets of inputs: bit i of a value is plane i of y (or x).
            reg = {f"%{i}": 1 << i for i in range(2 * nx)}
            for op in filter(None, ops.split("\n")):
                kind, args = op.rstrip(";").split(" ", 1)
                args = args.split(", ")
                if kind == "lop3.b32":
                    assert args.pop() == "0x96"
                acc = 0
                for a in args[1:]:
                    acc ^= reg[a]
                reg[args[0]] = acc
            for p in range(pairs):
                cols = [mul(int(n) << shift, 1 << b) for b in range(bits)]
                if name.startswith("sub"):
                    assert all(mul(int(n) << shift, 256 << b) == c << 8 and c < 256 for b, c in enumerate(cols))
                for r in range(bits):
                    want = 1 << (p * bits + r)
                    for b in range(bits):
                        if (cols[b] >> r) & 1:
                            want ^= 1 << (nx + p * bits + b)
                    assert reg[f"%{p * bits + r}"] == want, (name, bits, shift, n, p, r)
