"""Writes slice_net.cuh: the jump tables of XOR networks of slice_field.cuh.

    python gen_slice_net.py > slice_net.cuh

For every nibble position q of a constant's tower coordinates and every nibble
value n, the network of x ^= (n << 4q) * y on bit planes: y's planes are first
combined into a few shared terms, then each plane of x takes its terms two at
a time (three-input XORs).  Each table is one PTX block: an indexed uniform
branch over the 16 networks.  Written as a C++ switch the compiler makes a
tree of compares of it and hoists terms that several networks share above the
jump, and the kernels then spill.
"""
import itertools
import random

CANTOR = {8: [1, 214, 152, 146, 86, 200, 88, 230],
          16: [0x0001, 0xACCA, 0x3C0E, 0x163E, 0xC582, 0xED2E, 0x914C, 0x4012,
               0x6C98, 0x10D8, 0x6A72, 0xB900, 0xFDB8, 0xFB34, 0xFF38, 0x991E]}
POLY = {8: 0x11D, 16: 0x1002D}


def field(bits):
    """(multiplication, Cantor -> tower) on Cantor coordinates."""
    basis, poly = CANTOR[bits], POLY[bits]

    def pmul(a, b):
        r = 0
        while b:
            if b & 1:
                r ^= a
            b >>= 1
            a <<= 1
            if a >> bits:
                a ^= poly
        return r

    def combine(vecs, c):
        r = 0
        for i, v in enumerate(vecs):
            if (c >> i) & 1:
                r ^= v
        return r

    def inverse(vecs):
        rows = [(v, 1 << i) for i, v in enumerate(vecs)]
        for p in range(bits):
            s = next(i for i in range(p, bits) if (rows[i][0] >> p) & 1)
            rows[p], rows[s] = rows[s], rows[p]
            for i in range(bits):
                if i != p and (rows[i][0] >> p) & 1:
                    rows[i] = (rows[i][0] ^ rows[p][0], rows[i][1] ^ rows[p][1])
        return [c for _, c in rows]

    inv = inverse(basis)

    def mul(a, b):
        return combine(inv, pmul(combine(basis, a), combine(basis, b)))

    tower = []
    for i in range(bits):
        v = 1 << (i & 3)
        if i & 4:
            v = mul(v, 1 << 4)
        if i & 8:
            v = mul(v, 1 << 8)
        tower.append(v)
    tinv = inverse(tower)

    def tmul(a, b):
        return combine(tinv, mul(combine(tower, a), combine(tower, b)))

    return tmul


def cost(rows, temps):
    return sum((len(r) + 1) // 2 for r in rows) + len(temps)


def network(rows, tries, rng):
    """Shared terms (lists of 2 or 3 signals) that make the rows cheap."""
    best = None
    for _ in range(tries):
        cur, temps, nxt = [set(r) for r in rows], [], 100
        while True:
            counts = {}
            for r in cur:
                s = sorted(r)
                for size in (2, 3):
                    for c in itertools.combinations(s, size):
                        counts[c] = counts.get(c, 0) + 1
            base, options = cost(cur, temps), []
            for c, k in counts.items():
                if k < 2:
                    continue
                gain = -1
                for r in cur:
                    if set(c) <= r:
                        n = len(r)
                        gain += (n + 1) // 2 - (n - len(c) + 2) // 2
                if gain > 0 or (gain == 0 and rng.random() < 0.02):
                    options.append((gain, rng.random(), c))
            if not options:
                break
            options.sort(reverse=True)
            pick = options[0] if rng.random() < 0.7 else rng.choice(options[:6])
            c = set(pick[2])
            for r in cur:
                if c <= r:
                    r -= c
                    r.add(nxt)
            temps.append((nxt, sorted(c)))
            nxt += 1
            if cost(cur, temps) > base:
                break
        if best is None or cost(cur, temps) < cost(best[0], best[1]):
            best = (cur, temps)
    return best


def emit_xor(dst, srcs):
    """dst = XOR of srcs, or dst ^= srcs when dst is not a new name."""
    out, acc, rest = [], None, list(srcs)
    if dst.startswith("%%") or dst.startswith("t"):
        acc = rest.pop(0)
    else:
        acc = dst
    while rest:
        if len(rest) >= 2:
            out.append(f"lop3.b32 {dst}, {acc}, {rest.pop(0)}, {rest.pop(0)}, 0x96;")
        else:
            out.append(f"xor.b32 {dst}, {acc}, {rest.pop(0)};")
        acc = dst
    return out


def emit_table(bits, q, pairs, nets, prefix="mac"):
    name = f"{prefix}{pairs if pairs > 1 else ''}_nibble"
    nx = bits * pairs
    args = ", ".join(f"uint32_t *x{p}, const uint32_t *y{p}" for p in range(pairs))
    print("template <>")
    targs = f"{bits}, {4 * q}" if prefix == "mac" else f"{4 * q}"
    print(f"__device__ __forceinline__ void {name}<{targs}>(uint32_t n, {args}) {{")
    print('  asm volatile(')
    most = max(len(t) for _, t in nets[1:])
    print(f'      "{{\\n\\t.reg .b32 t<{most + 1}>;\\n"')
    print('      "T: .branchtargets ' + ", ".join(f"N{n}" for n in range(16)) + ';\\n\\t"')
    print(f'      "brx.idx.uni %{2 * nx}, T;\\n"')
    for n in range(1, 16):
        rows, temps = nets[n]
        body = []
        for p in range(pairs):
            def sig(s, p=p):
                return f"t{s - 100}" if s >= 100 else f"%{nx + p * bits + s}"
            for t, c in temps:
                body += emit_xor(f"t{t - 100}", [sig(s) for s in c])
            for r in range(bits):
                if rows[r]:
                    body += emit_xor(f"%{p * bits + r}", [sig(s) for s in sorted(rows[r])])
        lines = [f"N{n}:\\n\\t"] + [b + "\\n\\t" for b in body] + ["bra.uni N0;\\n"]
        print('      "' + '"\n      "'.join(_wrap(lines)) + '"')
    print('      "N0:\\n\\t}"')
    outs = ", ".join(f'"+r"(x{p}[{r}])' for p in range(pairs) for r in range(bits))
    ins = ", ".join(f'"r"(y{p}[{r}])' for p in range(pairs) for r in range(bits))
    print(f"      : {outs}")
    print(f'      : {ins}, "r"(n));')
    print("}")


def _wrap(parts, width=108):
    lines, cur = [], ""
    for p in parts:
        if cur and len(cur) + len(p) > width:
            lines.append(cur)
            cur = ""
        cur += p
    return lines + [cur]


def main():
    print("// slice_net.cuh -- written by gen_slice_net.py; see there.\n")
    rng = random.Random(20)
    for bits in (8, 16):
        tmul = field(bits)
        for q in range(bits // 4):
            nets, total = [None], 0
            for n in range(1, 16):
                cols = [tmul(n << (4 * q), 1 << b) for b in range(bits)]
                rows = [{b for b in range(bits) if (cols[b] >> r) & 1} for r in range(bits)]
                net = network(rows, 400 if bits == 8 else 60, rng)
                nets.append(net)
                total += cost(*net)
            print(f"// GF(2^{bits}), nibble {q}: {total / 15:.1f} XOR instructions a network on average.")
            for pairs in (1, 2):
                emit_table(bits, q, pairs, nets)
    # GF(2^16)'s subfield GF(256), which maps each half of the planes to itself.
    tmul = field(16)
    for q in range(2):
        nets = [None]
        for n in range(1, 16):
            cols = [tmul(n << (4 * q), 1 << b) for b in range(8)]
            assert all(c < 256 and tmul(n << (4 * q), 256 << b) == c << 8 for b, c in enumerate(cols))
            nets.append(network([{b for b in range(8) if (cols[b] >> r) & 1} for r in range(8)], 400, rng))
        print(f"// GF(256) in GF(2^16), nibble {q}: "
              f"{sum(cost(*n) for n in nets[1:]) / 15:.1f} XOR instructions a network on average.")
        for pairs in (1, 2):
            emit_table(8, q, pairs, nets, "sub")


if __name__ == "__main__":
    main()
