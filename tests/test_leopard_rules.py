"""CPU: the rules that send Leopard work to the bit-sliced kernels
(leo_rules.hpp) against times measured on one B200: on either side of every
line of a rule, the kernels it picks took at most 8% longer than the others."""
import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
ENCODE, RECONSTRUCT, VERIFY = 0, 1, 2

_DRIVER = """
#include <cstdio>
#include "leo_rules.hpp"
int main() {
  unsigned bits, op, k, p;
  unsigned long long len, stripes;
  while (scanf("%u %u %u %u %llu %llu", &bits, &op, &k, &p, &len, &stripes) == 6) {
    unsigned m = 1, n = 1;
    while (m < p) m *= 2;
    while (n < m + k) n *= 2;
    puts(SLICED ? "1" : "0");
  }
}
"""


def _picks(tmp_path, expr, bits, cases):
    src = tmp_path / "rules.cpp"
    src.write_text(_DRIVER.replace("SLICED", expr))
    exe = tmp_path / "rules"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "rustfs-erasure-codec_b200" / "csrc"), str(src), "-o", str(exe)], check=True)
    text = "".join("%d %d %d %d %d %d\n" % (bits, *c[:5]) for c in cases)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.split()
    assert len(out) == len(cases)
    return [x == "1" for x in out]


def _check(cases, picks):
    slow = [(c, sliced) for c, sliced in zip(cases, picks) if c[6 if sliced else 5] > 1.08 * min(c[5:])]
    assert not slow


# (operation, k, parity, shard length, stripes, us in the register-stage kernels, us bit-sliced)
GF8 = [
    (ENCODE, 9, 9, 65536, 1, 8, 10),
    (ENCODE, 16, 16, 64, 1, 8, 12),
    (ENCODE, 16, 16, 262144, 1, 10, 12),
    (ENCODE, 16, 16, 4096, 256, 25, 19),
    (ENCODE, 32, 16, 256, 64, 12, 14),
    (ENCODE, 32, 16, 262144, 4, 35, 29),
    (ENCODE, 60, 9, 4096, 64, 21, 22),
    (ENCODE, 60, 9, 4096, 128, 31, 27),
    (VERIFY, 24, 16, 64, 1, 17, 12),
    (VERIFY, 60, 9, 4096, 1, 23, 21),
    (VERIFY, 32, 16, 65536, 1, 17, 14),
    (VERIFY, 16, 16, 65536, 4, 15, 16),
    (VERIFY, 32, 16, 262144, 4, 39, 33),
    (VERIFY, 17, 17, 256, 1, 14, 12),
    (ENCODE, 17, 17, 512, 1, 12, 10),
    (ENCODE, 64, 32, 64, 256, 16, 21),
    (ENCODE, 64, 32, 128, 64, 15, 17),
    (ENCODE, 64, 32, 512, 1, 21, 14),
    (ENCODE, 224, 32, 64, 256, 37, 49),
    (ENCODE, 224, 32, 512, 1, 49, 37),
    (ENCODE, 224, 32, 4096, 64, 88, 53),
    (ENCODE, 60, 64, 64, 1, 12, 14),
    (ENCODE, 128, 64, 64, 64, 19, 21),
    (ENCODE, 128, 64, 256, 256, 23, 31),
    (ENCODE, 128, 64, 512, 64, 21, 21),
    (ENCODE, 10, 100, 896, 64, 23, 20),
    (ENCODE, 128, 64, 4096, 64, 72, 48),
    (ENCODE, 180, 64, 1024, 32, 27, 31),
    (ENCODE, 180, 64, 65536, 1, 31, 29),
    (ENCODE, 180, 64, 262144, 1, 94, 43),
    (VERIFY, 60, 64, 512, 1, 19, 16),
    (VERIFY, 128, 64, 1024, 16, 25, 23),
    (VERIFY, 180, 64, 512, 64, 31, 31),
    (VERIFY, 180, 64, 4096, 64, 103, 68),
    (ENCODE, 100, 100, 64, 1, 18, 25),
    (ENCODE, 100, 100, 16384, 1, 19, 25),
    (ENCODE, 100, 100, 256, 256, 27, 37),
    (ENCODE, 100, 100, 131072, 1, 49, 27),
    (ENCODE, 120, 128, 65536, 4, 90, 43),
    (ENCODE, 10, 100, 1024, 1, 17, 19),
    (ENCODE, 10, 100, 4096, 64, 74, 39),
    (VERIFY, 100, 100, 16384, 1, 23, 27),
    (VERIFY, 120, 128, 131072, 1, 59, 34),
    (RECONSTRUCT, 9, 9, 64, 1, 14, 10),
    (RECONSTRUCT, 10, 4, 4096, 1, 13, 11),
    (RECONSTRUCT, 10, 4, 262144, 1, 15, 10),
    (RECONSTRUCT, 128, 64, 64, 1, 45, 35),
    (RECONSTRUCT, 128, 64, 4096, 64, 242, 96),
]


def test_gf8_rule_picks_the_faster_kernels(tmp_path):
    _check(GF8, _picks(tmp_path, "rsgpu::slice_pays(int(op), k, m, n, len, len * stripes)", 8, GF8))


GF16 = [
    (ENCODE, 20, 33, 2048, 1, 14, 19),
    (ENCODE, 20, 33, 65536, 2, 21, 25),
    (ENCODE, 60, 64, 65536, 2, 25, 25),
    (ENCODE, 60, 64, 65536, 4, 45, 33),
    (ENCODE, 60, 64, 2112, 64, 26, 31),
    (ENCODE, 120, 64, 4096, 4, 21, 22),
    (ENCODE, 120, 64, 65536, 1, 23, 25),
    (ENCODE, 120, 64, 65536, 2, 35, 29),
    (ENCODE, 120, 64, 2112, 64, 37, 43),
    (VERIFY, 180, 64, 32768, 1, 29, 31),
    (ENCODE, 180, 64, 2112, 32, 29, 35),
    (ENCODE, 180, 64, 2048, 64, 47, 37),
    (ENCODE, 200, 60, 2048, 1, 29, 25),
    (ENCODE, 200, 60, 2112, 64, 55, 61),
    (ENCODE, 200, 60, 16384, 1, 29, 26),
    (ENCODE, 100, 128, 2048, 1, 17, 21),
    (ENCODE, 100, 128, 16384, 2, 19, 25),
    (ENCODE, 100, 128, 65536, 2, 51, 33),
    (ENCODE, 200, 128, 2048, 16, 25, 26),
    (ENCODE, 200, 128, 2048, 32, 39, 31),
    (ENCODE, 200, 128, 2112, 32, 39, 45),
    (ENCODE, 300, 128, 2112, 16, 31, 37),
    (ENCODE, 300, 128, 2048, 32, 51, 37),
    (ENCODE, 100, 200, 1024, 1, 20, 25),
    (ENCODE, 256, 256, 16384, 1, 21, 25),
    (ENCODE, 256, 256, 2048, 16, 39, 29),
    (ENCODE, 400, 200, 1024, 4, 29, 27),
    (ENCODE, 400, 200, 1024, 16, 29, 31),
    (ENCODE, 400, 200, 2048, 16, 53, 32),
    (ENCODE, 600, 256, 2048, 4, 35, 29),
    (ENCODE, 600, 256, 1024, 64, 131, 100),
    (ENCODE, 500, 500, 1024, 1, 35, 27),
    (ENCODE, 500, 500, 1024, 16, 35, 38),
    (ENCODE, 500, 500, 2048, 16, 68, 39),
    (ENCODE, 1024, 512, 1024, 8, 51, 35),
    (ENCODE, 1024, 512, 1088, 16, 52, 58),
    (ENCODE, 1024, 512, 1024, 32, 101, 96),
    (ENCODE, 100, 1000, 1024, 16, 61, 54),
    (ENCODE, 2048, 1024, 1024, 1, 117, 33),
    (ENCODE, 2048, 1024, 2112, 64, 1071, 838),
    (VERIFY, 60, 64, 65536, 1, 21, 29),
    (VERIFY, 60, 64, 65536, 4, 51, 37),
    (VERIFY, 128, 100, 65536, 1, 31, 33),
    (VERIFY, 128, 100, 65536, 2, 54, 36),
    (VERIFY, 256, 256, 1024, 16, 25, 31),
    (VERIFY, 60, 200, 65536, 1, 76, 35),
    (VERIFY, 1024, 512, 1024, 16, 55, 61),
    (VERIFY, 1024, 512, 4096, 1, 55, 33),
    (RECONSTRUCT, 40, 16, 1024, 1, 39, 23),
    (RECONSTRUCT, 64, 32, 2048, 4, 43, 25),
    (RECONSTRUCT, 1024, 512, 1024, 1, 162, 38),
]


def test_gf16_rule_picks_the_faster_kernels(tmp_path):
    _check(GF16, _picks(tmp_path, "rsgpu::slice16_pays(int(op), k, m, n, len, stripes)", 16, GF16))


@pytest.mark.parametrize("cases", [GF8, GF16])
@pytest.mark.parametrize("sliced", [False, True])
def test_a_wrong_rule_is_seen(cases, sliced):
    with pytest.raises(AssertionError):
        _check(cases, [sliced] * len(cases))
