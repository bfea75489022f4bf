"""CPU: the rule that picks a kernel for misaligned classic shards
(classic_rules.hpp) against times measured on one B200: on either side of its
lines, the kernel it picks took at most 10% longer than the other."""
import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
WRITE, VERIFY = 0, 1

# (operation, outputs, shard length, stripes, us by bytes, us by words), inputs in the comment
TIMES = [
    (WRITE, 4, 20001, 16, 8, 12),        # 10
    (WRITE, 4, 50001, 16, 14, 12),
    (WRITE, 4, 20001, 64, 21, 16),
    (WRITE, 4, 100003, 16, 25, 16),
    (WRITE, 4, 5001, 512, 41, 39),       # 12
    (WRITE, 4, 1029, 512, 12, 14),
    (WRITE, 4, 20001, 16, 12, 17),       # 24
    (WRITE, 4, 10001, 64, 14, 16),       # 16
    (WRITE, 6, 500001, 1, 15, 19),       # 10
    (WRITE, 6, 5001, 256, 31, 37),
    (WRITE, 6, 20001, 64, 31, 25),
    (WRITE, 20, 20001, 16, 69, 113),     # 50
    (WRITE, 20, 1029, 512, 99, 142),
    (WRITE, 20, 50001, 16, 92, 127),
    (WRITE, 20, 5001, 256, 172, 248),
    (WRITE, 20, 100003, 16, 208, 144),
    (WRITE, 8, 100003, 16, 58, 39),      # 20
    (VERIFY, 4, 50001, 4, 9, 12),        # 12
    (VERIFY, 4, 20001, 16, 12, 12),
    (VERIFY, 4, 50001, 16, 19, 12),      # 10
    (VERIFY, 4, 1029, 64, 10, 12),       # 24
    (VERIFY, 20, 20001, 16, 78, 119),    # 50
    (VERIFY, 20, 5001, 157, 150, 208),
    (VERIFY, 20, 1029, 512, 110, 165),
    (VERIFY, 20, 20001, 64, 250, 207),
    (VERIFY, 8, 10001, 64, 31, 31),      # 20
]

_DRIVER = """
#include <cstdio>
#include "classic_rules.hpp"
int main() {
  unsigned verify, outs;
  unsigned long long len, stripes;
  while (scanf("%u %u %llu %llu", &verify, &outs, &len, &stripes) == 4)
    puts(rsgpu::words_pay(verify, outs, len, stripes) ? "1" : "0");
}
"""


def _picks(tmp_path, cases):
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(_DRIVER)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(ROOT / "rustfs-erasure-codec_b200" / "csrc"),
                    str(src), "-o", str(exe)], check=True)
    text = "".join("%d %d %d %d\n" % c[:4] for c in cases)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.split()
    assert len(out) == len(cases)
    return [x == "1" for x in out]


def _slow(picks):
    return [c for c, words in zip(TIMES, picks) if c[5 if words else 4] > 1.1 * min(c[4:])]


def test_rule_picks_the_faster_kernel(tmp_path):
    assert not _slow(_picks(tmp_path, TIMES))


@pytest.mark.parametrize("words", [False, True])
def test_a_wrong_rule_is_seen(words):
    assert _slow([words] * len(TIMES))


def test_short_shards_and_empty_launches_go_by_bytes(tmp_path):
    assert not any(_picks(tmp_path, [(op, outs, length, stripes, 0, 0) for op in (WRITE, VERIFY) for outs in (1, 4, 5, 200)
                                     for length in (1, 3, 4, 11, 12, 100) for stripes in (1, 100000)]))
