"""CPU: the rules that pick a kernel for misaligned classic shards and for
verifies of few inputs (classic_rules.hpp), updates among them, against times measured on one B200: on
either side of their lines, the kernel they pick took at most 10% longer than the
other."""
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

STAGED = 2
# (, inputs, shard length, stripes, us with tables in registers, us staged)
FEW_INPUTS = [
    (STAGED, 1, 1024, 1024, 8, 12),
    (STAGED, 1, 4096, 1024, 11, 12),
    (STAGED, 1, 65536, 64, 10.3, 8.4),
    (STAGED, 1, 1048576, 256, 225, 200),
    (STAGED, 2, 1024, 1024, 10, 14),
    (STAGED, 2, 4096, 1024, 12, 15),
    (STAGED, 2, 1048576, 8, 16.5, 14.5),
    (STAGED, 3, 262144, 256, 86, 90),
    (STAGED, 4, 4096, 1024, 15, 20),
]

UPDATE = 3
# (, outputs + 1000 * inputs, shard length, stripes, us by bytes, us by words)
UPDATES = [
    (UPDATE, 1004, 4194301, 1, 43, 70),
    (UPDATE, 1004, 16777213, 1, 145, 192),
    (UPDATE, 3004, 16777213, 1, 278, 299),
    (UPDATE, 5004, 4194301, 1, 78, 88),
    (UPDATE, 5004, 16777213, 1, 410, 317),
    (UPDATE, 10004, 1048573, 1, 43, 43),
    (UPDATE, 10004, 4194301, 1, 145, 109),
    (UPDATE, 5008, 4194301, 1, 120, 143),
    (UPDATE, 10008, 4194301, 1, 234, 199),
    (UPDATE, 10020, 4194301, 1, 458, 517),
    (UPDATE, 20020, 4194301, 1, 724, 679),
    (UPDATE, 50020, 1048573, 1, 474, 425),
    (UPDATE, 50020, 4194301, 1, 1751, 1238),
]

_DRIVER = """
#include <cstdio>
#include "classic_rules.hpp"
int main() {
  unsigned verify, outs;
  unsigned long long len, stripes;
  while (scanf("%u %u %llu %llu", &verify, &outs, &len, &stripes) == 4)
    puts((verify == 3   ? rsgpu::words_pay_update(outs / 1000, outs % 1000, len, stripes)
          : verify == 2 ? rsgpu::verify_staged(outs, len, stripes)
                        : rsgpu::words_pay(verify, outs, len, stripes))
             ? "1" : "0");
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


def _slow(cases, picks):
    return [c for c, second in zip(cases, picks) if c[5 if second else 4] > 1.1 * min(c[4:])]


@pytest.mark.parametrize("cases", [TIMES, FEW_INPUTS, UPDATES])
def test_rule_picks_the_faster_kernel(tmp_path, cases):
    assert not _slow(cases, _picks(tmp_path, cases))


@pytest.mark.parametrize("cases", [TIMES, FEW_INPUTS, UPDATES])
@pytest.mark.parametrize("second", [False, True])
def test_a_wrong_rule_is_seen(cases, second):
    assert _slow(cases, [second] * len(cases))


def test_short_shards_and_empty_launches_go_by_bytes(tmp_path):
    assert not any(_picks(tmp_path, [(op, outs, length, stripes, 0, 0) for op in (WRITE, VERIFY) for outs in (1, 4, 5, 200)
                                     for length in (1, 3, 4, 11, 12, 100) for stripes in (1, 100000)]))
