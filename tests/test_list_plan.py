"""The joins' candidate list: its size and the buckets of its grouping, over the numbers of rows
and of appending warps that the joins take (the header's host code, compiled here)."""
import os
import subprocess

import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "gpu_hdbscan_b200", "csrc", "list_plan.h")
ROWS = sorted({b + e for p in range(1, 32) for b in (1 << p, 511 << p) if b < 1 << 31
               for e in (-257, -129, -128, -2, -1, 0, 1, 2) if 2 <= b + e < (1 << 31) - 1})


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    """{(rows, warps): (slots, chunk, shift)}"""
    d = tmp_path_factory.mktemp("plan")
    src = d / "plan.cpp"
    src.write_text(f"""#include <cstdio>
#include "{HEADER}"
int main() {{
  long long n, w;
  while (scanf("%lld %lld", &n, &w) == 2)
    printf("%lld %u %d\\n", (long long)hdb::knn::list_slots(n, w), hdb::knn::list_chunk(n, w),
           hdb::knn::bucket_shift(n));
}}""")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-o", str(d / "plan"), str(src)])
    keys = [(n, w) for n in ROWS for w in (4, 1184, 4736, 9472)]
    out = subprocess.run([str(d / "plan")], input="\n".join(f"{n} {w}" for n, w in keys), text=True,
                         stdout=subprocess.PIPE, check=True).stdout.split("\n")
    return {key: tuple(int(x) for x in line.split()) for key, line in zip(keys, out)}


def test_slots_hold_the_candidates_and_the_tails(plan):
    for (n, w), (slots, chunk, _) in plan.items():
        assert slots >= min(64 * n + w * chunk, 1 << 31)
        assert slots >= min(96 * n, 64 << 20)


def test_a_block_steps_past_the_list_in_32_bits(plan):
    """The grouping walks a bucket's slots in steps of a block's 512 threads."""
    assert all(slots + 512 <= 1 << 32 for slots, _, _ in plan.values())


def test_buckets_take_the_fewest_digits(plan):
    """The buckets and the one of the unused slots behind them, in digits of 9 bits."""
    for (n, _), (_, _, shift) in plan.items():
        values = -(-n >> shift) + 1
        assert 3 <= shift <= 8
        if n <= 511 * 256:
            assert values <= 1 << 9
        elif n <= 1 << 25:
            assert values <= 1 << 18, n
        else:
            assert values <= 1 << 27
