"""The order of a kernel's row blocks and the rules that choose it, compiled for the host: an order changes no result, so nothing on the device
shows a block that is taken twice, one that is left out, or a rule that counts the wrong bytes."""
import subprocess

import pytest

from torch_mlu_b200 import build

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "block_order.cuh"
#include "kernels.h"
using namespace sdpa_b200;

static int failed = 0;
static void check(bool ok, const char* what, int a, int b, int c, int d) {
  if (!ok && failed++ < 20) std::printf("%s: %d %d %d %d\n", what, a, b, c, d);
}

int main() {
  // every (rank, head) has one slot, the ranks behind all groups come last
  for (int heads = 1; heads <= 70; heads += heads < 8 ? 1 : 3)
    for (int ranks = 1; ranks <= 9; ++ranks)
      for (int group = 1; group <= 32 && group <= heads; group += group < 6 ? 1 : 5)
        for (int tail = 0; tail <= ranks / 2; ++tail) {
          const BlockOrder o = block_order(heads, ranks, group, tail);
          std::vector<int> seen(heads * ranks, 0);
          for (int slot = 0; slot < o.slots; ++slot) {
            int rank, head;
            if (!block_of_slot(o, slot, rank, head)) continue;
            const bool in_range = rank >= 0 && rank < ranks && head >= 0 && head < heads;
            check(in_range, "out of range", heads, ranks, group, slot);
            if (in_range) ++seen[rank * heads + head];
            check((rank >= ranks - tail) == (slot >= o.front_slots), "tail", heads, ranks, group, slot);
          }
          for (int n : seen) check(n == 1, "not once", heads, ranks, group, tail);
        }
  // groups cover the heads with at most one short one
  for (int heads = 1; heads <= 300; ++heads)
    for (double mb = 0.2; mb < 100; mb *= 1.7)
      for (int even = 0; even < 2; ++even) {
        const int n = heads_per_l2_group(mb * 1048576, heads, 48.0 * 1048576, even != 0);
        check(n >= 1 && n <= heads && (n == heads || n <= 32), "group", heads, static_cast<int>(mb * 10), even, n);
      }
  // causal forward: the ranks behind all groups and the keys that they see stay in L2 together
  const double mb = 1048576.0;
  check(tail_ranks(16, 4 * mb, 0) == 8, "as many as half", 16, 0, 0, tail_ranks(16, 4 * mb, 0));
  check(tail_ranks(16, 10 * mb, 0) == 3, "as many as fit", 16, 0, 0, tail_ranks(16, 10 * mb, 0));
  check(tail_ranks(16, 10 * mb, 13 * mb) == 1, "behind a prefix", 16, 13, 0, tail_ranks(16, 10 * mb, 13 * mb));
  check(tail_ranks(2, 28 * mb, 86 * mb) == 0, "behind a long prefix", 2, 86, 0, tail_ranks(2, 28 * mb, 86 * mb));
  check(tail_ranks(1, 1 * mb, 0) == 0, "a single rank", 1, 0, 0, tail_ranks(1, 1 * mb, 0));
  return failed != 0;
}
"""


def test_every_block_once_and_the_rules_that_order_them(tmp_path):
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("no nvcc here")
    source, program = tmp_path / "orders.cu", tmp_path / "orders"
    source.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-I", build.CSRC, "-I", build.INCLUDE, "-o", str(program), str(source)], check=True, capture_output=True)
    result = subprocess.run([str(program)], capture_output=True, text=True)
    assert result.returncode == 0, result.stdout
