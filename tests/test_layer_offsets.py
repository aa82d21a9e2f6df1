"""The byte offset of a node within its layer, at the largest layers that 32-bit DOF
indices allow (357,913,941 nodes of a bounded grid's two layers or more, 715,827,882 of
a periodic cell's one) and on both sides of 2^32 bytes."""
import pytest

from host_cpp import run_cpp

PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "tg_index.h"
int main(int, char** a) {
  const int no = std::atoi(a[1]);
  const bool narrow = tg::narrow_layer(int64_t(no) + 1);  // this node is the last one
  std::printf("%lld %lld %d",
              narrow ? (long long)tg::node_bytes<float, true>(no)
                     : (long long)tg::node_bytes<float, false>(no),
              (long long)tg::node_bytes<double, false>(no), narrow ? 1 : 0);
}
"""


@pytest.mark.parametrize("node", [0, 1, 178956970, 178956971, 192028000, 357913940,
                                  357913941, 715827881])
def test_node_offset(tmp_path, node):
    out = run_cpp(tmp_path, PROGRAM, node).stdout.split()
    assert [int(v) for v in out] == [12 * node, 24 * node, int(12 * node + 11 < 2 ** 32)]


def test_a_layer_never_has_more_nodes():
    """What the grid check accepts: three DOFs a node below 2^31, two layers or more."""
    assert (2 ** 31 - 1) // 3 // 2 <= 357913941 and 12 * 357913941 < 2 ** 32
