"""The problem setup's loop over host threads: every part runs once, and what a part
throws -- in a thread or where threads have run out -- reaches the caller after the
others have ended, instead of ending the process."""
import pytest

from host_cpp import run_cpp

PROGRAM = """
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include "tg_host_parallel.h"
int main(int, char** a) {
  const int64_t n = std::atoll(a[1]), nodes = std::atoll(a[2]), bad = std::atoll(a[3]);
  std::atomic<int64_t> items{0}, wrong{0};
  const char* end = "returned";
  try {
    tg::host_parallel(n, nodes, [&](int64_t lo, int64_t hi, int part) {
      if (lo < 0 || hi > n || part < 0 || part >= 16) ++wrong;
      if (lo <= bad && bad < hi) throw std::bad_alloc();
      items += hi - lo;
    });
  } catch (const std::bad_alloc&) {
    end = "bad_alloc";
  }
  std::printf("%s %lld %lld", end, (long long)items.load(), (long long)wrong.load());
}
"""


@pytest.mark.parametrize("n,nodes", [(1000, 1), (1000, 1 << 20), (3, 1 << 20), (16, 1 << 20),
                                     (17, 1 << 21)])
def test_every_item_once(tmp_path, n, nodes):
    assert run_cpp(tmp_path, PROGRAM, n, nodes, -1).stdout == f"returned {n} 0"


@pytest.mark.parametrize("bad", [0, 500, 999])
@pytest.mark.parametrize("nodes", [1, 1 << 20])
def test_an_exception_reaches_the_caller(tmp_path, nodes, bad):
    done = run_cpp(tmp_path, PROGRAM, 1000, nodes, bad)
    end, items, wrong = done.stdout.split()
    assert done.returncode == 0 and end == "bad_alloc" and int(wrong) == 0
    assert int(items) < 1000
