"""The counting and numbering of an unscreened class's quartets (csrc/buckets.cuh), compiled
for the host: exact past 2^32, where a class of a large molecule lies."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcmurchie-davidson_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "buckets.cuh"
using namespace mmdg;

// args: same, groups of the bra list, their sizes, groups of the ket list, their sizes
int main(int, char** v) {
  TensorBuckets tb = {};
  int x = 1, at = 0;
  const int same = atoi(v[x++]);
  tb.nbg = atoi(v[x++]);
  for (int g = 0; g < tb.nbg; ++g) tb.bstart[g] = at, at += atoi(v[x++]);
  tb.bstart[tb.nbg] = at;
  tb.nkg = atoi(v[x++]);
  at = 0;
  for (int g = 0; g < tb.nkg; ++g) tb.kstart[g] = at, at += atoi(v[x++]);
  tb.kstart[tb.nkg] = at;
  unsigned long long total = 0, items = 0;
  for (int k = 0; k < tb.nbg * tb.nkg; ++k) {
    const unsigned long long n = bucket_quartets(tb, same, k);
    total += n;
    items += bucket_items(n, 0);
    // first, last and a few slots between, both sides of 2^32 among them
    const unsigned long long probe[] = {0, 1, n / 3, n / 2, (1ull << 32) - 1, 1ull << 32, n - 2, n - 1};
    for (unsigned long long s : probe) {
      if (s >= n) continue;
      int ib, jk;
      bucket_slot(tb, same, k, s, ib, jk);
      printf("slot %d %llu %d %d\n", k, s, ib, jk);
    }
  }
  printf("total %llu %llu\n", total, items);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("buckets")
    (d / "b.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "b.cpp"), "-o", str(d / "b")])
    return str(d / "b")


@pytest.mark.parametrize("same,bra,ket", [
    (0, [3], [2, 5]),
    (1, [4, 3], [4, 3]),
    (1, [65535], [65535]),           # a (a + 1) just inside 32 bits
    (1, [65703], [65703]),           # 362 one-primitive s shells
    (1, [100000, 90000], [100000, 90000]),
    (0, [72828], [63903]),           # (ps|ss) of (H2O)51, more than 2^32 quartets in one bucket
    (0, [30000, 40000], [50000, 22000]),
])
def test_quartets_are_counted_and_numbered_exactly(program, same, bra, ket):
    out = subprocess.check_output([program, str(same), str(len(bra)), *map(str, bra), str(len(ket)), *map(str, ket)],
                                  text=True).split("\n")
    n, m = sum(bra), sum(ket)
    total, items = map(int, out[-2].split()[1:])
    assert total == (n * (n + 1) // 2 if same else n * m)
    assert total <= items < total + 32 * len(bra) * len(ket) and items % 32 == 0
    for line in out[:-2]:
        k, s, ib, jk = map(int, line.split()[1:])
        gb, gk = divmod(k, len(ket))
        i, j = ib - sum(bra[:gb]), jk - sum(ket[:gk])
        assert 0 <= i < bra[gb] and 0 <= j < ket[gk]
        assert s == (i * (i + 1) // 2 + j if same and gb == gk else i * ket[gk] + j)
        if same and gb == gk:
            assert j <= i
