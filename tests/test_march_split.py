"""The split of a z march among blocks (csrc/march.h) against trying every
number of layers, and its cost where layers are many (compiled here with g++;
no GPU).  The time limit is 30 times what the split takes and a fourteenth of
what trying every number takes."""
import ctypes as C
import os
import random
import subprocess
import time

import pytest

from sparlab_gb300 import build as B

SOURCE = """
#include "march.h"
extern "C" long long march_layers(long long c, long long n, long long s) { return simp::march_layers(c, n, s); }
extern "C" long long march_layers_by_trying(long long c, long long n, long long s) {
  long long best = n, steps = INT64_MAX;
  for (long long l = 1; l <= n; ++l) {
    const long long t = (c * ((n + l - 1) / l) + s - 1) / s * (l + 2);
    if (t < steps) steps = t, best = l;
  }
  return best;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("march")
    (d / "m.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", B.CSRC, str(d / "m.cpp"), "-o",
                           str(d / "m.so")])
    m = C.CDLL(str(d / "m.so"))
    for f in (m.march_layers, m.march_layers_by_trying):
        f.argtypes, f.restype = [C.c_longlong] * 3, C.c_longlong
    return m


def test_fewest_steps(lib):
    rng = random.Random(3)
    for _ in range(20000):
        c, n, s = (int(2 ** rng.uniform(0, e)) for e in (14, 10, 10))
        assert lib.march_layers(c, n, s) == lib.march_layers_by_trying(c, n, s), (c, n, s)
    for n in (60001, 131072):
        assert lib.march_layers(1, n, 304) == lib.march_layers_by_trying(1, n, 304)


def test_cost_does_not_grow_with_the_layers(lib):
    t0 = time.perf_counter()
    for _ in range(100):
        lib.march_layers(1, 10_000_000, 304)
    assert time.perf_counter() - t0 < 0.5
