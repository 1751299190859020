"""How two products share the workers of one launch: host arithmetic, compiled with the host compiler alone."""
import ctypes as C
import math
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ferrograd_b200", "csrc")
SHIM = """
#include "conv_plan.cuh"
extern "C" double runs(uint64_t pairs, uint64_t n0, double w0, uint64_t n1, double w1, uint32_t* out) {
    const PairRuns r = pair_runs(pairs, n0, w0, n1, w1);
    out[0] = r.extra; out[1] = r.run[0]; out[2] = r.run[1];
    return r.cost;
}
"""


@pytest.fixture(scope="module")
def runs(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair_runs")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "shim.so"), str(d / "shim.cpp")], check=True)
    lib = C.CDLL(str(d / "shim.so"))
    lib.runs.restype = C.c_double
    lib.runs.argtypes = [C.c_uint64, C.c_uint64, C.c_double, C.c_uint64, C.c_double, C.c_void_p]

    def call(pairs, n0, w0, n1, w1):
        out = (C.c_uint32 * 3)()
        return lib.runs(pairs, n0, w0, n1, w1, out), list(out)
    return call


def walk(pairs, n0, n1, extra, run):
    """What every worker does, as the kernel computes it."""
    for p in range(pairs):
        more = p < extra
        first = list(range(p, n0, pairs))
        r0 = p * run[0] if more else extra * run[0] + (p - extra) * run[1]
        yield first, list(range(r0, min(r0 + (run[0] if more else run[1]), n1)))


def test_every_tile_once_and_no_worker_beyond_the_cost(runs):
    rng = random.Random(1)
    for _ in range(400):
        pairs, n0, n1 = rng.choice((1, 2, 66, 74)), rng.randint(1, 700), rng.randint(1, 700)
        w1 = rng.uniform(1, 20)
        w0 = w1 * rng.uniform(1, 8)
        cost, (extra, *run) = runs(pairs, n0, w0, n1, w1)
        seen = [], []
        for a, b in walk(pairs, n0, n1, extra, run):
            seen[0].extend(a)
            seen[1].extend(b)
            assert len(a) * w0 + len(b) * w1 <= cost + 1e-6
        assert sorted(seen[0]) == list(range(n0)) and sorted(seen[1]) == list(range(n1))
        # no smaller cost holds all tiles
        more, less = math.ceil(n0 / pairs) * w0, n0 // pairs * w0
        lower = cost - 1e-6
        if lower > more:
            s0, s1 = int((lower - more) / w1 + 1e-9), int((lower - less) / w1 + 1e-9)
            assert (n0 % pairs) * s0 + (pairs - n0 % pairs) * s1 < n1


def test_the_layer_it_is_for(runs):
    # 128 tiles with twice the k of 256 others on 74 pairs: seven short times, where two launches take four and four
    cost, (extra, *run) = runs(74, 128, 2.0, 256, 1.0)
    assert cost == 7.0 and extra == 54 and run == [3, 5]
