"""The split of the conversion kernel's work over the SMs: host arithmetic, compiled with the host compiler alone."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ferrograd_b200", "csrc")
SHIM = """
#include "conv_plan.cuh"
extern "C" {
uint64_t sms_beside(int sms, int exchange, int reserved) { return fg_sms_beside(sms, exchange != 0, reserved); }
uint64_t grid(uint64_t units, uint32_t split, uint64_t sms) { return conv_grid(units, split, sms); }
// one product (N2 = 0) or two; clusters of any size fill the SMs
double plan(uint32_t M, uint32_t N, uint32_t K, uint32_t batch, uint32_t N2, uint32_t K2, uint64_t sms, uint64_t all, uint32_t* bn, uint32_t* split) {
    const ConvShape sh[2] = {{M, N, K, batch}, {M, N2, K2, batch}};
    const ConvPlan p = conv_plan(sh, N2 ? 2 : 1, sms, [&](uint32_t, uint32_t s) { return conv_clusters_beside((int)(all / s), sms, all); });
    *bn = p.bn; *split = p.split;
    return p.cycles;
}
uint32_t fixed(uint32_t K, uint32_t K2, uint32_t split, uint32_t largest) {
    const ConvShape sh[2] = {{128, 128, K, 1}, {128, 128, K2, 1}};
    return conv_plan_fixed(sh, K2 ? 2 : 1, 64, split, [&](uint32_t, uint32_t s) { return s <= largest ? 9 : 0; }).split;
}
std::atomic<int> known[2];
int asked_once(int which, int answers, int value, int* asked) {
    return fg_asked_once(known[which], -7, [&](int* n) { ++*asked; *n = value; return answers != 0; });
}
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("conv_plan")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "shim.so"), str(d / "shim.cpp")], check=True)
    lib = C.CDLL(str(d / "shim.so"))
    lib.sms_beside.restype = lib.grid.restype = C.c_uint64
    lib.grid.argtypes = [C.c_uint64, C.c_uint32, C.c_uint64]
    lib.plan.restype = C.c_double
    lib.plan.argtypes = [C.c_uint32] * 6 + [C.c_uint64] * 2 + [C.c_void_p] * 2
    return lib


def plan(lib, M, N, K, sms, batch=1, second=(0, 0)):
    bn, split = C.c_uint32(), C.c_uint32()
    cycles = lib.plan(M, N, K, batch, *second, sms, 148, C.byref(bn), C.byref(split))
    return bn.value, split.value, cycles


def test_a_running_exchange_keeps_its_sms(shim):
    # persistent CTAs take an SM each: with 16 of 148 held by the exchange, 132 of them walk all units
    assert shim.sms_beside(148, 0, 16) == 148 and shim.sms_beside(148, 1, 0) == 148
    free = shim.sms_beside(148, 1, 16)
    assert free == 132
    for units in (1, 131, 132, 133, 148, 149, 4000):
        assert shim.grid(units, 1, free) == min(units, 132)
        assert shim.grid(units, 1, 148) == min(units, 148)
    assert shim.grid(20, 5, free) == 100          # clusters do not walk: one for each unit


def test_the_plan_counts_the_sms_that_are_left(shim):
    # 140 tiles of 128 x 128 are one round of 148 SMs and two of 132
    M, N, K = 128 * 10, 128 * 14, 1024
    whole, beside = plan(shim, M, N, K, 148), plan(shim, M, N, K, 132)
    assert whole[:2] == (128, 1) and beside[2] > whole[2]
    # shares: two for each SM at most
    for tiles in range(1, 80):
        for sms in (148, 132):
            bn, split, _ = plan(shim, 128 * tiles, 128, 4096, sms)
            assert split == 1 or tiles * (128 // bn) * split <= 2 * sms


@pytest.mark.parametrize("sms", [148, 132, 2, 1])
def test_every_shape_has_a_plan(shim, sms):
    for M in (1, 128, 129, 5000):
        for N in (1, 64, 65, 4097):
            for K in (1, 32, 128, 129, 70000):
                for batch in (1, 7):
                    for second in ((0, 0), (N, 1), (3 * N, K)):
                        bn, split, cycles = plan(shim, M, N, K, sms, batch, second)
                        shortest = min(K, second[1]) if second[0] else K
                        assert bn in (64, 128) and cycles > 0
                        assert split == 1 or 2 * split <= (shortest + 31) // 32        # two k-blocks for every share


def test_given_shares_shrink_to_what_can_run(shim):
    # two k-blocks of 32 for each share, of the shorter k; clusters that can be launched
    assert shim.fixed(512, 0, 8, 8) == 8 and shim.fixed(480, 0, 8, 8) == 7 and shim.fixed(512, 130, 8, 8) == 2
    assert shim.fixed(32, 0, 5, 8) == 1 and shim.fixed(4096, 4096, 8, 4) == 4


def test_a_query_that_failed_is_asked_again(shim):
    # an answer is kept, zero too; a failure is not: the next call asks again
    asked = C.c_int(0)
    ask = lambda which, answers, value: shim.asked_once(which, answers, value, C.byref(asked))          # noqa: E731
    assert ask(0, 0, 5) == -7 and ask(0, 0, 5) == -7 and asked.value == 2
    assert ask(0, 1, 5) == 5 and asked.value == 3
    assert ask(0, 1, 9) == 5 and ask(0, 0, 9) == 5 and asked.value == 3
    assert ask(1, 1, 0) == 0 and ask(1, 1, 3) == 0 and asked.value == 4


# Of a few k-blocks and more than one unit per CTA, what a unit waits for is the store of its tile: narrow tiles where they take fewer of those
# in all, wide ones where a wide tile per CTA is all there is, or the k is long.
@pytest.mark.parametrize("M,N,K,width", [(15064, 400, 1, 64), (4390, 632, 2, 64), (3520, 744, 3, 64), (1920, 1384, 96, 64), (4096, 512, 32, 128),
                                         (6000, 256, 32, 128), (2048, 1024, 1024, 128)])
def test_the_width_of_a_short_k(shim, M, N, K, width):
    assert plan(shim, M, N, K, 148)[:2] == (width, 1)
