"""The waits of the fixed-point kernels' cutters on the `finished` barriers (fx_turns.h,
used by fx.cuh), walked through every order of events.

A cutter warp hands over the products of a launch one by one; the finishers complete
them in order, any time after.  Before product n the cutter waits for the earlier ones
by the parity of a phase: the wait ends if the phase that the barrier is in has the
other parity.  Checked at every wait, for every number of products that the
finishers may have completed by then and may complete later without this cutter: the
wait ends exactly when its product is finished, so that it neither ends early nor lasts
for good.
"""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parament_gb300", "csrc")

SHIM = r"""
#include "fx_turns.h"
extern "C" {
uint32_t bars() { return pgb::fx::kFinishedBars; }
uint32_t bar(uint32_t n) { return pgb::fx::finished_bar(n); }
uint32_t parity(uint32_t n) { return pgb::fx::finished_parity(n); }
uint32_t before(uint32_t n, int needs) { return pgb::fx::finished_before(n, needs != 0); }
}
"""


class OneBarrier:
    """All products on one barrier."""
    @staticmethod
    def bars():
        return 1

    @staticmethod
    def bar(n):
        return 0

    @staticmethod
    def parity(n):
        return n & 1

    @staticmethod
    def before(n, needs):
        return 0 if n == 0 else n - (0 if needs else 1)


@pytest.fixture(scope="module")
def turns(tmp_path_factory):
    d = tmp_path_factory.mktemp("turns")
    src, so = d / "t.cpp", d / "t.so"
    src.write_text(SHIM)
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)])
    return ctypes.CDLL(str(so))


def walk(t, products, needs):
    """The waits that would end early or never, as (n, product waited for, finished)."""
    wrong, seen = [], 0
    for n in range(products):
        for p in range(seen, t.before(n, needs(n))):
            # p products at least are finished (the waits before), n at most.
            for done in range(p, n + 1):
                phase = sum(1 for q in range(done) if t.bar(q) == t.bar(p))  # phases completed
                ended = (phase & 1) != t.parity(p)
                if ended != (done > p):
                    wrong.append((n, p, done))
        seen = max(seen, t.before(n, needs(n)))
    return wrong


ORDERS = {"independent": lambda n: False, "each needs the last": lambda n: True, "mixed": lambda n: n % 5 in (1, 2),
          "one at the end": lambda n: n > 20}


@pytest.mark.parametrize("order", ORDERS)
def test_every_wait_ends_when_its_product_is_finished(turns, order):
    assert walk(turns, 40, ORDERS[order]) == []


def test_one_barrier_would_not_do():
    assert walk(OneBarrier, 40, ORDERS["independent"])


def test_the_kernels_use_these_turns():
    src = open(os.path.join(CSRC, "fx.cuh")).read()
    assert "finished[kFinishedBars]" in src
    assert src.count("s.finished[finished_bar(") == 2
    assert "finished_parity(seen)" in src and "finished_before(n, " in src
