"""The launch rules of csrc/launch_rules.h, compiled for the host, over their
whole range."""
from __future__ import annotations

import ctypes as C
import subprocess
import threading
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "chatcarlo_b200" / "csrc"
SHIM = """
#include "launch_rules.h"
extern "C" int ring_allowed(int ring, int issuers, int regions) { return cc::issue_ring_allowed(ring, issuers, regions); }
extern "C" long long unit_batch(long long batch_size, long long n) { return cc::unit_batch(batch_size, n); }
extern "C" long long batches_of(long long n, long long batch_size) { return cc::batches_of(n, batch_size); }
extern "C" long long units_per_batch(long long batch_size) { return cc::units_per_batch(batch_size); }
extern "C" int unit_at(long long k, long long n, long long batch_size, int n_batches, int group, int shift, long long* out) {
    int slot = -1;
    const int ok = cc::unit_at(k, n, batch_size, n_batches, group, shift, out[0], out[1], slot);
    out[2] = slot;
    return ok;
}
static cc::SmemLimits limits;
static size_t allowed[4];           // what the device would hold, by kernel (a fake of it)
extern "C" size_t allow(long kernel, int device, size_t bytes, int fail) {
    const int e = limits.raise((const void*)kernel, device, bytes, [&](size_t most) {
        if (!fail) allowed[kernel] = most;
        return fail;
    });
    return e ? 0 : allowed[kernel];
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(d / "shim.cpp"), "-o", str(d / "shim.so")],
                   check=True)
    lib = C.CDLL(str(d / "shim.so"))
    for f in (lib.unit_batch, lib.batches_of, lib.units_per_batch):
        f.restype, f.argtypes = C.c_longlong, [C.c_longlong] * (1 if f is lib.units_per_batch else 2)
    lib.allow.restype, lib.allow.argtypes = C.c_size_t, [C.c_long, C.c_int, C.c_size_t, C.c_int]
    lib.unit_at.argtypes = [C.c_longlong] * 3 + [C.c_int] * 3 + [C.c_void_p]
    return lib


class _Bar:
    """An mbarrier of one arrival: a wait by parity passes when the phase in
    progress has the other one."""

    def __init__(self):
        self.done = 0

    def passes(self, parity):
        return self.done & 1 != parity


def _reads_stale_slot(ring, issuers, regions, late, planes=40):
    """The plane-stationary convolution's hand-offs with the loads into the slot
    of plane `late`, from that plane on, landing only when nothing else can
    move: whether an issuer's instructions of some plane read a slot that does
    not hold it."""
    full, empty = [_Bar() for _ in range(ring)], [_Bar() for _ in range(ring)]
    rfull, rfree = [_Bar() for _ in range(regions)], [_Bar() for _ in range(regions)]
    holds = [None] * ring
    load, pending, epi = 0, [], 0
    nxt, seen = list(range(issuers)), [False] * issuers      # an issuer's next plane, and whether its "full" wait is over
    while min(nxt) < planes:
        moved = False
        if load < planes and (load < ring or empty[load % ring].passes((load // ring - 1) & 1)):
            if load >= late and (load - late) % ring == 0:
                pending.append(load)
            else:
                holds[load % ring] = load
                full[load % ring].done += 1
            load += 1
            moved = True
        for w in range(issuers):
            p = nxt[w]
            if p < planes and not seen[w] and full[p % ring].passes((p // ring) & 1):
                seen[w] = moved = True
            if seen[w] and (p < regions or rfree[p % regions].passes((p // regions - 1) & 1)):
                if holds[p % ring] != p:
                    return True
                seen[w] = False
                rfull[p % regions].done += 1
                empty[p % ring].done += 1
                nxt[w] += issuers
                moved = True
        # the epilogue waits for the planes in order; an output is read, and plane epi - 2 released, with plane epi
        if epi < planes and rfull[epi % regions].passes((epi // regions) & 1):
            if epi >= 2:
                rfree[(epi - 2) % regions].done += 1
            epi += 1
            moved = True
        if not moved:
            assert pending, (ring, issuers, regions, late)      # else the hand-offs themselves are stuck
            holds[late % ring] = pending.pop(0)
            full[late % ring].done += 1
    return False


def test_rings_of_alternate_issuers(rules):
    """Two issuing warps on five regions, and one on any: no late load is read
    before it lands on a ring that the rule allows; it is on 3 and 5 planes."""
    for issuers, regions in ((2, 5), (1, 5), (1, 6), (1, 8)):
        for ring in range(2, 13):
            stale = any(_reads_stale_slot(ring, issuers, regions, late) for late in range(30))
            allowed = bool(rules.ring_allowed(ring, issuers, regions))
            assert not (allowed and stale), (ring, issuers, regions)
            assert allowed != (issuers == 2 and ring in (3, 5)), (ring, issuers, regions)
    assert _reads_stale_slot(3, 2, 5, 1) and _reads_stale_slot(5, 2, 5, 1)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000, 10_007, 4_000_000, 2 ** 40])
def test_units_are_bounded_by_the_histories(rules, n):
    """Whatever the batch size, a launch's counter runs over at most
    n / 16 + 2 batches + 1 units."""
    for size in (1, 2, 31, 32, 33, 1000, 200_000, 10 ** 9, 2 ** 62, 2 ** 63 - 1):
        nb = rules.batches_of(n, size)
        assert nb == -(-n // size)
        units = rules.units_per_batch(rules.unit_batch(size, n)) * nb
        assert n <= 32 * units and 16 * units <= n + 32 * nb + 16, (n, size)


@pytest.mark.parametrize("n,size", [(1, 2 ** 62), (33, 10 ** 9), (5_003, 5_003), (5_003, 700), (640, 20), (2_000, 999), (64, 1)])
@pytest.mark.parametrize("group,shift", [(1, 0), (3, 0), (16, 0), (16, 2)])
def test_units_cover_every_history_once(rules, n, size, group, shift):
    """Every history in one unit of its own batch, in that batch's slots."""
    nb, b = rules.batches_of(n, size), rules.unit_batch(size, n)
    out, seen, k = (C.c_longlong * 3)(), [], 0
    while rules.unit_at(k, n, b, nb, group, shift, out):
        first, end, slot = out
        assert 0 <= end - first <= 32
        if end > first:
            assert first // b == (end - 1) // b == slot >> shift
            seen += range(first, end)
        k += 1
    assert k == rules.units_per_batch(b) * nb and sorted(seen) == list(range(n))


def test_shared_memory_limits_only_rise(rules):
    """A launch's own size set between another thread's setting and its launch
    would make that launch fail; a failed setting is not taken for a limit."""
    assert rules.allow(0, 0, 60_000, 0) == 60_000
    assert rules.allow(0, 0, 50_000, 0) == 60_000
    assert rules.allow(0, 0, 90_000, 7) == 0 and rules.allow(0, 0, 70_000, 0) == 70_000
    assert rules.allow(1, 0, 50_000, 0) == 50_000                  # another kernel
    assert rules.allow(0, 1, 55_000, 0) == 55_000                  # another device
    seen = []

    def work(bytes_):
        seen.append(all(rules.allow(2, 0, bytes_, 0) >= bytes_ for _ in range(20_000)))

    threads = [threading.Thread(target=work, args=(b,)) for b in (50_000, 80_000, 60_000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert seen == [True] * 3
