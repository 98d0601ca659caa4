"""Shares of the cycle kernel's CTAs (csrc/cycle_split.h, the functions that the
kernel and its launcher use, compiled here for the host): no right-hand side may
own more nodes per CTA than the chosen instance has room for, whichever others
are still active."""
import ctypes as C
import itertools
import random
import shutil
import subprocess

import pytest

from ultrasound_solver_b200 import build

SOURCE = r"""
#include "cycle_split.h"
using namespace usv;
extern "C" void shape(int bytes, int scenes, const long long* sizes, int nrhs, int sms, int* ctas, int* room) {
    const CycleShape s = cycle_shape(bytes, scenes != 0, sizes, nrhs, sms);
    *ctas = s.ctas;
    *room = s.ctas ? cycle_capacity(bytes, s.instance) : 0;
}
// most nodes per CTA over the active right-hand sides; -1: a CTA is left over or used twice.
// units: 1 for each right-hand side of a single scene, else its nodes
extern "C" int most(const long long* sizes, const long long* units, const unsigned char* active, int nrhs,
                    int ctas) {
    unsigned act = 0, total = 0, seen = 0, before = 0, last = 0;
    for (int b = 0; b < nrhs; ++b)
        if (active[b]) ++act, total += unsigned(units[b]);
    int most = 0;
    for (int b = 0; b < nrhs; ++b)
        if (active[b]) {
            const unsigned first = cycle_first_cta(ctas, act, seen, before, total);
            before += unsigned(units[b]);
            ++seen;
            const unsigned end = cycle_first_cta(ctas, act, seen, before, total);
            if (first != last || end <= first) return -1;
            last = end;
            const int per = cycle_cta_nodes(int(sizes[b]), int(end - first));
            if ((long long)per * (end - first) < sizes[b]) return -1;
            most = per > most ? per : most;
        }
    return last == unsigned(ctas) ? most : -1;
}
extern "C" int segments(int groups, int nodes) { return cycle_segments(groups, nodes); }
extern "C" int task_room(int groups, int capacity) { return cycle_task_room(groups, capacity); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("split")
    (d / "split.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I", str(build.CSRC),
                    str(d / "split.cpp"), "-o", str(d / "split.so")], check=True)
    return C.CDLL(str(d / "split.so"))


def _array(values):
    return (C.c_longlong * len(values))(*values)


def _check(lib, nbytes, sizes, subsets, sms=148, units=None):
    """Shape of the batch, after a look at the given subsets of it."""
    ctas, room = C.c_int(), C.c_int()
    lib.shape(nbytes, 0 if units else 1, _array(sizes), len(sizes), sms, C.byref(ctas), C.byref(room))
    if ctas.value:
        for active in subsets:
            flags = bytes(1 if b in active else 0 for b in range(len(sizes)))
            most = lib.most(_array(sizes), _array(units or sizes), flags, len(sizes), ctas.value)
            assert 0 < most <= room.value, (sizes, sorted(active), most, room.value)
    return ctas.value, room.value


def _all_subsets(count):
    return [set(s) for k in range(1, count + 1) for s in itertools.combinations(range(count), k)]


@pytest.mark.parametrize("nbytes,edges", [
    # a share that grows past the room of the all-active split when a scene leaves
    (4, (12, 42, 64, 64)),
    (4, (12, 81, 63, 69, 42)),
    (4, (34, 52, 23, 33, 59, 8, 44, 40)),
    (8, (15, 42, 49, 74)),
    (8, (10, 40, 35, 35)),
    (16, (10, 33, 28, 45)),
])
def test_room_for_every_active_subset(lib, nbytes, edges):
    ctas, _ = _check(lib, nbytes, [n ** 3 for n in edges], _all_subsets(len(edges)))
    assert ctas > 0


def _orders(rng, sizes, count):
    """Active sets as the right-hand sides leave in the order of size and in random orders."""
    n = len(sizes)
    by_size = sorted(range(n), key=lambda b: sizes[b])
    for order in [by_size, by_size[::-1], *(rng.sample(range(n), n) for _ in range(count))]:
        for k in range(n):
            yield set(order[k:])


def test_room_for_a_batch_of_23_scenes(lib):
    edges = (24, 41, 42, 27, 36, 39, 31, 35, 34, 35, 20, 24, 43, 34, 47, 25, 41, 38, 39, 39, 32, 45, 28)
    sizes = [n ** 3 for n in edges]
    without = [set(range(len(sizes))) - {b} for b in range(len(sizes))]
    ctas, _ = _check(lib, 4, sizes, [*without, *_orders(random.Random(1), sizes, 50)])
    assert ctas > 0


@pytest.mark.parametrize("nbytes", [4, 8, 16])
def test_room_for_random_batches(lib, nbytes):
    rng = random.Random(nbytes)
    taken = 0
    for _ in range(1500):
        count = rng.randint(1, 40)
        top = rng.randint(6, 90)
        sizes = [rng.randint(3, top) * rng.randint(3, top) * rng.randint(3, top) for _ in range(count)]
        ctas, _ = _check(lib, nbytes, sizes, _orders(rng, sizes, 2), sms=rng.choice([148, 148, 132, 64, 8]))
        taken += ctas > 0
    assert taken > 500  # the others are too large, or more right-hand sides than SMs


@pytest.mark.parametrize("nbytes", [4, 8, 16])
def test_room_for_one_scene(lib, nbytes):
    rng = random.Random(nbytes + 1)
    for nrhs in [1, 2, 3, 4, 7, 30, 147, 148, 149]:
        for _ in range(40):
            n = rng.randint(8, 1_250_000 // nrhs)
            ctas, _ = _check(lib, nbytes, [n] * nrhs, [set(range(k)) for k in range(1, nrhs + 1)],
                             units=[1] * nrhs)
            assert ctas == 0 if nrhs > 148 else ctas >= 0


@pytest.mark.parametrize("capacity", [1024, 2048, 4096, 8192, 16384])
def test_room_for_the_sums_of_every_dots_task(lib, capacity):
    """All restarts up to the largest (112: 28 groups of four vectors) and all
    node counts of an instance; lane sums of at most 128 nodes."""
    for restart in range(1, 113):
        most = (restart + 3) // 4
        room = lib.task_room(most, capacity)
        for groups in {1, most // 2 or 1, most - 1 or 1, most}:
            for nodes in {64, 4096, 4160, 8192, 8256, 12288, 12352, capacity - 64, capacity}:
                if nodes <= capacity:
                    segs = lib.segments(groups, nodes)
                    assert groups * segs <= room
                    assert -(-nodes // segs) <= 4096


@pytest.mark.parametrize("nbytes,sizes,scenes,taken", [
    (4, [104 ** 3], False, True), (4, [112 ** 3], False, False), (4, [74 ** 3] * 4, False, False),
    (8, [84 ** 3], False, True), (8, [88 ** 3], False, False), (8, [60 ** 3] * 4, False, False),
    (16, [66 ** 3], False, True), (16, [68 ** 3], False, False), (16, [43 ** 3] * 4, False, False),
    (4, [48 ** 3, 80 ** 3, 64 ** 3] * 2, True, True), (4, [80 ** 3] * 4, True, False),
    (8, [70 ** 3, 70 ** 3, 64 ** 3], True, True), (16, [45 ** 3] * 3 + [40 ** 3], True, False),
])
def test_cycle_kernel_only_where_overlapped_solves_keep_up(lib, nbytes, sizes, scenes, taken):
    """Sizes at which solves on several streams were timed with and without it."""
    ctas, _ = _check(lib, nbytes, sizes, [], units=None if scenes else [1] * len(sizes))
    assert (ctas > 0) == taken
