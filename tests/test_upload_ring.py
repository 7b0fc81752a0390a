"""The placement rule of the descriptor rings (csrc/sbg_ring.h), compiled for the
host: over the pushes and launches of division calls of any length, no block is
overwritten while a launch that reads it has not run."""
import ctypes as C
import random
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "simd_bigint_b200" / "csrc"
SHIM = """
#include "sbg_ring.h"
extern "C" int place(sbg::RingSpace* r, size_t bytes, size_t least, size_t* off) { return r->place(bytes, least, off); }
"""
FITS = 0
STEP, JOB, FIX, BASE, COPY = 80, 96, 72, 24, 32      # descriptor bytes, as in sbg_div.cu


class Space(C.Structure):
    _fields_ = [("cap", C.c_size_t), ("head", C.c_size_t)]


@pytest.fixture(scope="module")
def place(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    so = tmp_path_factory.mktemp("ring") / "ring.so"
    subprocess.run([gxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-x", "c++", "-", "-I", str(CSRC), "-o", str(so)],
                   input=SHIM, text=True, check=True)
    fn = C.CDLL(str(so)).place
    fn.argtypes = [C.POINTER(Space), C.c_size_t, C.c_size_t, C.POINTER(C.c_size_t)]
    fn.restype = C.c_int
    return fn


class Ring:
    """Blocks as (offset, end, [launches still to be queued], last launch queued)."""

    def __init__(self, place, least):
        self.place, self.least, self.space, self.blocks = place, least, Space(), []

    def push(self, clock, nbytes, readers):
        """The block of `nbytes` that `readers` later launches read."""
        off = C.c_size_t()
        act = self.place(C.byref(self.space), nbytes, self.least, C.byref(off))
        a, b = off.value, off.value + nbytes
        assert b <= self.space.cap and a % 256 == 0
        if act != FITS:
            clock["drained"] = clock["now"]
        for x in self.blocks:
            hit = act == 2 or (a < x["end"] and x["off"] < b)      # a reallocation takes every block
            if hit and (x["left"] > 0 or x["last"] > clock["drained"]):
                return None
        self.blocks = [x for x in self.blocks if act != 2 and not (a < x["end"] and x["off"] < b)]
        blk = {"off": a, "end": b, "left": readers, "last": 0}
        self.blocks.append(blk)
        return blk


def _launch(clock, blk):
    clock["now"] += 1
    blk["left"] -= 1
    blk["last"] = clock["now"]


def _division(clock, jobs, keep, n, rounds):
    """One batch of n divisions with `rounds` Newton rounds; False where a block
    that is still needed gets overwritten."""
    steps = keep.push(clock, BASE * n + STEP * n * rounds, 1 + 2 * rounds)
    if steps is None:
        return False
    _launch(clock, steps)                             # base cases

    def products():
        blk = jobs.push(clock, JOB * n, 1)
        if blk is not None:
            _launch(clock, blk)
        return blk is not None

    for _ in range(rounds):
        for _ in range(2):
            if not products():
                return False
            _launch(clock, steps)
    fix = keep.push(clock, FIX * n, 2)
    if fix is None:
        return False
    for _ in range(2):
        if not products():
            return False
        _launch(clock, fix)
    for first in range(0, n, 4096):
        blk = jobs.push(clock, COPY * min(4096, n - first), 1)
        if blk is None:
            return False
        _launch(clock, blk)
    return True


def _calls(rng, most):
    return [(int(rng.choice([1, 40, 1000, most]) * rng.uniform(0.5, 1)) + 1, rng.randrange(1, 15)) for _ in range(40)]


@pytest.mark.parametrize("least_jobs,least_keep", [(32 << 20, 4 << 20), (256, 256), (1 << 16, 1 << 20)])
def test_no_block_is_overwritten_before_its_last_reader(place, least_jobs, least_keep):
    for seed in range(20):
        clock = {"now": 0, "drained": 0}
        jobs, keep = Ring(place, least_jobs), Ring(place, least_keep)
        for n, rounds in _calls(random.Random(seed), 100000):
            assert _division(clock, jobs, keep, n, rounds), (seed, n, rounds)


def test_one_ring_for_both_would_overwrite_the_steps(place):
    """What the second ring is for: with one, long batches lose their steps."""
    def ok(n, rounds):
        clock = {"now": 0, "drained": 0}
        ring = Ring(place, 32 << 20)
        return _division(clock, ring, ring, 1, 1) and _division(clock, ring, ring, n, rounds)
    assert ok(1000, 9)
    assert not ok(36000, 5) and not ok(24000, 9)
