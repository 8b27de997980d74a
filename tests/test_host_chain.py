"""How calls with host buffers are ordered (awesome-cute_b200/csrc/w4a16_host_chain.h), against a model of the stream.

The model knows of every kernel when it may start and when it lets its successor start, and so which earlier kernels may still
be running when it touches its buffers.  Random sequences of host-buffer calls, GEMMs on device buffers and work of other
origin, over a handful of buffers, must never touch what a kernel that may still be running reads or writes."""
import ctypes
import os
import random

import pytest

import __graft_entry__ as entry

LIB = os.path.join(entry.ROOT, "tests", "cpp", "libhost_chain.so")
FIRST, LATE, EARLY = 0, 1, 2        # enum CopyIn


class Buffers(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in ("a_host", "a_stage", "c_stage", "c_host")] + [
        (n, ctypes.c_size_t) for n in ("a_bytes", "c_bytes")]


def library():
    if not os.path.exists(LIB):
        entry._make(os.path.dirname(LIB))
    lib = ctypes.CDLL(LIB)
    vp, ci, u64, bp = ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64, ctypes.POINTER(Buffers)
    lib.chain_new.restype = vp
    lib.chain_delete.argtypes = [vp]
    lib.chain_order.argtypes = [vp, ci, vp, u64, bp]
    lib.chain_record.argtypes = [vp, ci, vp, u64, ci, bp]
    lib.chain_forget.argtypes = [vp]
    return lib


class Race(Exception):
    pass


def clash(a, b):
    return any(x < y + m and y < x + n for x, n in a for y, m in b)


class Stream:
    """One stream.  A kernel: the earlier kernels that are over when it starts, and when it lets its successor start."""

    def __init__(self, first_signals="after its wait"):
        self.kernels = []           # (reads, writes, over at its start, signal)
        self.first_signals = first_signals

    def launch(self, reads, writes, signal, access="after its wait", ordinary=False):
        i = len(self.kernels)
        everything = set(range(i))
        over = everything
        if i and not ordinary:      # programmatic launch: starts when the one before lets it
            _, _, before, sig = self.kernels[-1]
            over = before if sig == "at its start" else set(range(i - 1)) if sig == "after its wait" else everything
        # (a kernel that has waited has waited for everything before it: none ends before it has)
        for j in everything - (over if access == "at its start" else everything):
            r, w = self.kernels[j][:2]
            if clash(reads, w) or clash(writes, r) or clash(writes, w):
                raise Race("kernel %d touches what kernel %d, possibly unfinished, uses" % (i, j))
        self.kernels.append((reads, writes, over, signal))

    def host_call(self, how, b):
        a_host, a_stage = (b.a_host, b.a_bytes), (b.a_stage, b.a_bytes)
        c_stage, c_host = (b.c_stage, b.c_bytes), (b.c_host, b.c_bytes)
        self.launch([a_host], [a_stage], self.first_signals if how == FIRST else "at its start",
                    "at its start" if how == EARLY else "after its wait")
        self.launch([a_stage], [c_stage, c_host], "at its start")

    def mul(self, a, c):
        self.launch([a], [c], "at its start")

    def other(self, a, c):
        self.launch([a], [c], "at its end", ordinary=True)


class Caller:
    """The library's side: the launch counter and the chain."""

    def __init__(self, lib, stream):
        self.lib, self.chain, self.stream, self.launches = lib, lib.chain_new(), stream, 0
        self.taken = []

    def host(self, b):
        how = self.lib.chain_order(self.chain, 0, 1, self.launches, b)
        self.stream.host_call(how, b)
        self.launches += 1
        self.lib.chain_record(self.chain, 0, 1, self.launches, how, b)
        self.taken.append(how)

    def mul(self, a, c):
        self.stream.mul(a, c)
        self.launches += 1


def layer(i, o, size=64):
    """A call that reads host buffer i and writes host buffer o, with staging buffers of its own unless i or o say so."""
    return Buffers(0x1000 * (1 + i), 0x100000 + 0x1000 * i, 0x200000 + 0x1000 * o, 0x1000 * (1 + o), size, size)


def sequence(lib, seed, **kw):
    rng = random.Random(seed)
    host = [0x1000 * i for i in range(1, 9)]
    dev = [0x100000 + 0x1000 * i for i in range(1, 9)]
    caller = Caller(lib, Stream(**kw))
    few = rng.choice([3, 8])
    for _ in range(30):
        kind = rng.choice(["host"] * 6 + ["mul", "other"])
        pick = lambda pool: rng.choice(pool[:few]) + rng.choice([0, 0, 0, 32])
        if kind == "host":
            caller.host(Buffers(pick(host), pick(dev), pick(dev), pick(host), 64, 64))
        elif kind == "mul":
            caller.mul((pick(dev), 64), (pick(dev), 64))
        else:
            caller.stream.other((pick(host + dev), 64), (pick(host + dev), 64))
    lib.chain_delete(caller.chain)


def test_no_call_touches_what_may_be_in_use():
    lib = library()
    for seed in range(3000):
        sequence(lib, seed)


def test_the_model_sees_a_copy_in_that_signals_before_it_waits():
    """Two layers read what a third has written (a fan-out): the first reader's copy-in waits, but had it let its GEMM start
    before, the second reader's copy-in could start while the writer runs."""
    lib = library()
    with pytest.raises(Race):
        for seed in range(300):
            sequence(lib, seed, first_signals="at its start")


def test_what_each_kind_of_sequence_costs():
    lib = library()
    caller = Caller(lib, Stream())              # layers that share nothing: one call in eight waits first
    for i in range(27):
        caller.host(layer(2 * i, 2 * i + 1))
    assert caller.taken == ([FIRST] + [EARLY] * 7) * 3 + [FIRST, EARLY, EARLY]
    caller = Caller(lib, Stream())              # each reads what the one before has written: the GEMM still prefetches
    for i in range(6):
        caller.host(layer(i, i + 1))
    assert caller.taken == [FIRST] + [LATE] * 5
    caller.mul((1, 1), (3, 1))                  # a GEMM whose buffers the chain does not know
    caller.host(layer(20, 21))
    assert caller.taken[-1] == FIRST
    caller.host(layer(22, 23))
    assert caller.taken[-1] == EARLY
    lib.chain_forget(caller.chain)
    caller.host(layer(24, 25))
    assert caller.taken[-1] == FIRST
