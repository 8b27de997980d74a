"""How calls with host buffers are ordered (awesome-cute_b200/csrc/w4a16_host_chain.h), against a model of the stream.

The model knows of every kernel when it may start and when it lets its successor start, and so which earlier kernels may still
be running when it touches its buffers.  Random sequences of host-buffer calls, GEMMs on device buffers and work of other
origin, over a handful of buffers and from one or several threads, must never touch what a kernel that may still be running
reads or writes."""
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


class Place(ctypes.Structure):
    _fields_ = [("dev", ctypes.c_int), ("stream", ctypes.c_void_p), ("id", ctypes.c_ulonglong), ("capture", ctypes.c_ulonglong)]


def library():
    if not os.path.exists(LIB):
        entry._make(os.path.dirname(LIB))
    lib = ctypes.CDLL(LIB)
    vp, ci, u64, bp, pp = ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64, ctypes.POINTER(Buffers), ctypes.POINTER(Place)
    lib.chain_new.restype = vp
    lib.chain_delete.argtypes = [vp]
    lib.chain_order.argtypes = [vp, pp, u64, bp]
    lib.chain_record.argtypes = [vp, pp, u64, u64, ci, bp]
    lib.chain_forget.argtypes = [vp, pp]
    return lib


class Race(Exception):
    pass


def clash(a, b):
    return any(x < y + m and y < x + n for x, n in a for y, m in b)


class Call:
    """A call of one thread: when it began and, once it has returned, when it did."""

    def __init__(self, began=0):
        self.began, self.returned = began, None


class Stream:
    """One stream.  A kernel: the earlier kernels that are over when it starts, and when it lets its successor start.  Only
    what calls that had returned before a call began have launched is in order with that call."""

    def __init__(self, first_signals="after its wait"):
        self.kernels = []           # (reads, writes, over at its start, signal, call)
        self.first_signals = first_signals
        self.call = Call()          # the call that launches

    def launch(self, reads, writes, signal, access="after its wait", ordinary=False):
        i = len(self.kernels)
        everything = set(range(i))
        over = everything
        if i and not ordinary:      # programmatic launch: starts when the one before lets it
            _, _, before, sig, _ = self.kernels[-1]
            over = before if sig == "at its start" else set(range(i - 1)) if sig == "after its wait" else everything
        # (a kernel that has waited has waited for everything before it: none ends before it has)
        for j in everything - (over if access == "at its start" else everything):
            r, w, _, _, call = self.kernels[j]
            ordered = call is self.call or call.returned is not None and call.returned <= self.call.began
            if ordered and (clash(reads, w) or clash(writes, r) or clash(writes, w)):
                raise Race("kernel %d touches what kernel %d, possibly unfinished, uses" % (i, j))
        self.kernels.append((reads, writes, over, signal, self.call))

    def copy_in(self, how, b):
        self.launch([(b.a_host, b.a_bytes)], [(b.a_stage, b.a_bytes)], self.first_signals if how == FIRST else "at its start",
                    "at its start" if how == EARLY else "after its wait")

    def gemm(self, b):
        self.launch([(b.a_stage, b.a_bytes)], [(b.c_stage, b.c_bytes), (b.c_host, b.c_bytes)], "at its start")

    def mul(self, a, c):
        self.launch([a], [c], "at its start")

    def other(self, a, c):
        self.launch([a], [c], "at its end", ordinary=True)


class Library:
    """The library's side: the process's counter and the chain.  host() and mul() are one call each, step by step."""

    def __init__(self, lib, streams):
        self.lib, self.chain, self.streams, self.count = lib, lib.chain_new(), streams, 0
        self.clock = 0
        self.taken = []

    def __del__(self):
        self.lib.chain_delete(self.chain)

    def tick(self):
        self.clock += 1
        return self.clock

    def place(self, stream, capture=0):
        return Place(0, stream + 1, 0 if capture else 1, capture)

    def on(self, stream, call):
        self.streams[stream].call = call
        return self.streams[stream]

    def host(self, stream, b):
        call = Call(self.tick())
        seen = self.count
        how = self.lib.chain_order(self.chain, self.place(stream), seen, b)
        self.taken.append(how)
        yield
        self.on(stream, call).copy_in(how, b)
        yield
        self.count += 1
        yield
        self.on(stream, call).gemm(b)
        yield
        self.count += 1
        yield
        self.lib.chain_record(self.chain, self.place(stream), seen, self.count, how, b)
        self.count += 1
        call.returned = self.tick()

    def mul(self, stream, a, c):
        call = Call(self.tick())
        self.count += 1
        yield
        self.on(stream, call).mul(a, c)
        yield
        self.count += 1
        call.returned = self.tick()

    def other(self, stream, a, c):
        call = Call(self.tick())
        self.on(stream, call).other(a, c)
        call.returned = self.tick()
        yield

    def run(self, call):
        for _ in call:
            pass


def layer(i, o, size=64):
    """A call that reads host buffer i and writes host buffer o, with staging buffers of its own unless i or o say so."""
    return Buffers(0x1000 * (1 + i), 0x100000 + 0x1000 * i, 0x200000 + 0x1000 * o, 0x1000 * (1 + o), size, size)


def sequence(lib, seed, threads=1, streams=1, **kw):
    """Every thread makes its calls one after the other; the threads' steps are interleaved at random."""
    rng = random.Random(seed)
    host = [0x1000 * i for i in range(1, 9)]
    dev = [0x100000 + 0x1000 * i for i in range(1, 9)]
    few = rng.choice([3, 8])
    pick = lambda pool: (rng.choice(pool[:few]) + rng.choice([0, 0, 0, 32]), 64)
    library = Library(lib, [Stream(**kw) for _ in range(streams)])

    def thread():
        for _ in range(30):
            kind, stream = rng.choice(["host"] * 6 + ["mul", "other"]), rng.randrange(streams)
            if kind == "host":
                yield from library.host(stream, Buffers(pick(host)[0], pick(dev)[0], pick(dev)[0], pick(host)[0], 64, 64))
            else:
                pool = dev if kind == "mul" else host + dev
                yield from getattr(library, kind)(stream, pick(pool), pick(pool))

    running = [thread() for _ in range(threads)]
    while running:
        t = rng.choice(running)
        for _ in range(rng.choice([1, 1, 3, 20])):
            if next(t, t) is t:
                running.remove(t)
                break


@pytest.mark.parametrize("threads,streams", [(1, 1), (1, 2), (2, 1), (2, 2), (3, 2)])
def test_no_call_touches_what_may_be_in_use(threads, streams):
    lib = library()
    for seed in range(1500):
        sequence(lib, seed, threads, streams)


def test_the_model_sees_a_copy_in_that_signals_before_it_waits():
    """Two layers read what a third has written (a fan-out): the first reader's copy-in waits, but had it let its GEMM start
    before, the second reader's copy-in could start while the writer runs."""
    lib = library()
    with pytest.raises(Race):
        for seed in range(300):
            sequence(lib, seed, first_signals="at its start")


def test_what_each_kind_of_sequence_costs():
    lib = library()
    calls = Library(lib, [Stream()])            # layers that share nothing: one call in eight waits first
    for i in range(19):
        calls.run(calls.host(0, layer(2 * i, 2 * i + 1)))
    assert calls.taken == ([FIRST] + [EARLY] * 7) * 2 + [FIRST, EARLY, EARLY]
    calls = Library(lib, [Stream()])            # each reads what the one before has written: the GEMM still prefetches
    for i in range(6):
        calls.run(calls.host(0, layer(i, i + 1)))
    assert calls.taken == [FIRST] + [LATE] * 5
    calls.run(calls.host(0, layer(4, 9)))       # a fan-out: the second reader of a result
    assert calls.taken[-1] == FIRST
    calls = Library(lib, [Stream()])            # four layers over and over, each with buffers of its own
    for i in range(12):
        calls.run(calls.host(0, layer(2 * (i % 4), 2 * (i % 4) + 1)))
    assert calls.taken == [FIRST, EARLY, EARLY, EARLY] * 3
    calls.run(calls.mul(0, (1, 1), (3, 1)))     # a GEMM whose buffers the chain does not know
    for i, want in ((20, FIRST), (22, EARLY)):
        calls.run(calls.host(0, layer(i, i + 1)))
        assert calls.taken[-1] == want
    lib.chain_forget(calls.chain, calls.place(0))
    calls.run(calls.host(0, layer(24, 25)))
    assert calls.taken[-1] == FIRST


def test_a_launch_of_another_thread_in_the_middle_of_a_call():
    """A GEMM that another thread enqueues between a call's own launches and its record is not taken for the call's own."""
    lib = library()
    calls = Library(lib, [Stream()])
    calls.run(calls.host(0, layer(0, 1)))
    for steps in range(1, 6):
        for i in (2, 6):                        # (the first one alone, so that the second finds the chain whole)
            call = calls.host(0, layer(10 * steps + i, 10 * steps + i + 1))
            if i == 6:
                for _ in range(steps):
                    next(call)
                calls.run(calls.mul(0, (0x100000 + 0x1000 * 99, 64), (3, 1)))
            calls.run(call)
        calls.run(calls.host(0, Buffers(0x99000, 0x100000 + 0x1000 * 99, 0x5000000, 0x98000, 64, 64)))
        assert calls.taken[-1] == FIRST, steps


def test_captured_calls_are_not_in_front_of_eager_ones():
    """A call that is captured runs at the graph's launch, not where the chain has seen it: what was open before the capture is
    still open behind it, and the first call after it, as the first call inside it, waits first."""
    lib = library()
    calls = Library(lib, [Stream()])
    calls.run(calls.host(0, layer(0, 1)))
    order = lambda capture, b: lib.chain_order(calls.chain, calls.place(0, capture), calls.count, b)

    def captured(capture, b):
        seen, how = calls.count, order(capture, b)
        calls.count += 2
        lib.chain_record(calls.chain, calls.place(0, capture), seen, calls.count, how, b)
        calls.count += 1
        return how

    assert order(0, layer(2, 3)) == EARLY
    assert [captured(7, layer(i, i + 1)) for i in (4, 6, 7)] == [FIRST, EARLY, LATE]
    assert captured(8, layer(20, 21)) == FIRST
    assert order(0, layer(2, 3)) == FIRST
    assert order(8, layer(2, 3)) == EARLY


def test_a_handle_that_comes_back_is_another_stream():
    lib = library()
    calls = Library(lib, [Stream()])
    calls.run(calls.host(0, layer(0, 1)))
    for place, want in ((Place(0, 1, 1, 0), EARLY), (Place(0, 1, 2, 0), FIRST), (Place(1, 1, 1, 0), FIRST)):
        assert lib.chain_order(calls.chain, place, calls.count, layer(2, 3)) == want
