"""The ordering rules of the sparse exchange, replayed without a GPU: the edges
that the planner returns (the communicator emits exactly these) are carried out
on model streams whose history is the set of operations that precede their next
one, for every interleaving of selections and exchange halves with at most two
open, on one rank and on more, alone and among half-precision exchanges."""
import ctypes as C
import itertools

import pytest

from singa_b200 import _lib

SELECT, EXCHANGE, LOCAL, SYNCH_HALF, FLUSH_HALF, WAIT = 16, 17, 18, 4, 3, 7
# bit: (source, target); marks and waits of a slot's events are written out below
EDGES = [("compute", "c1"), ("compute", "s"), ("c1", "s"), None, ("s", "c1"), ("s", "c2"), ("s", "compute"),
         ("c1", "compute"), ("c2", "compute")]


class Model(object):
    def __init__(self):
        self.state = (C.c_ubyte * 4)()
        self.streams = {k: set() for k in ("compute", "c1", "s", "c2")}
        self.events = {"c2done": set()}
        self.slots = [0, 0]                       # of the next selection / exchange half

    def plan(self, call):
        edges = (C.c_uint * 4)()
        assert _lib.lib().sgb_comm_order_plan(self.state, call, edges, None) == 0
        return list(edges)

    def emit(self, bits, slot=0):
        st, ev = self.streams, self.events
        for k, edge in enumerate(EDGES):
            if edge and bits >> k & 1:
                st[edge[1]] |= st[edge[0]]
        if bits & 8:
            st["s"] |= ev["c2done"]
        if bits & 512:
            ev["c2done"] = set(st["c2"])
        if bits & 16384:
            st["c1"] |= ev["consumed", slot]
        if bits & 1024:
            ev["selected", slot] = set(st["c1"])
        if bits & 2048:
            st["s"] |= ev["selected", slot]
        if bits & 4096:
            st["c2"] |= ev["selected", slot]
        if bits & 8192:
            ev["consumed", slot] = set(st["c2"])

    def run(self, stream, op):
        before = set(self.streams[stream])
        self.streams[stream].add(op)
        return before

    def select(self, k):
        slot, self.slots[0] = self.slots[0], 1 - self.slots[0]
        pre, before, after, post = self.plan(SELECT)
        assert before == after == 0
        self.run("compute", ("produced", k))
        self.emit(pre, slot)
        seen = self.run("c1", ("select", k))
        assert ("produced", k) in seen
        if k >= 2:                                # the slot's payload has been sent, or read in place
            assert ("gather", k - 2) in seen or ("dense", k - 2) in seen
        self.emit(post, slot)

    def exchange(self, k, local):
        slot, self.slots[1] = self.slots[1], 1 - self.slots[1]
        pre, before, after, post = self.plan(LOCAL if local else EXCHANGE)
        assert pre == 0
        later = ("select", k + 1) in self.streams["c1"]
        self.emit(before, slot)
        if not local:
            seen = self.run("s", ("gather", k))
            assert ("select", k) in seen
            assert not later or ("select", k + 1) not in seen        # only its own selection
            assert k == 0 or ("dense", k - 1) in seen                # the receive buffer is free
        self.emit(after, slot)
        seen = self.run("c2", ("dense", k))
        assert ("select", k) in seen and (local or ("gather", k) in seen)
        assert not (local and later) or ("select", k + 1) not in seen
        self.emit(post, slot)

    def half(self, call):
        pre, before, after, post = self.plan(call)
        self.emit(pre)
        self.run("c1", ("cast",))
        self.emit(before)
        self.run("s", ("reduce",))
        self.emit(after)
        self.run("c2", ("widen",))
        self.emit(post)

    def wait(self):
        pre, before, after, post = self.plan(WAIT)
        self.emit(before)
        everything = set().union(*self.streams.values())
        assert self.streams["compute"] == everything
        self.slots = [0, 0]
        assert list(self.state) == [0, 0, 0, 0]


def interleavings(n):
    for seq in itertools.product("SE", repeat=2 * n):
        opened = 0
        for step in seq:
            opened += 1 if step == "S" else -1
            if not 0 <= opened <= 2:
                break
        else:
            if seq.count("S") == n:
                yield seq


@pytest.mark.parametrize("local", [True, False])
@pytest.mark.parametrize("among", [None, SYNCH_HALF, FLUSH_HALF])
def test_every_interleaving(local, among):
    count = 0
    for n in (1, 2, 3, 5):
        for seq in interleavings(n):
            m = Model()
            for _ in range(2):                    # a second step behind the wait
                begun = ended = 0
                for step in seq:
                    if step == "S":
                        m.select(begun)
                        begun += 1
                    else:
                        m.exchange(ended, local)
                        ended += 1
                        if among is not None:
                            m.half(among)
                m.wait()
                m.streams = {k: set() for k in m.streams}
                m.events = {k: set() for k in m.events}
            count += 1
    assert count == 1 + 2 + 4 + 16


def test_one_call_is_the_two_halves():
    lib = _lib.lib()
    a, b = (C.c_ubyte * 4)(0, 0, 0, 1), (C.c_ubyte * 4)(0, 0, 0, 1)
    one, sel, exc, res = (C.c_uint * 4)(), (C.c_uint * 4)(), (C.c_uint * 4)(), C.c_int()
    assert lib.sgb_comm_order_plan(a, 5, one, C.byref(res)) == 0 and res.value == 2
    assert lib.sgb_comm_order_plan(b, SELECT, sel, C.byref(res)) == 0 and res.value == 1
    assert lib.sgb_comm_order_plan(b, EXCHANGE, exc, C.byref(res)) == 0 and res.value == 2
    assert list(a) == list(b)
    assert list(one) == [sel[0] | sel[3], exc[1], exc[2], exc[3]] and exc[1] & 8
    for call in (8, 15, 19, -1):
        assert lib.sgb_comm_order_plan(a, call, one, None) != 0
