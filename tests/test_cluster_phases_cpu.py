"""The phases of a cluster's sums (csrc/cluster_phase.h), on a model of the
mbarriers, slots and messages of kernels_pcg_resident.cu.

The model interleaves the CTAs' steps and the deliveries of their messages in
every order (two CTAs) or in random ones (four).  A phase's sum must be that of
the phase's own messages, no row is published while a copy of it is under way,
and no CTA may wait for ever.  Every CTA may give up a wait: then all come to
the end, and nothing is sent to one that has left.  The number of messages and
the bytes that a phase expects come from the kernel's header.
"""
import ctypes as C
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "fortfem_b200", "csrc")


@pytest.fixture(scope="module")
def header(tmp_path_factory):
    d = tmp_path_factory.mktemp("phase")
    src, so = d / "phase.cpp", d / "phase.so"
    src.write_text('#include "cluster_phase.h"\n'
                   'extern "C" int messages(int nv) { return ffg::phase_messages(nv); }\n'
                   'extern "C" unsigned bytes(int nv, int n, unsigned c) '
                   '{ return ffg::phase_bytes(nv, n, c); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(src), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    return lib.messages, lambda nv, n, copied: lib.bytes(nv, n, C.c_uint(copied))


COPY = 128  # bytes of a copied slice


class Model:
    """n CTAs that run the same program, a list of
      S0 S1 S2  a phase of that many sums;
      X0 X1 X2  the same with the exchange: CTA c copies a slice to CTA c + 1 alone;
      P         publish: the source of the copies is written;
      B         the barrier, of messages as well;
      H         a barrier that pairs with the one at a CTA's end (barrier.cluster).
    Steps of a phase: send (arrive with the expected bytes, a message to every CTA
    and the copy), wait, read.  States are plain tuples, so that they can be hashed.
    give_up: the first CTA may give up any wait, and once it has, so may the others."""

    def __init__(self, n, program, messages, bytes_, give_up=False):
        self.n, self.program, self.give_up = n, program.split(), give_up
        self.messages, self.bytes = messages, bytes_
        self.end = len(self.program)

    def start(self):
        # per CTA: (operation, step, phase, barrier), two mbarriers of the phases and
        # two of the barriers (completed, pending, bytes), two slot sets of n phases;
        # what is in flight.  Operations: the program's, its end (gave up: step 1),
        # and then left the kernel.
        cta = ((0, 0, 1, 1), ((0, 1, 0),) * 2 + ((0, self.n, 0),) * 2, ((0,) * self.n,) * 2)
        return (cta,) * self.n, ()

    def done(self, state):
        return all(c[0][0] >= self.end for c in state[0])

    def _bar(self, bars, par, arrive, tx):
        done, pending, left = bars[par]
        pending, left = pending - arrive, left + tx
        if pending == 0 and left == 0:
            done, pending = done + 1, 1 if par < 2 else self.n
        new = list(bars)
        new[par] = (done, pending, left)
        return tuple(new)

    def moves(self, state):
        """The states that one step of a CTA or one delivery leads to."""
        ctas, flight = state
        given = any(o[0][:2] == (self.end, 1) or o[0][0] > self.end for o in ctas)
        for c in range(self.n):
            (at, step, k, b), bars, slots = ctas[c]
            if at >= self.end:
                continue
            op, sent, last, others = self.program[at], flight, False, ctas
            nv, par = int(op[1]) if len(op) > 1 else 0, k % 2
            if step == 1 and self.give_up and op != "H" and (c == 0 or given):
                yield (ctas[:c] + (((self.end, 1, k, b), bars, slots),) + ctas[c + 1:], flight)
            if step == 0 and op in ("S0", "S1", "S2", "X0", "X1", "X2", "B"):
                assert all(o[0][0] <= self.end for o in ctas), f"CTA {c} sends to one that left"
            if op == "P":
                assert given or not any(f[0] == "copy" and f[2] == c for f in flight), \
                    f"CTA {c} overwrites what is being copied (operation {at})"
                last = True
            elif op == "B":
                if step == 0:
                    sent = flight + tuple(("here", d, c, b) for d in range(self.n))
                elif bars[2 + b % 2][0] % 2 == ((b - 1) >> 1) % 2:
                    continue
                else:
                    b, last = b + 1, True
            elif op == "H":
                if step == 1:
                    if any(o[0][0] < self.end and o[0][:2] < (at, 1) for o in ctas):
                        continue
                    # whoever was at its end is free to leave
                    others = tuple((((self.end + 1,) + o[0][1:],) + o[1:])
                                   if o[0][0] == self.end else o for o in ctas)
                    last = True
            elif step == 0:
                copies = ()
                if op[0] == "X":
                    copies = (("copy", (c + 1) % self.n, c, k),)
                    assert not any(f[:3] == copies[0][:3] for f in flight), \
                        f"two copies of CTA {c} to one place (operation {at})"
                bars = self._bar(bars, par, 1, self.bytes(nv, self.n, COPY * len(copies)))
                sent = flight + copies + tuple(
                    ("sum", d, c, k) for d in range(self.n)) * self.messages(nv)
            elif step == 1:
                # try_wait.parity: true while the barrier is in the other parity
                if bars[par][0] % 2 == ((k - 1) >> 1) % 2:
                    continue
            else:
                assert nv == 0 or all(g == k for g in slots[par]), \
                    f"CTA {c} sums {slots[par]} in phase {k}"
                k, last = k + 1, True
            pos = (at + 1, 0, k, b) if last else (at, step + 1, k, b)
            yield others[:c] + ((pos, bars, slots),) + others[c + 1:], tuple(sorted(sent))
        for i, (kind, d, c, k) in enumerate(flight):
            if i and flight[i - 1] == flight[i]:
                continue
            pos, bars, slots = ctas[d]
            if kind == "sum":
                row = list(slots[k % 2])
                row[c] = k
                slots = (tuple(row), slots[1]) if k % 2 == 0 else (slots[0], tuple(row))
            if kind == "here":
                bars = self._bar(bars, 2 + k % 2, 1, 0)
            else:
                bars = self._bar(bars, k % 2, 0, -8 if kind == "sum" else -COPY)
            yield ctas[:d] + ((pos, bars, slots),) + ctas[d + 1:], flight[:i] + flight[i + 1:]

    def explore(self):
        todo, seen = [self.start()], set()
        while todo:
            s = todo.pop()
            if s in seen:
                continue
            seen.add(s)
            after = list(self.moves(s))
            assert after or self.done(s), f"nothing can move: {s}"
            todo.extend(after)
        return len(seen)

    def walk(self, rng):
        s = self.start()
        while not self.done(s) or s[1]:
            after = list(self.moves(s))
            assert after, f"nothing can move: {s}"
            s = rng.choice(after)


# The cluster's loops in kernels_pcg_resident.cu, the published vector replicated.
LOOPS = {
    # residual norms, (r, z); then two iterations
    "fp64": "S2 S1 P X0 S1 S2 P X0 S1 S2",
    "mixed": "S2 P X1 S1 P X2 S1 P X2",
    # an iteration, its reliable update, the next iteration
    "update": "P X1 S1 P X2 B P X0 S1 P X1 S1 P X2",
    # the update that changes to the direct form, an iteration, an update in it
    "direct": "P X1 S1 P X2 B P X0 S1 S1 P X0 S1 S2 B S1 S1 P X0 S1 S2",
    # the change to the FP64 loop (two barriers on end), its vector in global memory
    "global": "X1 S1 X2 B B S2 B S1 S2 B S1 S2 B B B S1",
}


@pytest.mark.parametrize("loop", LOOPS)
def test_every_interleaving_of_two_ctas(header, loop):
    assert Model(2, LOOPS[loop], *header).explore() > 100


@pytest.mark.parametrize("loop", LOOPS)
def test_every_interleaving_with_waits_given_up(header, loop):
    assert Model(2, LOOPS[loop], *header, give_up=True).explore() > 100


@pytest.mark.parametrize("loop", LOOPS)
def test_random_interleavings_of_four_ctas(header, loop):
    rng = random.Random(len(loop))
    for _ in range(60):
        Model(4, LOOPS[loop], *header).walk(rng)


def test_the_model_finds_the_phase_that_waits_for_nobody():
    """Without a message in a phase of no sums, a CTA overtakes another by two."""
    quiet = Model(3, "S2 S0 S1 S2", lambda nv: nv, lambda nv, n, copied: 8 * nv * n + copied)
    with pytest.raises(AssertionError, match="sums"):
        quiet.explore()


@pytest.mark.parametrize("loop", ["S1 P X2 P X0 B S1 P X1 S1 P X2",   # p published at once
                                  "P X0 S1 P X1 P X0 S1 S2"])         # z copied, then p
def test_the_model_finds_a_publish_during_the_copies(header, loop):
    with pytest.raises(AssertionError, match="cop"):
        Model(2, loop, *header).explore()


def test_the_model_finds_a_barrier_that_lets_a_cta_leave(header):
    with pytest.raises(AssertionError, match="left"):
        Model(2, LOOPS["update"].replace("B", "H"), *header, give_up=True).explore()
