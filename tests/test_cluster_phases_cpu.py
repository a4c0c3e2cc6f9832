"""The phases of a cluster's sums (csrc/cluster_phase.h), on a model of the
mbarriers, slots and messages of kernels_pcg_resident.cu.

The model interleaves the CTAs' steps and the deliveries of their messages in
every order (two CTAs) or in random ones (four).  A phase's sum must be that of
the phase's own messages, and no CTA may wait for ever.  The number of messages
and the bytes that a phase expects come from the kernel's header.
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
    return lib.messages, lambda nv, n: lib.bytes(nv, n, C.c_uint(0))


class Model:
    """n CTAs that run the same list of phases (their counts of sums), no copies.

    Steps of CTA c in phase k: send (arrive with the expected bytes, one message
    to every CTA), wait, read.  State is a plain tuple so that it can be hashed."""

    def __init__(self, n, phases, messages, bytes_):
        self.n, self.phases, self.messages, self.bytes = n, phases, messages, bytes_

    def start(self):
        # per CTA: (phase, step), two mbarriers (completed, pending, bytes), two
        # slot sets of n phases; the messages in flight
        cta = ((1, 0), ((0, 1, 0), (0, 1, 0)), ((0,) * self.n, (0,) * self.n))
        return (cta,) * self.n, ()

    def done(self, state):
        return all(c[0][0] > len(self.phases) for c in state[0])

    @staticmethod
    def _bar(bars, par, arrive, tx):
        done, pending, left = bars[par]
        pending, left = pending - arrive, left + tx
        if pending == 0 and left == 0:
            done, pending = done + 1, 1
        new = list(bars)
        new[par] = (done, pending, left)
        return tuple(new)

    def moves(self, state):
        """The states that one step of a CTA or one delivery leads to."""
        ctas, flight = state
        for c in range(self.n):
            (k, step), bars, slots = ctas[c]
            if k > len(self.phases):
                continue
            par, nv = k % 2, self.phases[k - 1]
            sent = flight
            if step == 0:
                bars = self._bar(bars, par, 1, self.bytes(nv, self.n))
                sent = flight + tuple((d, c, k) for d in range(self.n)) * self.messages(nv)
            elif step == 1:
                # try_wait.parity: true while the barrier is in the other parity
                if bars[par][0] % 2 == ((k - 1) >> 1) % 2:
                    continue
            else:
                got = slots[par]
                if nv > 0 and any(g != k for g in got):
                    raise AssertionError(f"CTA {c} sums {got} in phase {k}")
            pos = (k, step + 1) if step < 2 else (k + 1, 0)
            yield ctas[:c] + ((pos, bars, slots),) + ctas[c + 1:], tuple(sorted(sent))
        for i, (d, c, k) in enumerate(flight):
            if i and flight[i - 1] == flight[i]:
                continue
            pos, bars, slots = ctas[d]
            row = list(slots[k % 2])
            row[c] = k
            slots = (row, slots[1]) if k % 2 == 0 else (slots[0], row)
            new = (pos, self._bar(bars, k % 2, 0, -8), tuple(map(tuple, slots)))
            yield ctas[:d] + (new,) + ctas[d + 1:], flight[:i] + flight[i + 1:]

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


# sums per phase: the FP64 loop (exchange of p, (p, q), then (r, r) and (r, z)),
# the mixed loop, and a direct one that looks at the wall limit
LOOPS = [[2, 1, 0, 1, 2, 0, 1, 2], [2, 1, 1, 2, 1, 2, 0, 1, 1], [1, 2, 1, 0, 1, 2, 1, 0]]


@pytest.mark.parametrize("phases", LOOPS)
def test_every_interleaving_of_two_ctas_sums_its_own_phase(header, phases):
    assert Model(2, phases, *header).explore() > 100


@pytest.mark.parametrize("phases", LOOPS)
def test_random_interleavings_of_four_ctas(header, phases):
    rng = random.Random(len(phases))
    for _ in range(60):
        Model(4, phases, *header).walk(rng)


def test_the_model_finds_the_phase_that_waits_for_nobody():
    """Without a message in a phase of no sums, a CTA overtakes another by two."""
    quiet = Model(2, LOOPS[0], lambda nv: nv, lambda nv, n: 8 * nv * n)
    with pytest.raises(AssertionError):
        quiet.explore()
