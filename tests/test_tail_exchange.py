"""The cluster tail's exchanges (ddc-svd_gb300/csrc/tail.cu) under any delivery
order: a model of its CTAs, records and mbarriers in which every remote store
may arrive as late as the barriers allow.  A wait must end with all of its
column's records there, and no record may overwrite one still to be read."""
import os
import random
import re

import pytest

TAIL = os.path.join(os.path.dirname(__file__), "..", "ddc-svd_gb300", "csrc", "tail.cu")


def ex1_bars():
    with open(TAIL) as f:
        return int(re.search(r"constexpr int kEx1Bars = (\d+);", f.read()).group(1))


class Barrier:
    """One arrival and a transaction count per phase (mbarrier, expected count 1)."""

    def __init__(self):
        self.phase, self.pending, self.tx = 0, 1, 0

    def _flip(self):
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, 1

    def arm(self, n):
        self.tx += n
        self.pending -= 1
        self._flip()

    def complete(self, n):
        self.tx -= n
        self._flip()


def run(C, slices, cols_per_slice, bars, rng):
    """One schedule; returns what went wrong, or None.  CTA s owns slice s; a column of
    slice s is live until it is factored."""
    nt = slices * cols_per_slice
    bar1 = [[Barrier() for _ in range(bars)] for _ in range(C)]
    bar2 = [Barrier() for _ in range(C)]
    rec1 = [[{}, {}] for _ in range(C)]  # by column parity: sender -> column
    rec2 = [{} for _ in range(C)]
    col, step = [0] * C, ["send"] * C
    flight = []

    def first_live(i):
        return (i + 1) // cols_per_slice

    while any(i < nt for i in col):
        ready = [k for k in range(C) if col[k] < nt and (
            step[k] == "send"
            or (step[k] == "wait1" and bar1[k][col[k] % bars].phase > col[k] // bars)
            or (step[k] == "wait2" and bar2[k].phase > col[k]))]
        # an old record may be held back for long: late ones are delivered last, mostly
        moves = ready * 8 + (["deliver"] if flight else [])
        if not moves:
            return "deadlock"
        mv = rng.choice(moves)
        if mv == "deliver":
            q = min(len(flight) - 1, int(len(flight) * rng.random() ** 0.3))
            kind, src, dst, i = flight.pop(q)
            # the record before it in the place is read until its reader sends the next column's
            sent = i - 1 if kind == 1 else i
            if i >= 2 and (col[dst], step[dst] != "send") < (sent, True):
                return "record overwritten before it was read"
            if kind == 1:
                rec1[dst][i % 2][src] = i
                bar1[dst][i % bars].complete(8)
            else:
                rec2[dst][src] = i
                bar2[dst].complete(8)
            continue
        k, i = mv, col[mv]
        owners = range(first_live(i), slices)
        if step[k] == "send":
            bar1[k][i % bars].arm(8 * C)
            if i < nt - 1:
                bar2[k].arm(8 * len(owners))
            flight += [(1, k, d, i) for d in range(C)]
            step[k] = "wait1"
        elif step[k] == "wait1":
            if any(rec1[k][i % 2].get(s) != i for s in range(C)):
                return "wait of exchange 1 over before its records were there"
            if i < nt - 1 and k in owners:
                flight += [(2, k, d, i) for d in range(C)]
            if i == nt - 1:
                col[k] = nt
            step[k] = "wait2"
        else:
            if any(rec2[k].get(s) != i for s in owners):
                return "wait of exchange 2 over before its records were there"
            col[k], step[k] = i + 1, "send"
    return None


SHAPES = [(3, 1, 8), (4, 2, 4), (4, 4, 3), (8, 3, 3)]


@pytest.mark.parametrize("C,slices,width", SHAPES)
def test_waits_end_with_their_records(C, slices, width):
    rng = random.Random(C * 100 + slices)
    bad = {run(C, slices, width, ex1_bars(), rng) for _ in range(800)} - {None}
    assert not bad, bad


def test_model_finds_the_gap_of_a_single_barrier():
    """One barrier for both parities: a record of the next column completes the phase of a
    CTA without a slice, for which nobody waited."""
    rng = random.Random(1)
    assert "wait of exchange 1 over before its records were there" in {run(3, 1, 8, 1, rng) for _ in range(800)}
