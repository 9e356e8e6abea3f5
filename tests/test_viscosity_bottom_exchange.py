"""The exchange of the viscosity bottom cycle (k_vbottom), run as a model on the
CPU under adversarial orders of warps and messages.

The split of a pass over the cluster's CTAs, the values a pass delivers and the
threads that take part come from the kernel's own header.  The model holds each
CTA's two mbarriers (a phase completes when it has been armed and its bytes are
in; a waiter sees the phase's parity only), the warps, and every value as a
message that may arrive at any later moment.  A run is good when no value
counts on another pass's phase, no barrier is armed twice in a phase, every
warp finds all of a pass's values behind its wait, and all warps reach the end.
"""
import ctypes as C
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BLOCK = 256
SHIM = """
#include "viscosity_split.h"
using namespace uaamg;
extern "C" {
int part_lo(int size, int nc, int j) { return vb_part(size, nc, j).lo; }
int part_cnt(int size, int nc, int j) { return vb_part(size, nc, j).cnt; }
int values(const int* gs, int nc, int g) { return vb_values(gs, nc, g); }
int threads(const int* cnt, int block) { return vb_threads(cnt, block); }
}
"""
PASSES = [0, 1, 2, 3, 4, 5] * 2 + [6] + [5, 4, 3, 2, 1, 0] * 2  # one visit's exchanges; 6: all rows


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    src, lib = d / "shim.cpp", d / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "uaamg_b200", "csrc"), "-o", str(lib),
                    str(src)], check=True)
    return C.CDLL(str(lib))


def starts(sizes):
    gs = [0]
    for s in sizes:
        gs.append(gs[-1] + s)
    return gs


class Plan:
    """What the kernel does for groups of these sizes on nc row CTAs.  words: CTAs without rows send a word and the
    passes count it; warps: only the warps with rows take part, with a barrier over them after each wait."""

    def __init__(self, split, sizes, nc, words=True, warps=True):
        gs = starts(sizes)
        garr = (C.c_int * 7)(*gs)
        self.nc, self.barrier = nc, warps
        cnt = [[split.part_cnt(s, nc, j) for s in sizes] for j in range(nc)]
        for c in cnt:
            c.append(sum(c))
        self.rows = cnt
        self.nwarps = [(split.threads((C.c_int * 6)(*c[:6]), BLOCK) if warps else BLOCK) // 32 for c in cnt]
        if words:
            self.expect = [split.values(garr, nc, g) for g in range(7)]
        else:
            self.expect = [gs[g + 1] - gs[g] for g in range(6)] + [gs[6]]
        # messages of (CTA, warp, group): rows are one message per warp (weight: how many values)
        self.sends = {}
        for j in range(nc):
            for g in range(7):
                for w in range(self.nwarps[j]):
                    n = sum(i % BLOCK // 32 == w for c in (cnt[j][g:g + 1] if g < 6 else cnt[j][:6]) for i in range(c))
                    if words and w == 0 and cnt[j][g] == 0:
                        n += 1
                    self.sends[j, w, g] = n


class Broken(Exception):
    pass


def run(plan, visits, rng, changes=40):
    """One run under random priorities, changed now and then; raises Broken."""
    order = PASSES * visits
    nc = plan.nc
    phase = [[0, 0] for _ in range(nc)]
    armed = [[False, False] for _ in range(nc)]
    tx = [[0, 0] for _ in range(nc)]
    got = [[0] * len(order) for _ in range(nc)]
    warps = [(j, w) for j in range(nc) for w in range(plan.nwarps[j])]
    at = {k: [0, "send"] for k in warps}  # pass, step
    here = [0] * nc  # warps at the CTA's barrier
    flight = {}      # (from CTA, to CTA) -> [[pass, n], ...]; any of them may arrive next
    prio = {k: rng.random() for k in warps}
    chan = {(a, b): rng.random() for a in range(nc) for b in range(nc)}

    def settle(j, q):
        if armed[j][q] and tx[j][q] == 0:
            armed[j][q] = False
            phase[j][q] += 1

    def step(key):
        j, w = key
        p, what = at[key]
        g, q = order[p], p & 1
        if what == "send":
            if w == 0:
                if armed[j][q] or phase[j][q] != p >> 1:
                    raise Broken("armed in another pass's phase")
                armed[j][q] = True
                tx[j][q] += plan.expect[g]
                settle(j, q)
            n = plan.sends[j, w, g]
            if n:
                for b in range(nc):
                    flight.setdefault((j, b), []).append([p, n])
            at[key][1] = "wait"
            return True
        if what == "wait":
            if (phase[j][q] & 1) == (p >> 1 & 1):  # try_wait.parity: the phase of this parity is not complete
                return False
            if got[j][p] != plan.expect[g]:
                raise Broken("went on without all values")
            at[key][1] = "barrier"
            if not plan.barrier:
                at[key][:] = [p + 1, "send"]
                return True
            here[j] += 1
            if here[j] == plan.nwarps[j]:
                here[j] = 0
                for v in range(plan.nwarps[j]):
                    at[j, v][:] = [p + 1, "send"]
            return True
        return False

    def deliver(ch):
        box = flight[ch]
        p, n = box.pop(rng.randrange(len(box)))
        if not box:
            del flight[ch]
        j, q = ch[1], p & 1
        if phase[j][q] != p >> 1:
            raise Broken("a value counted on another pass's phase")
        got[j][p] += n
        tx[j][q] -= n
        settle(j, q)

    left = set(warps)
    change = set(rng.sample(range(60 * len(warps)), min(changes, 60 * len(warps))))
    i = 0
    while left:
        i += 1
        if i in change:
            prio[rng.choice(warps)] = rng.random()
            chan[rng.choice(list(chan))] = rng.random()
        for _, key in sorted([(prio[k], k) for k in left] + [(chan[c], ("m", c)) for c in flight], key=lambda v: v[0]):
            if key[0] == "m":
                deliver(key[1])
                break
            if step(key):
                left = {k for k in left if at[k][0] < len(order)}
                break
        else:
            raise Broken("stuck")


# equal groups; one row more than the CTAs hold evenly; a channel of a thin sheet (groups too small for every CTA, one
# after the other); empty groups; a CTA without any row; one CTA; groups of more rows than a CTA has threads
SHAPES = [((70, 70, 70, 70, 70, 70), 2), ((97, 95, 96, 98, 64, 33), 3), ((130, 129, 4, 3, 131, 128), 3),
          ((66, 0, 0, 65, 0, 7), 2), ((4, 3, 2, 4, 1, 0), 3), ((5, 1, 0, 3, 2, 2), 1), ((600, 520, 9, 5, 4, 300), 2)]


@pytest.mark.parametrize("sizes,nc", SHAPES, ids=str)
def test_every_order_ends_with_every_value(split, sizes, nc):
    plan = Plan(split, sizes, nc)
    rng = random.Random(7)
    for _ in range(40):
        run(plan, 2, rng)


def test_the_model_finds_missing_synchronisation(split):
    """Without words from CTAs that have no row, and without a barrier over the warps, an order exists that goes wrong."""
    def broken(plan):
        rng = random.Random(11)
        for _ in range(300):
            try:
                run(plan, 2, rng)
            except Broken:
                return True
        return False

    assert broken(Plan(split, (130, 129, 4, 3, 131, 128), 3, words=False))
    assert broken(Plan(split, (70, 70, 70, 70, 70, 70), 2, warps=False))


@pytest.mark.parametrize("nc", range(1, 17))
def test_parts_cover_the_rows_and_values_are_what_is_sent(split, nc):
    rng = random.Random(nc)
    for _ in range(200):
        sizes = [rng.choice((0, 1, 2, 3, nc - 1, nc, nc + 1, rng.randrange(300), rng.randrange(4000))) for _ in range(6)]
        gs = (C.c_int * 7)(*starts(sizes))
        idle = [0] * 7
        rows = [0] * nc
        for g, size in enumerate(sizes):
            at = 0
            for j in range(nc):
                n = split.part_cnt(size, nc, j)
                assert n >= 0 and split.part_lo(size, nc, j) == at
                at += n
                rows[j] += n
                idle[g] += n == 0
            assert at == size
        idle[6] = sum(r == 0 for r in rows)
        for g in range(7):
            assert split.values(gs, nc, g) == (sizes[g] if g < 6 else sum(sizes)) + idle[g]
