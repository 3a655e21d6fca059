"""The order that the float product's kernel keeps by barriers, in a model on the host: who waits for which phase, under random delays.

An mbarrier's wait by parity returns when the phase it names is over, and as well when the phase before that one has not even ended.  The
kernel's maps from a block to its stage, barriers, issuer and group of splitting warps come from the library; the model runs the kernel's
roles over them with barriers that behave as mbarriers do."""
from __future__ import annotations

import ctypes
import heapq
import random

import pytest


class _Barrier:
    def __init__(self, count):
        self.count = self.left = count
        self.phase = self.arrivals = 0      # phases that have ended

    def arrive(self):
        self.arrivals += 1
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1


def _kernel_order(b, groups):
    from janis_b200.csrc.build import core_library
    out = (ctypes.c_int * 8)()
    form = core_library().janis_gemm_f32_order
    form.argtypes, form.restype = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p], None
    form(b, groups, out)
    return tuple(out)


def _stage_order(b, groups):
    """A stage's own barriers: 3 stages, chunks of 2 blocks."""
    return b % 3, b % 3, (b // 3) & 1, (b // 2) & 1, b % groups, 3, 3, 2


def _early_returns(order, groups, n_blocks, seed):
    """Runs the kernel's roles once; the waits that returned before their phase had ended, and stages read with other than their block."""
    rng = random.Random(seed)
    _, _, _, _, _, stages, pairs, chunk = order(0, groups)
    blocks = [order(b, groups) for b in range(n_blocks)]
    n_chunks = -(-n_blocks // chunk)
    full, empty = [_Barrier(2) for _ in range(pairs)], [_Barrier(1) for _ in range(pairs)]
    there, taken = [_Barrier(1) for _ in range(2)], [_Barrier(1) for _ in range(2)]
    holds = [[None, None] for _ in range(stages)]           # the blocks whose W and x a stage holds
    faults, pipe = [], []                                    # pipe: the products and commits issued, in order
    scale = [10.0 ** rng.uniform(-1, 1) for _ in range(6)]   # how slow each role is in this run

    def slow(role):
        return rng.expovariate(1.0) * scale[role] * (8.0 if rng.random() < 0.1 else 1.0)

    def wait(barrier, parity, ended, what):
        while (barrier.phase & 1) == parity:
            yield None                                      # asked again when something has happened
        if barrier.phase < ended:
            faults.append(what)

    def copy(b):                                            # a copy of x lands by itself, in no order
        yield slow(0)
        holds[blocks[b][0]][1] = b
        full[blocks[b][1]].arrive()

    def loader():
        for b in range(n_blocks):
            if b >= stages:
                yield from wait(empty[blocks[b - stages][1]], blocks[b - stages][2], (b - stages) // pairs + 1, ("x", b))
            yield slow(1)
            start(copy(b))

    def splitter(group):
        for b in range(n_blocks):
            if blocks[b][4] != group:
                continue
            if b >= stages:
                yield from wait(empty[blocks[b - stages][1]], blocks[b - stages][2], (b - stages) // pairs + 1, ("W", b))
            holds[blocks[b][0]][0] = None
            yield slow(2)
            holds[blocks[b][0]][0] = b
            full[blocks[b][1]].arrive()

    def issuer(who):
        for c in range(n_chunks):
            if blocks[c * chunk][3] != who:
                continue
            if c >= 2:
                yield from wait(taken[who], (c // 2 - 1) & 1, c // 2, ("taken", c))
            for b in range(c * chunk, min((c + 1) * chunk, n_blocks)):
                yield from wait(full[blocks[b][1]], blocks[b][2], b // pairs + 1, ("product", b))
                yield slow(3)
                pipe.append(("block", b))
            pipe.append(("chunk", who))

    def tensor_cores():
        while True:
            while not pipe:
                yield None
            kind, x = pipe[0]
            if kind == "block":
                if holds[blocks[x][0]] != [x, x]:
                    faults.append(("read", x, tuple(holds[blocks[x][0]])))
                yield slow(4)
                empty[blocks[x][1]].arrive()
            else:
                there[x].arrive()
            pipe.pop(0)

    def adder():
        for c in range(n_chunks):
            yield from wait(there[c & 1], (c // 2) & 1, c // 2 + 1, ("sums", c))
            yield slow(5)
            taken[c & 1].arrive()
        done.append(True)

    done, ready, parked, clock = [], [], [], [0.0, 0]

    def moved():
        return sum(b.arrivals for b in full + empty + there + taken), len(pipe)

    def start(role):
        clock[1] += 1
        heapq.heappush(ready, (clock[0], clock[1], role))

    for role in [loader(), issuer(0), issuer(1), tensor_cores(), adder()] + [splitter(g) for g in range(groups)]:
        start(role)
    while not done and not faults:
        if not ready:
            return [("stuck",)]                              # all of them wait
        clock[0], _, role = heapq.heappop(ready)
        before = moved()
        try:
            t = next(role)
        except StopIteration:
            t = -1.0
        if before != moved():                                # something for the others
            for r in parked:
                start(r)
            parked.clear()
        if t is None:
            parked.append(role)
        elif t >= 0.0:
            clock[1] += 1
            heapq.heappush(ready, (clock[0] + t, clock[1], role))
    return faults


@pytest.mark.parametrize("groups", [1, 2])
def test_no_wait_of_the_float_product_returns_a_phase_early(groups):
    for seed in range(1500):
        n = 3 + seed % 41
        assert _early_returns(_kernel_order, groups, n, seed) == [], (seed, n)


@pytest.mark.parametrize("groups", [1, 2])
def test_the_model_sees_waits_on_a_stages_own_barriers(groups):
    """With one pair of barriers a stage, a copy that overtakes another lets an issuer's wait (and one group of two, a splitter's) through."""
    faults = [f for seed in range(1500) for f in _early_returns(_stage_order, groups, 3 + seed % 41, seed)[:1]]
    assert any(f[0] == "product" for f in faults)
    assert any(f[0] == "W" for f in faults) == (groups == 2)
