"""CPU: the host-side plan of the weight-gradient kernel (how blocks of weight rows and token tiles are dealt to CTAs)."""
import ctypes as C
import heapq
import math
import random
import subprocess
import sys
import time

import pytest

from tests.conftest import ROOT

# dims (B, H, S, d_h, Hkuv, E, d_e) whose plans differ although they have the same number of weight blocks and token tiles
PAIRS = [((5, 4, 100, 64, 4, 9, 64), (5, 4, 100, 64, 4, 10, 64)), ((2, 8, 1500, 96, 8, 1, 64), (2, 8, 1500, 96, 8, 2, 64)),
         ((2, 8, 333, 96, 8, 9, 64), (2, 8, 333, 96, 8, 10, 64))]


def _bytes_in_fresh_process(shapes):
    src = ("import ctypes as C, sys\nfrom flashmhf_b200 import _lib\nlib = _lib.load()\n"
           f"for s in {shapes!r}: print(lib.flashmhf_backward_workspace_bytes(C.byref(_lib.Dims(*s, 0))))")
    r = subprocess.run([sys.executable, "-c", src], cwd=ROOT, capture_output=True, text=True, check=True)
    return [int(v) for v in r.stdout.split()]


@pytest.mark.parametrize("a,b", PAIRS)
def test_plan_does_not_depend_on_the_calls_before(a, b):
    ab, ba = _bytes_in_fresh_process([a, b]), _bytes_in_fresh_process([b, a])
    assert ab == ba[::-1]


# ------------------------------------------------------------------------------------------------ against a job-by-job simulation
SMS = 148                                                                 # what the library plans for where there is no GPU
SHAPE = {64: (128, 64, 0.8), 96: (128, 64, 1.0), 128: (64, 128, 1.8)}     # weight rows, tokens and us of a tile


def _plan(lib, dims, parts):
    from flashmhf_b200 import _lib
    out = _lib.BackwardPlan()
    assert lib.flashmhf_backward_plan(C.byref(_lib.Dims(*dims, 0)), parts, C.byref(out)) == 0
    return out


def _list_schedule(jobs):
    sms, end = [0.0] * SMS, 0.0
    for j in jobs:
        t = heapq.heappop(sms) + j
        heapq.heappush(sms, t)
        end = max(end, t)
    return end


class _Search:
    """Every plan of every family by a list schedule of its CTAs one by one; the shortest."""

    def __init__(self, dims, followed):
        B, H, S, dh, Hk, E, de = dims
        rows, tokens, us = SHAPE[dh]
        self.items, self.T = Hk * -(-E * de // rows), -(-S // tokens) * (H // Hk) * B
        self.fixed, self.launch, self.sums = 7 / us, 4 / us, Hk * E * de * 3 * dh * 4 / 4e6 / us
        self.followed = followed

    def _parts(self, n):
        per = -(-self.T // n)
        return per if -(-self.T // per) == n else None

    def cost(self, p):
        """Of a plan the library returned."""
        T, f, n = self.T, self.fixed, self.items
        if p.splits == 1:
            return -(-n // SMS) * (T + f) * (0.9 if self.followed else 1.0)
        rest, per, k = n - p.whole_blocks, p.tiles_per_split, p.splits
        add = self.launch + k * self.sums * rest / n
        if p.uneven_blocks:
            m = p.uneven_blocks
            return add + _list_schedule([T - p.small_tiles + f] * m + [per + f] * (n - m) + [T - per + f] * (n - m) + [p.small_tiles + f] * m)
        if p.whole_blocks or k == 2:
            return add + _list_schedule([T + f] * p.whole_blocks + [per + f] * ((k - 1) * rest) + [T - (k - 1) * per + f] * rest)
        return add + -(-n * k // SMS) * (per + f)

    def best(self):
        T, f, n = self.T, self.fixed, self.items
        found = [-(-n // SMS) * (T + f) * (0.9 if self.followed else 1.0)]
        for k in range(2, min(16, T) + 1):
            per = self._parts(k)
            if per is None:
                continue
            if k != 2:
                found.append(self.launch + k * self.sums + -(-n * k // SMS) * (per + f))
            else:
                base = _list_schedule([per + f] * n + [T - per + f] * n)
                least = base
                if T >= 32:
                    for small in range(max(1, T // 32), per, max(1, T // 32)):
                        for m in range(SMS // 4, n + 1, SMS // 4):
                            least = min(least, _list_schedule([T - small + f] * m + [per + f] * (n - m) + [T - per + f] * (n - m) +
                                                              [small + f] * m))
                found.append(self.launch + 2 * self.sums + (least if least <= 0.985 * base else base))
            if T >= 8 and k <= 6:
                for q in range(2, 4 * n // SMS + 2):
                    nd = q * SMS // 4
                    if nd < n:
                        found.append(_list_schedule([T + f] * nd + [per + f] * ((k - 1) * (n - nd)) + [T - (k - 1) * per + f] * (n - nd)) +
                                     self.launch + k * self.sums * (n - nd) / n)
        return min(found)


def _draw(rng, most_items=None, most_tokens=8192):
    while True:
        dh, H = rng.choice((64, 96, 128)), rng.choice((4, 8, 16))
        d = (rng.randint(1, 16), H, round(math.exp(rng.uniform(math.log(1), math.log(most_tokens)))), dh, rng.choice((H, H // 2)), rng.randint(1, 32),
             64 * rng.randint(1, 6))
        if most_items is None or d[4] * d[5] * d[6] // 64 <= most_items:
            return d


def test_plans_are_the_shortest_of_a_job_by_job_simulation(lib):
    rng = random.Random(5)
    seen = set()
    for i in range(60):
        d, followed = _draw(rng, 400, 1500), i % 2 == 0
        p, s = _plan(lib, d, 0 if followed else 2), _Search(d, followed)
        assert p.token_tiles == s.T
        assert p.predicted_tiles == pytest.approx(s.cost(p), rel=1e-9), d
        assert p.predicted_tiles == pytest.approx(s.best(), rel=1e-9), d
        seen.add("whole" if p.splits == 1 else "rest" if p.whole_blocks else "uneven" if p.uneven_blocks else "equal")
    assert seen >= {"whole", "rest", "equal"}


def test_planning_costs_microseconds_for_any_number_of_shapes(lib):
    """A plan of a new shape takes a few microseconds (simulated CTA by CTA: milliseconds, and up to a tenth of a second), and the
    thousandth shape no more than the first, again and again."""
    rng = random.Random(6)
    shapes = [_draw(rng) for _ in range(1000)]
    best = []
    for _ in range(3):
        t = time.perf_counter()
        for d in shapes:
            _plan(lib, d, 0)
            _plan(lib, d, 2)
        best.append((time.perf_counter() - t) / 2000)
    assert min(best) < 50e-6, best
