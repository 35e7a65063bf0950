"""The barrier protocol of the batched-decode kernel (csrc/w4a16_narrow.cu) as a discrete-event model.

An mbarrier wait names a phase by its parity alone, so it is only right where the phase before the one waited for is known
to be complete: otherwise "the phase with the other parity" is still the one before, and the wait passes a whole round of
the ring early.  The model runs the kernel's roles against barriers with exactly that rule and copies that land in any
order, and records every wait that passes before its round is complete.  Ring depths are those the launch code computes.
"""
import os
import random

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = open(os.path.join(ROOT, "sparse-quant_b200", "csrc", "w4a16_narrow.cu")).read()
SETS = 4                                                          # dequantiser sets that take stages in turn


def rings(T, G, blocks):
    """(Q, R, DR) of NarrowCfg<T, G>: shared-memory ring for this many out-feature blocks, A ring, group-sum ring."""
    r = 4 if T == 64 else 6
    dr = 2 if G == 64 and T >= 32 else 4
    x_stage, w_stage = 2 * T * 128, 16 * 512 + (128 // G) * 512
    q = (227 * 1024 - 1024 - 1024 - blocks * T * 128 * 4) // (x_stage + w_stage)
    return min(q, 16), r, dr


def test_the_model_uses_the_kernels_constants():
    assert "kRing = T == 64 ? 4 : 6;" in SOURCE
    assert "kDRing = T == 32 && G == 64 ? 2 : (T == 64 && G == 64 ? 2 : 4);" in SOURCE
    assert "kMaxStages = 16;" in SOURCE and "kNarrowSmem = 227 * 1024;" in SOURCE
    assert "(kNarrowSmem - 1024 - kBarBytes - blocks * kRedBytes) / (kXStage + kWStage)" in SOURCE


class Bar:
    def __init__(self, count):
        self.count, self.pending, self.tx, self.phase = count, count, 0, 0      # phase = completed rounds
        self.overrun = False

    def _turn(self):
        if self.pending == 0 and self.tx == 0:
            self.phase += 1
            self.pending = self.count

    def arrive(self, tx=0):
        if self.pending == 0:
            self.overrun = True                                   # more arrivals than the round expects: undefined
            return
        self.tx += tx
        self.pending -= 1
        self._turn()

    def complete(self, tx):
        self.tx -= tx
        self._turn()

    def passes(self, parity):
        return (self.phase & 1) != parity


def simulate(Q, R, DR, total, seed, guarded, previous_ends=0, held=lambda role: True):
    """-> list of (role, stage) whose wait passed a round early, plus ('overrun', name) for barriers hit too often and
    ('counts the previous grid', role, stage) for waits that were already running when the previous grid of a programmatic
    launch ended; `held` says which roles wait for that grid before they wait for anything the activations set off."""
    rng = random.Random(seed)
    ready, done = [Bar(3) for _ in range(Q)], [Bar(1) for _ in range(Q)]
    wfull, wempty = [Bar(2) for _ in range(Q)], [Bar(1) for _ in range(Q)]
    early, landing, now = [], [], [0]

    def wait(role, bars, it):                                     # wait for the round of stage `it` (it < 0: passes at once)
        since = now[0]
        while not bars[it % Q].passes((it // Q) & 1):
            yield 1
        if since < previous_ends <= now[0] and bars is not wfull:
            early.append(("counts the previous grid", role, it))
        if bars[it % Q].phase < it // Q + 1:
            early.append((role, it))

    def latency():
        return rng.choice((20, 25, 30)) if rng.random() < 0.85 else rng.randrange(100, 600)

    def after_previous(role):
        while held(role) and now[0] < previous_ends:
            yield 1

    def weights(role):
        for it in range(total):
            if it == Q:
                yield from after_previous("weights")
            if it >= Q:
                yield from wait(role, wempty, it - Q)
            wfull[it % Q].arrive(1)
            landing.append([latency(), wfull[it % Q]])
            yield 2

    def activations():
        while now[0] < previous_ends:
            yield 1
        for it in range(total):
            if it >= Q:
                yield from wait("x", done, it - Q)
            ready[it % Q].arrive(1)
            landing.append([latency(), ready[it % Q]])
            yield 2

    def mma():
        yield from after_previous("MMA")
        for it in range(total):
            yield from wait("mma", ready, it)
            yield 4
            done[it % Q].arrive()

    def dequantiser(s):
        for it in range(s, total, SETS):
            if R <= it < R + SETS and guarded(Q, R) and it >= Q:
                yield from after_previous("dequantisers")
            if guarded(Q, R) and it >= Q:
                yield from wait("dequantiser, stage before", done, it - Q)
            yield from wait("dequantiser", wfull, it)
            yield 2
            wempty[it % Q].arrive()
            if R <= it < R + SETS:
                yield from after_previous("dequantisers")
            if it >= R:
                yield from wait("dequantiser, A slot", done, it - R)
            yield 6
            ready[it % Q].arrive()

    def epilogue():
        for it in range(min(DR, total)):
            ready[it % Q].arrive()
        yield from after_previous("scale and accumulate")
        for it in range(total):
            yield from wait("epilogue", done, it)
            yield 3
            if it + DR < total:
                ready[(it + DR) % Q].arrive()

    procs = [[0, p] for p in (weights("w"), weights("zs"), activations(), mma(), epilogue())] + [[0, dequantiser(s)] for s in range(SETS)]
    for now[0] in range(400 * total + previous_ends):
        for c in landing:
            c[0] -= 1
            if c[0] == 0:
                c[1].complete(1)
        landing[:] = [c for c in landing if c[0] > 0]
        live = False
        for p in procs:
            if p[1] is None:
                continue
            live = True
            p[0] -= 1
            if p[0] <= 0:
                try:
                    p[0] = next(p[1])
                except StopIteration:
                    p[1] = None
        if not live or early:
            break
    else:
        early.append(("never ends", total))
    early += [("overrun", n) for n, bars in (("ready", ready), ("done", done), ("wfull", wfull), ("wempty", wempty)) if any(b.overrun for b in bars)]
    return early


SHAPES = [(T, G, b) for T in (16, 32, 64) for G in (64, 128) for b in range(1, 25) if rings(T, G, b)[0] >= rings(T, G, b)[1]]


def kernel_guards(Q, R):
    """What the kernel does: with rings so shallow that a set's own history does not vouch for the stage's last round, its
    dequantisers wait for that round's MMAs before they look at the weights' barrier."""
    role = SOURCE.split("---- dequantisers")[1].split("---- scale and accumulate")[0]
    there = "GUARD && it >= Q" in role and "done_bar(st), phase ^ 1u" in role and \
        "guard(int stages) { return stages < kRing + kDequantSets; }" in SOURCE and "guard = T == 64 || Cfg::guard(pl.stages)" in SOURCE
    return there and Q < R + SETS


@pytest.mark.parametrize("T,G", sorted({s[:2] for s in SHAPES}))
def test_no_wait_passes_a_round_early(T, G):
    depths = sorted({rings(t, g, b) for t, g, b in SHAPES if (t, g) == (T, G)})
    for q, r, dr in depths:
        for seed in range(3):
            assert simulate(q, r, dr, 4 * q + 3, seed, kernel_guards) == [], (q, r, dr, seed)


def test_the_model_sees_the_early_pass_of_a_shallow_ring_without_the_wait():
    def found(q, r, dr):
        return any(simulate(q, r, dr, 5 * q + 3, seed, lambda *_: False) for seed in range(12))
    assert found(5, 4, 4) and found(6, 4, 2) and found(7, 4, 4)   # every depth the 64-token tile has
    assert not found(8, 4, 4) and not found(10, 6, 4)             # from R + 4 on a set's own history vouches for it


def _role(name):
    """The kernel's source from the role's headline to the next one."""
    return SOURCE.split("// ---- " + name)[1].split("// ---- ")[0]


def test_waits_behind_the_previous_grid_do_not_count_its_time():
    """Programmatic launch: the activations arrive when the previous grid has ended, however late.  Nobody may be inside a
    bounded wait for something they set off by then (the weights' own barriers are filled before)."""
    def kernel(role):
        names = {"weights": ("packed weights", "(zero, scale) rows"), "MMA": ("MMA",), "dequantisers": ("dequantisers",),
                 "scale and accumulate": ("scale and accumulate",)}[role]
        return all("after_previous()" in _role(n) for n in names)

    for q, r, dr in sorted({rings(T, G, b) for T, G, b in SHAPES if T < 64}):
        assert simulate(q, r, dr, 4 * q, 1, kernel_guards, previous_ends=600, held=kernel) == [], (q, r, dr)
    assert any("counts the previous grid" in e for e in simulate(10, 6, 4, 40, 1, kernel_guards, previous_ends=600, held=lambda role: False))


def test_a_lane_that_gives_up_does_not_leave_its_warp():
    """A bounded wait may end differently for two lanes (timer, abort flag), and behind it stand warp-wide instructions: the
    producers vote before they leave; in the other roles no wait ends a loop, and none gives up before the producers have."""
    kernel = SOURCE.split("narrow_kernel(const")[1].split("int g_force_blocks")[0]
    assert kernel.count("mbar_wait(") == 1 and "__all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, kWaitBudgetNs))" in kernel
    waits_on = kernel.split("auto wait_on")[1].split("};")[0]
    assert "> 2 * kWaitBudgetNs) { *abort_flag = kRunOut; return; }" in waits_on and "*abort_flag)" not in waits_on
    for name in ("packed weights", "activations", "(zero, scale) rows"):
        assert "wait_all(" in _role(name) and "wait_on(" not in _role(name)
    for name in ("MMA", "dequantisers", "scale and accumulate"):
        role = _role(name)
        assert "wait_on(" in role and "wait_all(" not in role
        assert role.replace("if (it >= total) break;", "").count("break") == 0
