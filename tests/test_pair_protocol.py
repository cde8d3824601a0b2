"""The barriers of the CTA-pair kernels (csrc/umma_gemm.cu) as a model on the CPU: two producers, one MMA
issuer, one epilogue per CTA and an engine that lands copies, runs MMAs and delivers commits on its own, under random
schedules.  umma_pair_kernel has three stages and hands an accumulator over per slab, umma_gram_kernel six stages and an
accumulator per tile of several slabs.  When the CTAs leave, no copy, MMA, commit or arrival may be under way, whether every wait was satisfied or
one was given up: it would write into shared memory that belongs to the next CTA.
"""
import os
import random
import re

import pytest

PAIR_STAGES, GRAM_STAGES = 3, 6


class Barrier:
    def __init__(self, need):
        self.need, self.pending, self.bytes, self.phase = need, need, 0, 0

    def _turn(self):
        if self.pending == 0 and self.bytes == 0:
            self.phase, self.pending = self.phase + 1, self.need

    def arrive(self, expect=0):
        assert self.pending > 0
        self.pending, self.bytes = self.pending - 1, self.bytes + expect
        self._turn()

    def land(self):
        self.bytes -= 1
        self._turn()

    def done(self, parity):
        return (self.phase & 1) != parity


def last_uses(count, slots):
    return range(max(0, count - slots), count)


def under_way_at_exit(slabs, seed, tail, fault_at=None, stages=PAIR_STAGES, per_tile=None):
    """per_tile: slabs of a tile where an accumulator is handed over per tile; None: per slab."""
    rnd = random.Random(seed)
    per_acc = per_tile or 1
    accs = slabs // per_acc
    full = [Barrier(1) for _ in range(stages)]
    empty = [[Barrier(1) for _ in range(stages)] for _ in range(2)]
    acc_full = [[Barrier(1) for _ in range(2)] for _ in range(2)]
    acc_empty = [Barrier(2) for _ in range(2)]
    engine, remote, mmas = [], [], []
    end = {"given_up": False, "multiplied": 0, "accs": 0, "copied": [0, 0]}
    fault = [False]

    def wait(bar, parity):
        while not bar.done(parity):
            if fault[0]:
                return False
            yield
        return True

    def drain(bar, parity):
        for _ in range(4000):
            if bar.done(parity):
                return
            yield

    def producer(rank):
        ok, it = True, 0
        while it < slabs:
            s = it % stages
            if it >= stages:
                ok = yield from wait(empty[rank][s], (it // stages - 1) & 1)
                if not ok:
                    break
            if rank == 0:
                full[s].arrive(expect=2)
            engine.append(full[s].land)
            it += 1
            yield
        if tail:
            for j in last_uses(it, stages):
                ok = ok and (yield from wait(empty[rank][j % stages], (j // stages) & 1))
        end["copied"][rank] = it
        end["given_up"] |= not ok

    def issuer():
        ok, it = True, 0
        while it < slabs:
            acc, first, last = it // per_acc, it % per_acc == 0, it % per_acc == per_acc - 1
            if per_tile and first and acc >= 2:
                ok = yield from wait(acc_empty[acc & 1], ((acc >> 1) - 1) & 1)
            ok = ok and (yield from wait(full[it % stages], (it // stages) & 1))
            if not per_tile and ok and acc >= 2:
                ok = yield from wait(acc_empty[acc & 1], ((acc >> 1) - 1) & 1)
            if not ok:
                break
            mmas.append((it, acc if last else None))
            end["accs"] += last
            it += 1
            yield
        end["multiplied"] = it
        end["given_up"] |= not ok

    def epilogue(rank):
        ok = True
        for it in range(accs):
            ok = yield from wait(acc_full[rank][it & 1], (it >> 1) & 1)
            if not ok:
                break
            if rank == 0:
                acc_empty[it & 1].arrive()
            else:
                remote.append(acc_empty[it & 1].arrive)
            yield
        end["given_up"] |= not ok

    def last_words(rank):
        for j in last_uses(end["multiplied"], stages):
            yield from drain(empty[rank][j % stages], (j // stages) & 1)
        for j in last_uses(end["accs"], 2):
            yield from drain(acc_full[rank][j & 1], (j >> 1) & 1)
        if rank == 0:
            for j in last_uses(max(end["copied"]), stages):
                yield from drain(full[j % stages], (j // stages) & 1)

    def play(actors, step=0):
        while actors:
            step += 1
            assert step < 400000, "a wait never ends"
            if step == fault_at:
                fault[0] = True
            k = rnd.random()
            if engine and k < 0.25:
                engine.pop(rnd.randrange(len(engine)))()
            elif mmas and k < 0.45:
                j, acc = mmas.pop(0)
                for rank in range(2):
                    engine.append(empty[rank][j % stages].arrive)
                    if acc is not None:
                        engine.append(acc_full[rank][acc & 1].arrive)
            elif remote and k < 0.6:
                remote.pop(rnd.randrange(len(remote)))()
            else:
                a = rnd.choice(actors)
                if next(a, "end") == "end":
                    actors.remove(a)

    play([producer(0), producer(1), issuer(), epilogue(0), epilogue(1)])
    while remote:               # the cluster barrier orders what threads did before it, not what the engine does
        remote.pop()()
    if tail and end["given_up"]:
        play([last_words(0), last_words(1)])
    return len(engine) + len(mmas)


@pytest.mark.parametrize("slabs", [1, 2, 3, 4, 5, 6, 7, 13])
@pytest.mark.parametrize("gives_up", [False, True])
def test_nothing_is_under_way_when_the_pair_leaves(slabs, gives_up):
    def runs(tail):
        for seed in range(150):
            yield under_way_at_exit(slabs, seed, tail, random.Random(seed).randrange(1, 60 * slabs) if gives_up else None)

    assert not any(runs(True))
    assert any(runs(False))     # without the waits at the end some schedule does leave something


@pytest.mark.parametrize("tiles,per_tile", [(1, 1), (1, 5), (1, 6), (1, 9), (2, 1), (2, 4), (3, 2), (3, 7), (5, 3), (6, 1)])
@pytest.mark.parametrize("gives_up", [False, True])
def test_nothing_is_under_way_when_the_pair_of_the_hessian_leaves(tiles, per_tile, gives_up):
    slabs = tiles * per_tile

    def runs(tail):
        for seed in range(100):
            yield under_way_at_exit(slabs, seed, tail, random.Random(seed).randrange(1, 60 * slabs) if gives_up else None, GRAM_STAGES, per_tile)

    assert not any(runs(True))
    assert any(runs(False))


def test_a_whole_warp_gives_up_a_wait_or_none_of_it():
    """What a warp does together behind a wait (shuffles, tensor memory loads) must be entered by all of its lanes: whole warps wait by
    mbar_wait, which takes a vote.  Lanes decide by themselves only where one lane alone issues copies or MMAs (umma_gemm_kernel) and
    where the answer decides about nothing but the lane's own further wait (a slab of the sweep)."""
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "moe_quant_b200", "csrc")
    text = {name: open(os.path.join(csrc, name)).read() for name in sorted(os.listdir(csrc)) if name.endswith((".cu", ".cuh"))}
    assert "return __all_sync(0xffffffffu, mbar_wait_lane(bar, parity, fault, code));" in text["mbarrier.cuh"]
    alone = {name: len(re.findall(r"(?<!bool )(?<!mq::)\bmbar_wait_lane\(", body)) for name, body in text.items() if name != "mbarrier.cuh"}
    assert {name: n for name, n in alone.items() if n} == {"sweep_super.cu": 1, "umma_gemm.cu": 2}
    assert sum(len(re.findall(r"\bmbar_wait\(", body)) for body in text.values()) > 20
