"""The barrier protocols of the tensor-core kernels, stepped on the CPU in random orders: copies land in any order, warps advance in
any order, and a wait by parity passes whenever the barrier's present phase has the other parity (the phase wanted, or an older one of
its parity). A kernel's waits are sound if in no order one passes early or is never answered. The kernels' numbers are read
from their sources."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "strix-halo-vulkan_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


class Bar:
    """An mbarrier: `count` arrivals end a phase."""

    def __init__(self, count):
        self.count, self.pending, self.phase = count, count, 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.phase, self.pending = self.phase + 1, self.count

    def passed(self, parity):
        return self.phase % 2 != parity


def explore(make, seeds):
    """Steps the agents make(rng) returns, each a generator that yields the condition it waits for, in random orders."""
    for seed in range(seeds):
        rng = random.Random(seed)
        agents = [[a, next(a)] for a in make(rng)]
        slow = rng.randrange(len(agents) + 1)      # one agent (or none) that seldom gets a turn
        while agents:
            ready = [x for x in agents if x[1]()]
            assert ready or all(getattr(x[0], "gi_code").co_name == "forever" for x in agents), f"order {seed}: every agent waits"
            if not ready:
                break
            pick = rng.choice(ready)
            if len(ready) > 1 and slow < len(agents) and pick is agents[slow] and rng.random() < 0.9:
                continue
            try:
                pick[1] = next(pick[0])
            except StopIteration:
                agents.remove(pick)


def always():
    return True


# ---- wgemm.cu: raw weight stages and operand slots -----------------------------------------------------------------------------------
def wgemm_numbers():
    s = source("wgemm.cu")
    nr256, nr = map(int, re.search(r"wg_nr\(\) \{ return NT == 256 \? (\d+) : (\d+); \}", s).groups())
    groups, na = map(int, re.search(r"WG_GROUPS = (\d+), WG_NA = (\d+)", s).groups())
    waits = re.search(r"bool wg_all_wait\(\) \{ return wg_nr<NT>\(\) != WG_GROUPS; \}", s) is not None
    return {256: nr256, 128: nr}, groups, na, waits


def wgemm_agents(rng, nr, groups, na, all_wait, n=18):
    r_full, r_empty = [Bar(1) for _ in range(nr)], [Bar(groups if all_wait else groups - 1) for _ in range(nr)]
    a_full, a_empty = [Bar(1) for _ in range(na)], [Bar(1) for _ in range(na)]
    stage, flying, slot, done = [None] * nr, [], [None] * na, [0]

    def loader():
        for it in range(n):
            yield lambda: r_empty[it % nr].passed((it // nr & 1) ^ 1)
            stage[it % nr] = None
            flying.append(it)

    def forever():       # the copies, in any order
        while True:
            yield lambda: bool(flying)
            it = flying.pop(rng.randrange(len(flying)))
            stage[it % nr] = it
            r_full[it % nr].arrive()

    def group(g):
        for it in range(n):
            half = (g + (groups - 2) * it) % groups
            s = it % nr
            if half > 1 and not all_wait:
                continue
            yield lambda: r_full[s].passed(it // nr & 1)
            if half > 1:
                r_empty[s].arrive()
                continue
            for _ in range(3):                 # the reads take a while
                assert stage[s] == it, f"group {g} reads super-block {stage[s]} for {it}"
                yield always
            r_empty[s].arrive()
            hx = 2 * it + half
            yield lambda: a_empty[hx % na].passed((hx // na & 1) ^ 1)
            assert done[0] > hx - na, f"operand {hx} overwrites one in use"
            slot[hx % na] = hx
            yield always
            a_full[hx % na].arrive()

    def tensor_core():
        for hx in range(2 * n):
            yield lambda: a_full[hx % na].passed(hx // na & 1)
            assert slot[hx % na] == hx
            yield always
            done[0] = hx + 1
            a_empty[hx % na].arrive()

    return [loader(), forever(), tensor_core()] + [group(g) for g in range(groups)]


@pytest.mark.parametrize("nt", [128, 256])
def test_dequantising_groups_read_the_super_block_they_wait_for(nt):
    nr, groups, na, waits = wgemm_numbers()
    explore(lambda rng: wgemm_agents(rng, nr[nt], groups, na, waits and nr[nt] != groups), 400)


def test_two_stages_want_every_group_at_every_super_block():
    _, groups, na, _ = wgemm_numbers()
    with pytest.raises(AssertionError, match="reads super-block"):
        explore(lambda rng: wgemm_agents(rng, 2, groups, na, False), 400)


# ---- attn_tc.cu: the softmax warps and the products of probabilities and values --------------------------------------------------------
def attn_agents(rng, nt, every_tile):
    s_full, p_full, pv_done = [Bar(1), Bar(1)], [Bar(4), Bar(4)], Bar(1)
    queue, done = [], [0]                      # the tensor core's work in order; products PV in O

    def forever():
        while True:
            yield lambda: bool(queue)
            kind, k = queue.pop(0)
            yield always
            if kind == "scores":
                s_full[k & 1].arrive()
            else:
                done[0] = k + 1
                yield always
                pv_done.arrive()

    def issue():
        queue.append(("scores", 0))
        for k in range(nt):
            if k + 1 < nt:
                queue.append(("scores", k + 1))
            yield lambda: p_full[k & 1].passed(k >> 1 & 1)
            queue.append(("values", k))

    def softmax():
        for k in range(nt):
            yield lambda: s_full[k & 1].passed(k >> 1 & 1)
            if k > 0 and rng.random() < 0.3:   # a maximum grew: O is rescaled
                yield lambda: pv_done.passed((k - 1) & 1)
                assert done[0] == k, f"O rescaled at tile {k} holds {done[0]} products"
            if k > 0 and every_tile:
                yield lambda: pv_done.passed((k - 1) & 1)
                assert done[0] == k
            yield always
            p_full[k & 1].arrive()
        yield lambda: pv_done.passed((nt - 1) & 1)
        assert done[0] == nt, f"O read with {done[0]} of {nt} products"

    return [forever(), issue()] + [softmax() for _ in range(4)]


@pytest.mark.parametrize("nt", [1, 2, 3, 4, 7])
def test_attention_reads_o_after_its_last_product(nt):
    s = source("attn_tc.cu")
    wait = s.find("      if (k > 0 && !(ok = warp_wait(&pv_done, (k - 1) & 1)))")
    explore(lambda rng: attn_agents(rng, nt, 0 <= wait < s.find("if (cb + AT_CELLS > c_hi)")), 400)


def test_attention_warps_want_every_product():
    with pytest.raises(AssertionError, match="O read with"):
        explore(lambda rng: attn_agents(rng, 4, False), 400)
