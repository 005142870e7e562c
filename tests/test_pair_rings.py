"""The rings of the CTA-pair GEMM's converting warps (gemm_tc2.cu) as an event model: barriers that know their phase by its parity only, loads
that land and commits that arrive in any order.  Whatever the order, a team may read no codes but its step's and write no operand stage before the tensor
cores are done with it.  The sizes of the rings are read from the kernel's source."""
import random
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "ratchet_b200" / "csrc" / "gemm_tc2.cu").read_text()
STEPS = 64


def constant(name):
    return int(re.search(rf"\b{name} = (\d+)", SOURCE).group(1))


def per_kind(name, kind):
    """`constexpr int name(int wk) { return wk == A ? x : wk == B ? y : z; }` of one kind."""
    body = re.search(rf"constexpr int {name}\(int wk\) {{ return (.*?); }}", SOURCE).group(1)
    return int(dict(re.findall(r"wk == (\w+) \? (\w+) :", body)).get(kind) or body.rsplit(":", 1)[-1])


class Barrier:
    def __init__(self, count):
        self.count, self.pending, self.phase = count, count, 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.pending, self.phase = self.count, self.phase + 1

    def passed(self, parity):            # mbarrier.test_wait.parity
        return (self.phase - 1) & 1 == parity


class Wrong(Exception):
    pass


def run(seed, teams, slots, stages, scale_slots, free_slots):
    """One CTA over STEPS steps of K, each agent as far as its waits let it, in an order drawn from `seed`; the events of hardware (a load, the arrival
    of a commit) come late by up to many of the agents' turns, whatever was asked for first.  free_slots: the ring that hands the stages on (0: the teams
    wait for the commits themselves).  Returns the steps that were done."""
    rng = random.Random(seed)
    raw_full, raw_empty = [Barrier(1) for _ in range(slots)], [Barrier(1) for _ in range(slots)]
    scale_full, scale_empty = [Barrier(1) for _ in range(scale_slots)], [Barrier(teams) for _ in range(scale_slots)]
    full, empty = [Barrier(2) for _ in range(stages)], [Barrier(1) for _ in range(stages)]        # the activations' load, a team
    free = [Barrier(1) for _ in range(free_slots)]
    held, flying, done = [None] * slots, [], set()

    def later(event):
        flying.append([rng.choice((0, 0, 0, 1, 30, 300)), event])

    def land(step):
        held[step % slots] = step
        raw_full[step % slots].arrive()

    def codes():
        for step in range(STEPS):
            while not raw_empty[step % slots].passed((step // slots + 1) & 1):
                yield
            later(lambda step=step: land(step))

    def scales():
        for group in range(STEPS // teams):
            while not scale_empty[group % scale_slots].passed((group // scale_slots + 1) & 1):
                yield
            scale_full[group % scale_slots].arrive()

    def activations():
        for step in range(STEPS):
            while not empty[step % stages].passed((step // stages + 1) & 1):
                yield
            if free_slots:
                free[step % free_slots].arrive()
            later(full[step % stages].arrive)

    def team(t):
        for step in range(t, STEPS, teams):
            slot, stage, group = step % slots, step % stages, step // teams
            scale = group % scale_slots
            while not scale_full[scale].passed(group // scale_slots & 1):
                yield
            while not raw_full[slot].passed(step // slots & 1):
                yield
            if held[slot] != step:
                raise Wrong(f"team {t} reads step {held[slot]}'s codes for step {step}")
            raw_empty[slot].arrive()
            scale_empty[scale].arrive()
            yield
            while not (free[step % free_slots].passed(step // free_slots & 1) if free_slots else empty[stage].passed((step // stages + 1) & 1)):
                yield
            if step >= stages and step - stages not in done:
                raise Wrong(f"team {t} writes step {step} over step {step - stages}")
            full[stage].arrive()

    def tensor_cores():
        for step in range(STEPS):
            while not full[step % stages].passed(step // stages & 1):
                yield
            for _ in range(rng.choice((0, 0, 1, 40))):
                yield
            done.add(step)
            later(empty[step % stages].arrive)

    agents = [codes(), scales(), activations(), tensor_cores()] + [team(t) for t in range(teams)]
    for _ in range(400 * STEPS):
        if not agents:
            break
        agent = rng.choice(agents)
        if next(agent, agents) is agents:
            agents.remove(agent)
        for event in flying:
            event[0] -= 1
        for event in [e for e in flying if e[0] < 0]:
            flying.remove(event)
            event[1]()
    return len(done)


@pytest.mark.parametrize("kind", ["WK_Q8", "WK_Q4K"])
def test_no_order_of_events_mixes_two_uses_of_a_slot(kind):
    sizes = constant("kTeams"), per_kind("raw_slots", kind), per_kind("stages2", kind), constant("kScaleSlots"), per_kind("free_slots", kind)
    for seed in range(150):
        assert run(seed, *sizes) == STEPS


# what the model sees: six slots of codes over four teams, and five stages whose commits may arrive out of order
@pytest.mark.parametrize("slots,stages", [(6, 4), (4, 5)])
def test_a_slot_that_changes_teams_is_found(slots, stages):
    with pytest.raises(Wrong):
        for seed in range(400):
            run(seed, 4, slots, stages, 2, 0)
