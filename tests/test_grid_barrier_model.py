"""The one-launch solver's grid barrier, modelled on the CPU: a block stores its
tag into one of kPSlotSets slots and polls the others' for the same tag; a near
barrier waits only for the blocks whose rows are gathered.  Every interleaving
of three blocks is followed: no block may miss a tag that is overwritten before
it was seen (it would poll to its limit)."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dcu_b200", "csrc", "persist.cu")

# barriers of a solve in order (persist.cu): start, residual, ||b||, two
# iterations, a verified residual that continues, one more iteration, the last residual
START, RESIDUAL, ITERATION = "F", "NF", "NFNFF"
SCHEDULE = START + RESIDUAL + "F" + 2 * ITERATION + RESIDUAL + "F" + ITERATION + RESIDUAL

# blocks whose rows each block gathers (itself always among them)
NEIGHBOURS = {"chain": [{0, 1}, {0, 1, 2}, {1, 2}], "apart": [{0}, {1}, {2}], "one way": [{0}, {0, 1}, {0, 2}]}


def lost_tag(sets, near):
    """A (block, barrier, slot) whose tag can be overwritten before it is seen, or None."""
    nb, last = 3, len(SCHEDULE)

    def needed(b, e):
        return frozenset(range(nb)) if SCHEDULE[e - 1] == "F" else frozenset(near[b])

    # per block: (barrier, slots still to be seen, or None before its own store)
    start = tuple((1, None) for _ in range(nb))
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()

        def tag(o, s):  # the last tag block o stored into slot set s
            e, wait = state[o]
            top = e if wait is not None else e - 1
            while top > 0 and top % sets != s:
                top -= 1
            return top

        for b in range(nb):
            e, wait = state[b]
            if e > last:
                continue
            if wait is None:
                steps = [(e, needed(b, e))]
            else:
                steps = []
                for o in wait:
                    t = tag(o, e % sets)
                    if t > e:
                        return b, e, o
                    if t == e:
                        steps.append((e, wait - {o}))
            for e2, w2 in steps:
                if w2 is not None and not w2:
                    e2, w2 = e2 + 1, None
                nxt = state[:b] + ((e2, w2),) + state[b + 1:]
                if nxt not in seen:
                    seen.add(nxt)
                    todo.append(nxt)
    return None


@pytest.mark.parametrize("near", sorted(NEIGHBOURS))
def test_no_tag_is_overwritten_before_it_is_seen(near):
    sets = re.search(r"constexpr int kPSlotSets = (\d+);", open(SRC).read())
    assert sets, "the number of slot sets is not stated"
    assert lost_tag(int(sets.group(1)), NEIGHBOURS[near]) is None


def test_the_model_finds_a_lost_tag():
    assert lost_tag(2, NEIGHBOURS["chain"]) is not None
    assert lost_tag(3, NEIGHBOURS["chain"]) is None
