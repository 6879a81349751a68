"""Order of the two stores of an interaction handoff (k_rounds.cu, tl_group and tl_wide), on the CPU.

A vertex of a block has a word in shared memory and one in global memory. Thread A applies the pair (s, u) inside the
block and moves u on to a pair with another block; u's owner B may then apply that pair and move u on to the next, which
the other block's thread R applies. Every interleaving of the three threads' loads and stores is followed: if each thread
writes the global word before the shared one, u always gets through its list; the other way round an older global word
can replace a newer one, and R waits for ever (the kernel: until its time limit). The sources are held to that order.
"""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lagrangian-microbes_gb300", "csrc")


def stuck(global_first):
    """Does some interleaving end with u short of its last pair? Positions of u: 0 the pair (s, u), 1 a pair that B
    applies across blocks, 2 one that R applies, 3 the end."""
    order = ("G", "S") if global_first else ("S", "G")
    # A and B: (position they write, stores left); R is one step
    start = (0, 0, (1, order), None)  # shared word, global word, A's stores, B's stores
    seen, todo, lost = set(), [start], False
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        S, G, a, b = state
        after = []
        for who, st in (("a", a), ("b", b)):
            if not st:
                continue
            pos, left = st
            S2, G2 = (pos, G) if left[0] == "S" else (S, pos)
            rest = (pos, left[1:]) if left[1:] else None
            after.append((S2, G2, rest, b) if who == "a" else (S2, G2, a, rest))
        if b is None and S == 1:
            after.append((S, G, a, (2, order)))  # B sees the pair and applies it
        if b is None and S == 2 and G > S:
            after.append((G, G, a, b))           # B pulls R's result
        if G == 2:
            after.append((S, 3, a, b))           # R sees itself named and applies
        if not after and S != 3:
            lost = True
        todo += after
    return lost


def test_a_handoff_gets_through_only_with_the_global_word_first():
    assert stuck(global_first=False)
    assert not stuck(global_first=True)


@pytest.mark.parametrize("word", ["u", "s"])
def test_kernels_publish_before_the_shared_word_shows_the_pair(word):
    with open(os.path.join(CSRC, "k_rounds.cu")) as f:
        lines = f.read().split("\n")
    published = [k for k, line in enumerate(lines) if re.search(rf"publish\(b\.wstate \+ {word}, nw{word}\)", line)]
    assert len(published) == 2  # tl_group and tl_wide
    for k in published:
        assert re.search(rf"st_sh\(.*, nw{word}\);", lines[k + 1])
    # the other stores of a global word are of vertices that the block does not own
    assert len([line for line in lines if re.search(rf"st_relaxed\(b\.wstate \+ {word}, nw{word}\)", line)]) == (2 if word == "u" else 0)
