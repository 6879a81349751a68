"""Which handoffs of the interaction publish a vertex's word (k_rounds.cu, tl_group and tl_wide), on the CPU.

A vertex u of a block has a word in shared memory and one in global memory. Its pairs, in order, are local ones (L: some
thread of the block applies the pair and moves u's shared word on), pairs across blocks that u's owner applies (D: u is
the lower endpoint) and pairs that another block applies (U: it looks at u's global word, writes it, and u's owner pulls
the result into the shared word). Every interleaving of the threads' loads and stores is followed. Published only before
a U, u always gets through its list; published before every pair across blocks, an older global word can replace a newer
one, and the other block waits for ever (the kernel: until its time limit).
"""

import itertools
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lagrangian-microbes_gb300", "csrc")


def stuck(pairs, publish):
    """Does some interleaving end with u short of its last pair? `publish`: the kinds of next pair that are published."""
    end = len(pairs)
    kind = lambda p: pairs[p] if p < end else "-"
    stores = lambda p: (("S", p),) + ((("G", p),) if kind(p) in publish else ())
    # shared and global position, stores still to come of the owner and of the local appliers (one thread a pair)
    todo, seen = [(0, 0, (), ())], set()
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        S, G, owner, others = state
        after = []

        def store(st, S=S, G=G):
            return (st[1], G) if st[0] == "S" else (S, st[1])

        if owner:
            after.append((*store(owner[0]), owner[1:], others))
        elif kind(S) == "D":
            after.append((S, G, stores(S + 1), others))
        elif kind(S) == "U" and G > S:
            after.append((S, G, (("S", G),), others))
        for k, thread in enumerate(others):
            rest = tuple(t for t in others[:k] + (thread[1:],) + others[k + 1:] if t)
            after.append((*store(thread[0]), owner, rest))
        if kind(S) == "L" and not any(("S", S + 1) in t for t in others):
            after.append((S, G, owner, tuple(sorted(others + (stores(S + 1),)))))
        if kind(G) == "U":  # another block sees itself named (before any store of u's block, the lists' first pair)
            after.append((S, G + 1, owner, others))
        if not after and S != end:
            return True
        todo += after
    return False


@pytest.mark.parametrize("length", [1, 2, 3, 4, 5])
def test_a_vertex_gets_through_every_sequence_of_pairs(length):
    sequences = ["".join(p) for p in itertools.product("LDU", repeat=length)]
    assert not [p for p in sequences if stuck(p, "U")]
    lost = [p for p in sequences if stuck(p, "DU")]
    assert all(re.search("LD.*U", p) for p in lost) and set(lost) >= {p for p in sequences if "LDU" in p}


def test_kernels_publish_what_another_block_applies_and_nothing_else():
    with open(os.path.join(CSRC, "k_rounds.cu")) as f:
        source = f.read()
    source = source[source.index("__device__ void tl_group("):source.index("__device__ bool rounds_tiled(")]
    for word in "us":  # tl_group and tl_wide
        assert len(re.findall(rf"if \(n{word}_id < lo\) st_relaxed\(b\.wstate \+ {word}, nw{word}\);", source)) == 2
    assert len(re.findall(r"\} else \{\s*st_relaxed\(b\.wstate \+ u, nwu\);", source)) == 2  # u belongs to another block
    assert source.count("st_relaxed(") == 6
