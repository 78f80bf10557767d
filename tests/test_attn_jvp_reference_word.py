"""CPU: the reference maximum that one softmax group of the head_dim-64 tangent kernel
(``ops/csrc/attn_jvp.cu``) publishes for the other, with the number of its step: whoever sees the number
has the maximum.  The accesses are read from the kernel's source and walked as the PTX memory model has
them: a vector access is one scalar access per element, in no order, and nothing else orders them."""
import itertools
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imfvideo_b200", "ops",
                      "csrc", "attn_jvp.cu")


def accesses(op):
    """The parts of the word that each scalar access of ``op`` (st, ld) covers."""
    kinds = re.findall(op + r"\.volatile\.shared(?:::cta)?\.(v2\.)?[a-z]+(\d+)", open(SOURCE).read())
    assert len(kinds) == 1, kinds
    vector, bits = bool(kinds[0][0]), int(kinds[0][1])
    assert bits * (2 if vector else 1) == 64
    return [("maximum",), ("step",)] if vector else [("maximum", "step")]


def test_number_of_a_step_comes_with_its_maximum():
    stores, loads = accesses("st"), accesses("ld")
    for st, ld in itertools.product(itertools.permutations(stores), itertools.permutations(loads)):
        for when in itertools.product(range(len(st) + 1), repeat=len(ld)):       # stores seen by each load
            if list(when) != sorted(when):
                continue
            got = {}
            for parts, seen in zip(ld, when):
                done = {p for a in st[:seen] for p in a}
                got.update({p: p in done for p in parts})
            assert got["maximum"] or not got["step"], (st, ld, when)
