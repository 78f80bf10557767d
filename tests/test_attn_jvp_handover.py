"""CPU: the hand-over between the two softmax groups and the two issuing warps of the head_dim-64
tangent kernel (``ops/csrc/attn_jvp.cu``), by walking every order in which its events can happen.

The order of a step's events is read from the kernel's source.  Modelled as the hardware has them: an
mbarrier wait sees the parity of the phase only; P V products run in the order of their steps, any
time after P is there (their V tile may be late); the arrival that a commit stands for comes any
time after its products, in order on one barrier and in none between two."""
import itertools
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imfvideo_b200", "ops",
                      "csrc", "attn_jvp.cu")
EVENTS = {"scores": r"mbar_wait\(&s\.s_full\[g\]", "see": r"ref_of_step\(", "publish": r"publish_ref\(|st\.volatile\.shared",
          "wait other": r"mbar_wait\(&s\.o_done\[g \^ 1\]", "rescale": r"tmem_st16\(tb \+ COL_O",
          "wait own": r"mbar_wait\(&s\.o_done\[g\]", "taken": r"mbar_arrive\(&s\.s_taken\[g\]\)",
          "store P": r"tmem_st16\(pc \+ c / 2", "P": r"mbar_arrive\(&s\.p_full\[g\]\)"}


def step_events():
    text = open(SOURCE).read()
    body = text[text.index("for (int j = j_own"):text.index("// ---- epilogue of this segment")]
    at = {}
    for name, pattern in EVENTS.items():
        hits = [m.start() for m in re.finditer(pattern, body)]
        assert len(hits) == 1, (name, len(hits))
        at[name] = hits[0]
    return sorted(at, key=at.get)


def walk(order, steps, outgrown):
    """None, or what goes wrong in some order of events.  ``outgrown``: the steps that move the reference.
    State: events done by either group, P V products run, arrivals on either o_done barrier, the newest
    step whose reference is published."""
    start = ((0, 0), 0, (0, 0), -1)
    seen, todo = {start}, [start]
    own = [list(range(g, steps, 2)) for g in (0, 1)]

    def done(pos, n, name):              # has the group of step n done `name` of it
        i = pos[n & 1] - (n // 2) * len(order)
        return i > order.index(name)

    while todo:
        state = todo.pop()
        pos, run, arrived, ref = state
        nxt = []
        for g in (0, 1):
            k, e = divmod(pos[g], len(order))
            if k == len(own[g]):
                continue
            n, name, par = own[g][k], order[e], k & 1
            passes = lambda bar, parity: (arrived[bar] & 1) != parity
            ref2 = ref
            if name == "scores" and n >= 2 and not done(pos, n - 2, "taken"):
                continue
            if name == "see" and ref < n - 1:
                continue
            if name == "publish":
                ref2 = n
            if name == "wait other" and n in outgrown and not passes(g ^ 1, par ^ 1 if g == 0 else par):
                continue
            if name == "rescale" and n in outgrown and run != n:
                return f"O is moved to the reference of step {n} with {run} P V products run"
            if name == "wait own" and not passes(g, par ^ 1):
                continue
            if name == "store P" and run < n - 1:
                return f"P of step {n} is stored over one that is still to be read ({run} products run)"
            nxt.append((tuple(p + (i == g) for i, p in enumerate(pos)), run, arrived, ref2))
        if run < steps and done(pos, run, "P"):
            nxt.append((pos, run + 1, arrived, ref))
        for b in (0, 1):
            if arrived[b] < (run + 1 - b) // 2:
                nxt.append((pos, run, tuple(a + (i == b) for i, a in enumerate(arrived)), ref))
        if not nxt and any(pos[g] < len(own[g]) * len(order) for g in (0, 1)):
            return f"no event can happen any more: {state}"
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 7])
def test_o_is_only_rescaled_between_its_products(steps):
    order = step_events()
    for some in itertools.product((False, True), repeat=steps - 1):
        outgrown = {n + 1 for n, x in enumerate(some) if x}
        wrong = walk(order, steps, outgrown)
        assert wrong is None, (outgrown, wrong)
