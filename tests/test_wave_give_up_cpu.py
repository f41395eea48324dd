"""What the CTAs of a decode cluster do when waits run out, as a model on the CPU: every order of their steps, with waits that
may run out at any moment.  No CTA may push into one that has left, and none may wait for ever.  How often a CTA that gave up
waits for the others is taken from the kernel's source."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "retrievalattention_b200", "csrc", "ri_wave_fused.cu")


def give_up_barriers() -> int:
    block = re.search(r"if \(s_abort\) \{(.*?)\n  \}", open(SOURCE).read(), re.S).group(1)
    assert block.count("cluster_arrive();") == block.count("cluster_wait();")
    return block.count("cluster_wait();")


def explore(ctas: int, lists: bool, last_owns: bool, barriers: int) -> None:
    """``lists``: the global-list form, with its cluster barrier in front of the attend phase.  ``last_owns``: whether the last CTA
    has outputs to finish; one that has none is sent no partial results and leaves without waiting for any."""
    # the steps of a CTA: c candidates awaited, b barrier, p results pushed, o results awaited, x left; g0, g1 .. giving up
    after_candidates = "b" if lists else "p"

    def successors(state):
        at, phase, arrived, pushed = state
        for i in range(ctas):
            step = at[i]

            def moved(to, phase=phase, arrived=arrived, pushed=pushed):
                return at[:i] + (to,) + at[i + 1:], phase, arrived, pushed

            if step == "c":
                yield moved(after_candidates)
                yield moved("g0")
            elif step == "p":
                assert "x" not in at[:ctas if last_owns else ctas - 1], f"a push into a CTA that has left: {state}"
                yield moved("o" if last_owns or i < ctas - 1 else "x", pushed=pushed | 1 << i)
            elif step == "o":
                yield moved("x" if pushed == (1 << ctas) - 1 else "g0")
                yield moved("g0")
            elif step == "b" or step[0] == "g":
                if not arrived >> i & 1:
                    yield moved(step, arrived=arrived | 1 << i)
        alive = [i for i in range(ctas) if at[i] != "x"]
        if alive and all(arrived >> i & 1 for i in alive):             # the barrier completes: every waiting CTA goes on
            nxt = {"b": "p", **{f"g{n}": f"g{n + 1}" if n + 1 < barriers else "x" for n in range(barriers)}}
            yield tuple("x" if s == "x" else nxt[s] for s in at), phase + 1, 0, pushed

    first = (("c",) * ctas, 0, 0, 0)
    seen, todo = {first}, [first]
    while todo:
        state = todo.pop()
        more = list(successors(state))
        assert more or all(s == "x" for s in state[0]), f"stuck: {state}"
        for s in more:
            if s not in seen:
                seen.add(s)
                todo.append(s)


@pytest.mark.parametrize("ctas", [1, 2, 3, 4])
@pytest.mark.parametrize("lists", [False, True])
@pytest.mark.parametrize("last_owns", [False, True])
def test_no_push_into_a_cta_that_has_left(ctas, lists, last_owns):
    explore(ctas, lists, last_owns, give_up_barriers())


def test_one_barrier_is_not_enough_behind_the_global_lists():
    with pytest.raises(AssertionError, match="has left"):
        explore(3, True, True, 1)
