"""The barrier protocol of the attention forward kernel, every interleaving of its three agents walked on the CPU.

MMA issuer, tensor pipe and softmax warps (one agent: each of their barriers collects all 128 threads) run fixed sequences of
waits, issues and arrivals. An mbarrier wait passes while the number of completed phases differs in parity from the phase
waited for, so a phase that is overtaken by the next one is missed and the wait never ends."""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).parents[1] / "param_decomp_b200" / "ops" / "csrc" / "attention_sm100.cu"


def _stuck_states(items: list[int], out_bars: int, rescale: bool) -> set[tuple[int, int, int]]:
    """States (issuer, pipe, softmax position) with no way on before everybody has finished. `items`: 64-key steps of each
    item the CTA walks; `rescale`: whether the softmax warps also wait for P V_{n-1} at every step after an item's first."""
    steps = [(j, n_sub) for n_sub in items for j in range(n_sub)]
    total = len(steps)
    out = lambda n: ("wait", f"o{n % out_bars}", n // out_bars)  # noqa: E731

    issuer: list[tuple] = [("issue", n) for n in range(min(2, total))]
    pipe = [f"s{n % 2}" for n in range(min(2, total))]  # barrier that the n-th tensor step completes
    opened = 0
    for n, (j, _) in enumerate(steps):
        issuer.append(("wait", f"p{n % 2}", n // 2))
        if j == 0:  # O of the item before has been read out (passes at once for the first)
            issuer.append(("wait", "oe", opened - 1))
            opened += 1
        issuer.append(("issue", len(pipe)))
        pipe.append(f"o{n % out_bars}")
        if n + 2 < total:
            issuer += [out(n), ("issue", len(pipe))]
            pipe.append(f"s{n % 2}")
    softmax: list[tuple] = []
    for n, (j, n_sub) in enumerate(steps):
        softmax.append(("wait", f"s{n % 2}", n // 2))
        if rescale and j > 0:
            softmax.append(out(n - 1))
        softmax.append(("arrive", f"p{n % 2}"))
        if j + 1 == n_sub:
            if out_bars == 1:
                softmax.append(out(n - 1))
            softmax += [out(n), ("arrive", "oe")]

    def phases(bar: str, t: int, s: int) -> int:
        return pipe[:t].count(bar) + sum(op == ("arrive", bar) for op in softmax[:s])

    def passes(op: tuple, t: int, s: int) -> bool:
        return op[0] != "wait" or (phases(op[1], t, s) - op[2]) % 2 == 1

    seen, todo, stuck = set(), [(0, 0, 0)], set()
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        i, t, s = state
        issued = sum(op[0] == "issue" for op in issuer[:i])
        nxt = []
        if i < len(issuer) and passes(issuer[i], t, s):
            nxt.append((i + 1, t, s))
        if t < issued:
            nxt.append((i, t + 1, s))
        if s < len(softmax) and passes(softmax[s], t, s):
            nxt.append((i, t, s + 1))
        todo += nxt
        if not nxt and state != (len(issuer), len(pipe), len(softmax)):
            stuck.add(state)
    return stuck


@pytest.mark.parametrize("rescale", [False, True])
@pytest.mark.parametrize("items", [[2], [4], [2, 2, 2], [6, 4, 2]])
def test_no_interleaving_of_the_forward_gets_stuck(items, rescale):
    found = re.search(r"constexpr int kOutBars = (\d+);", SOURCE.read_text())
    assert not _stuck_states(items, int(found.group(1)) if found else 1, rescale)


def test_one_output_barrier_misses_a_phase():
    """What the second barrier is for: with one, P V of an item's last step can end before the warps poll for the one before."""
    assert _stuck_states([2], 1, False) and _stuck_states([4, 2], 1, True)
