"""Host-side rules of the attention kernels and the order of their barriers, checked without a GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "keys_values_b200" / "csrc"


def _turns() -> int:
    """Barriers that the two MMA issuers of the dK / dV kernel use in turn (one where the source names no number)."""
    m = re.search(r"constexpr int BO_TURNS = (\d+)", (CSRC / "sdpa_bwd_sm100.cu").read_text())
    return int(m.group(1)) if m else 1


def _reachable_stalls(n: int, turns: int):
    """All interleavings of the producer, the two issuers and the compute warps of ``bwd_dkv_kernel`` over ``n`` query tiles.

    A thread is a list of ("arrive", barrier) and ("wait", barrier, phase); a wait goes by the PARITY of the phase, as the
    hardware's does, so it can be missed when the barrier moves on by two. Copies of Q and dO land at any later moment. Returns the states in which nothing can move although some thread has not ended, and the waits
    that went by on another phase than their own."""
    counts = {f"o_empty{s}": 2 for s in range(2)}
    producer, copies, a, b, compute = [], [], [], [], []
    for i in range(n):
        if i >= 3:
            producer.append(("wait", f"q_empty{i % 3}", i // 3 - 1))
        producer.append(("arrive", f"copy{2 * i}"))
        if i >= 2:
            producer.append(("wait", f"o_empty{i % 2}", i // 2 - 1))
        producer.append(("arrive", f"copy{2 * i + 1}"))
        if i >= 2:
            producer.append(("wait", f"q_empty{(i - 2) % 3}", (i - 2) // 3))
        producer.append(("arrive", f"statistics{i % 2}"))
        copies += [("wait", f"copy{2 * i}", 0), ("arrive", f"q_full{i % 3}"), ("wait", f"copy{2 * i + 1}", 0), ("arrive", f"o_full{i % 2}")]
    a += [("wait", "q_full0", 0), ("arrive", "x0"), ("arrive", "x1")]
    b += [("wait", "o_full0", 0), ("arrive", "y"), ("arrive", "o_empty0")]
    for i in range(n):
        more = i + 1 < n
        a.append(("wait", f"o_full{i % 2}", i // 2))
        b.append(("wait", f"q_full{i % 3}", i // 3))
        if more:
            a.append(("wait", f"q_full{(i + 1) % 3}", (i + 1) // 3))
            b.append(("wait", f"o_full{(i + 1) % 2}", (i + 1) // 2))
        for h in range(2):
            a.append(("wait", f"p{h}", i))
            a += [("arrive", f"o_empty{i % 2}")] * (h == 1) + [("arrive", f"x{h}")] * more
        a.append(("arrive", f"a_issued{i % turns}"))
        b += [("wait", f"a_issued{i % turns}", i // turns), ("wait", "ds", i), ("arrive", f"q_empty{i % 3}")]
        if more:
            b += [("arrive", "y"), ("arrive", f"o_empty{(i + 1) % 2}")]
        compute += [("wait", f"statistics{i % 2}", i // 2), ("wait", "x0", i), ("arrive", "p0"), ("wait", "x1", i), ("arrive", "p1"), ("wait", "y", i), ("arrive", "ds")]
    threads = (producer, copies, a, b, compute)

    def completed(state, bar):
        done = sum(sum(op == ("arrive", bar) for op in t[:at]) for t, at in zip(threads, state))
        return done // counts.get(bar, 1)

    stalls, wrong, seen, todo = [], [], set(), [(0,) * len(threads)]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        moved = False
        for k, t in enumerate(threads):
            if state[k] == len(t):
                continue
            op = t[state[k]]
            if op[0] == "wait":
                phases = completed(state, op[1])
                if (phases & 1) == (op[2] & 1):  # the phase of this parity is the one in progress
                    continue
                if phases != op[2] + 1:
                    wrong.append((state, op))
            moved = True
            todo.append(state[:k] + (state[k] + 1,) + state[k + 1:])
        if not moved and any(at < len(t) for at, t in zip(state, threads)):
            stalls.append(state)
    return stalls, wrong


def test_issuers_of_the_backward_never_miss_a_phase():
    stalls, wrong = _reachable_stalls(6, _turns())
    assert not stalls and not wrong
    assert _reachable_stalls(4, 1)[0]  # one barrier alone can be overrun: issuer A arrives twice before issuer B has looked
