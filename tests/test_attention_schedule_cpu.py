"""Host-side rules of the attention kernels and the order of their barriers, checked without a GPU."""
import re
from pathlib import Path

import pytest

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


def _division(B, units, nT):
    """Units (of ``B * units``) that a forward launch divides over the KV axis and their parts: a last wave at most half full, as many
    of every sequence, parts of equally many KV tiles, four at least, but for a shorter last one."""
    whole = B * units // 148 * 148 // B * B
    divided = B * units - whole
    if B * units % 148 == 0 or nT < 16 or 2 * divided > 148:
        return 0, 1
    tiles = -(-nT // min(148 // divided, nT // 4, 16))
    return divided, -(-nT // tiles)


@pytest.mark.parametrize("B,H,G,T,L,want", [
    (1, 32, 8, 256, 4096, (32, 4)),    # 32 KV tiles: parts of 8
    (2, 40, 8, 499, 7919, (12, 11)),   # 74 units of each sequence in a wave; 62 KV tiles in parts of 6 (12 would leave one empty)
    (1, 4, 1, 33, 2100, (1, 4)),       # 17 KV tiles: parts of 5, the last of 2
    (1, 4, 1, 33, 8192, (1, 16)),      # 64 KV tiles: parts of 4
    (3, 40, 8, 331, 2100, (21, 4)),    # 49 of each sequence in 147 SMs
    (1, 32, 8, 1024, 16384, (0, 1)), (1, 4, 1, 33, 1900, (0, 1))])  # a wave more than half full; a short cache
def test_partial_results_have_room_for_the_parts_that_are_launched(B, H, G, T, L, want):
    """Scratch of a forward call: tile ranges, positions, normalisers, and the rows of every part (a normaliser and the features),
    for pairs of query tiles or, at head size 256, for single ones."""
    from keys_values_b200.ops import cuda

    nT, nQT = -(-L // 128), -(-T // (128 // (H // G)))
    assert _division(B, G * -(-nQT // 2), nT) == want
    parts = [(n * p, rows, D) for (n, p), rows, D in ((want, 256, 128), (_division(B, G * nQT, nT), 128, 256))]
    words = 2 * -(-B * G * nT // 4) * 4 + B * G * (nT + nQT) * 128 + max(n * rows * (1 + D) for n, rows, D in parts)
    assert cuda.lib().kvb_sdpa_fwd_scratch_bytes(B, H, G, T, L) == 4 * words


@pytest.mark.parametrize("B,H,G,T,L", [(1, 32, 8, 2048, 16384), (5, 8, 8, 1000, 16384), (1, 40, 8, 421, 8192), (1, 1, 1, 1, 1), (1, 4, 1, 9, 1 << 23)])
def test_workspace_of_the_backward_stays_below_its_limit(B, H, G, T, L):
    """Beside dS the scratch of a backward call holds a copy of dO, statistics and tile ranges; dS takes one query tile of one (sequence,
    group) at least."""
    import ctypes

    from keys_values_b200.ops import cuda

    npos = 128 // (H // G)
    nT, nQT = -(-L // 128), -(-T // npos)
    other = -(-2 * B * G * nT * 4 // 256) * 256 + B * G * nQT * 1024 + -(-B * H * T * 256 // 256) * 256
    whole = B * G * nT * nQT << 15
    for limit in (0, 1 << 30, 1 << 27, 1 << 24, 1):
        ds = cuda.lib().kvb_sdpa_bwd_scratch_bytes_within(B, H, G, T, L, ctypes.c_longlong(limit)) - other
        assert ds % (nT << 15) == 0 and ds >= nT << 15
        assert ds <= max(limit or 1 << 30, nT << 15)
        assert ds == whole or whole > (limit or 1 << 30)
