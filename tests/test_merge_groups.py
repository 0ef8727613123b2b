"""The two-step merge of a split sequence, restated on the CPU: whatever the order in which the CTAs finish their pieces, every
group is merged once, the sequence is merged once, after all of its groups, and the counters are zero afterwards."""
import random

import pytest

GROUP, GROUP_FROM = 16, 32


def group_of(part, first, last):
    if last - first + 1 <= GROUP_FROM:
        return first, last
    g0 = first + (part - first) // GROUP * GROUP
    return g0, min(g0 + GROUP - 1, last)


@pytest.mark.parametrize("P", [1, 2, 31, 32, 33, 47, 48, 49, 148, 444, 4096])
def test_every_order(P):
    rng, first = random.Random(P), 5
    last = first + P - 1
    for _ in range(5):
        tickets, merged, final = {}, [], 0
        # (a merge is an event of its own: other CTAs may draw between a group's last ticket and the group's own)
        events = [("piece", p) for p in range(first, last + 1)]
        rng.shuffle(events)
        while events:
            kind, x = events.pop(0)
            if kind == "piece":
                a, b = group_of(x, first, last)
                old = tickets.get(b, 0)
                tickets[b] = old + 1
                if (old & 0xffff) == b - a:
                    tickets[b] -= b - a + 1
                    if P > GROUP_FROM:
                        events.insert(rng.randint(0, len(events)), ("group", (a, b)))
                    else:
                        final += 1
            else:
                merged.append(x)
                old = tickets.get(last, 0)
                tickets[last] = old + 0x10000
                n = (last - first) // GROUP + 1
                if old >> 16 == n - 1:
                    tickets[last] -= n << 16
                    final += 1
                    assert len(merged) == n
        assert final == 1
        assert not any(tickets.values())
        if P > GROUP_FROM:
            assert sorted(merged) == [(a, min(a + GROUP - 1, last)) for a in range(first, last + 1, GROUP)]
