"""The block schedule of the register-resident Jacobi sweep, restated: every
round places each of the 2 K blocks on one CTA, every pair meets once in 2 K - 1
rounds, and a block that stays is never sent."""
import pytest


def tournament(r, q, n):
    a, b = (r % (n - 1), n - 1) if q == 0 else ((r + q) % (n - 1), (r - q + n - 1) % (n - 1))
    return min(a, b), max(a, b)


def rounds(k):
    r = 0
    while k % 2 == 0:
        r, k = r + k, k // 2
    return r + 2 * k - 1


def blocks(ctas, r, c):
    size, upper, k = [], [], ctas
    while k % 2 == 0 and r >= k:
        r -= k
        size.append(k)
        k //= 2
        upper.append(c >= k)
        c -= k if c >= k else 0
    lists, places = [0, 1], [c, (c + r) % k]
    if k % 2 and k > 1:
        x, y = tournament(r, c, 2 * k)
        lists, places = [int(x >= k), int(y >= k)], [x % k, y % k]
    out = []
    for m, i in zip(lists, places):
        for n, up in zip(reversed(size), reversed(upper)):
            half = n // 2
            if up:
                i, m = ((i - 1 + n) % n if m else (i + half - 1) % n), 1
            else:
                i, m = (i + half if m else i), 0
        out.append(m * ctas + i)
    return tuple(out)


@pytest.mark.parametrize("ctas", [1, 2, 3, 4, 6, 7, 9, 17, 32, 40, 72, 144])
def test_every_pair_once_and_one_holder_per_block(ctas):
    seen, held, moved = set(), None, 0
    for r in range(rounds(ctas)):
        now = [blocks(ctas, r, c) for c in range(ctas)]
        assert sorted(x for p in now for x in p) == list(range(2 * ctas))
        for p in now:
            assert frozenset(p) not in seen
            seen.add(frozenset(p))
        if held is not None:
            moved += sum(len(set(a) - set(b)) for a, b in zip(held, now))
        held = now
    assert len(seen) == ctas * (2 * ctas - 1) == ctas * rounds(ctas)
    if ctas % 8 == 0:  # one block of the two, for most of the sweep
        assert moved <= 1.3 * ctas * rounds(ctas)
