"""The search step's mask arithmetic (search_step.cuh: the left mask one row ahead, the exact
leaf filter, the sentinel that is used up bit by bit) restated in Python: the filter against
brute force at every board size the masks must hold, and the whole step machine against the
oracle."""
import numpy as np
import pytest

M32 = 0xFFFFFFFF


def drop_leaves(a, nc, l, r):
    h = ((nc << 1) & M32) & ~(((l << 1) & M32) | r)
    return a & ((h ^ (-h & M32)) | (0x1FFFFFFF >> (32 - h.bit_length()))) if h else 0


def load(cols, ld, rd, n):
    nc = ((1 << n) - 1) & ~cols
    return nc, (ld << 1) & M32, rd, nc & ~(ld | rd)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 13, 21, 30, 31])
def test_filter_is_exact(n):
    rng = np.random.default_rng(n)
    mask = (1 << n) - 1
    for i in range(4000):
        density = rng.random(3)
        cols, ld, rd = (int(sum(1 << c for c in range(n) if rng.random() < p)) for p in density)
        ld |= int(rng.integers(0, 2)) << min(n, 31)  # a diagonal past the board may still be in the mask
        nc, l, r, a = load(cols, ld, rd, n)
        kept = drop_leaves(a, nc, l, r)
        want = 0
        for c in range(n):
            if a >> c & 1:
                b = 1 << c
                child = mask & ~(cols | b) & ~(((ld | b) << 1) | ((rd | b) >> 1))
                want |= (child != 0) << c
        assert kept == want, (n, cols, ld, rd)


def run_machine(state, extra_steps=0):
    """(count, nodes) of one state; the lane then parks for `extra_steps` more steps."""
    n = int(state["n"])
    nc, l, r, a = load(int(state["cols"]), int(state["ldiag"]), int(state["rdiag"]), n)
    nodes = bin(a).count("1")
    sols = nodes + (nc == 0) if nc & (nc - 1) == 0 else 0
    a = drop_leaves(a, nc, l, r)
    stack, parked = [(0x07FFFFFF, 0x60000000, 0xF0000000, 0)], 0
    while True:
        if a == 0:
            if len(stack) == 1:
                if parked == extra_steps:
                    return sols, nodes
                parked += 1
            a, nc, l, r = stack.pop()
        x = a & (a - 1)
        b = a ^ x
        if x:
            stack.append((x, nc, l, r))
        nc &= ~b
        l2 = (2 * b + l) & M32
        r = ((r + b) & M32) >> 1
        a = nc & ~(l2 | r)
        nodes += bin(a).count("1")
        if nc & (nc - 1) == 0:
            sols += bin(a).count("1")
        l = (l2 << 1) & M32
        a = drop_leaves(a, nc, l, r)


@pytest.mark.parametrize("n,d", [(4, 1), (5, 2), (6, 5), (8, 2), (10, 3), (12, 4)])
def test_step_machine_matches_oracle(nqb, nqo, n, d):
    pool = nqb.generate_pool(n, d)
    want, want_nodes = nqo.solve_states(pool)
    got = [run_machine(s, extra_steps=26) for s in pool]
    assert [g[0] * int(s["weight"]) for g, s in zip(got, pool)] == list(want)
    assert sum(g[1] for g in got) == want_nodes


def test_wide_boards_with_few_rows_left(nqb, nqo):
    boards = nqb.sample_boards(31, 60, 31, 31, 25, 29)
    want, want_nodes = nqo.solve_states(boards)
    got = [run_machine(s) for s in boards]
    assert [g[0] for g in got] == list(want)
    assert sum(g[1] for g in got) == want_nodes
