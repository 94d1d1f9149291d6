"""Host-only planner: how long axes are split (no GPU needed)."""
import pytest

from shafft_b200 import _sm100

MAX_ROW, MAX_COL = 4096, 2048  # longest row and column pass


def _smooth(limit, primes=(2, 3, 5, 7, 11, 13)):
    out = [1]
    for p in primes:
        nxt = []
        for v in out:
            while v <= limit:
                nxt.append(v)
                v *= p
        out = nxt
    return out


def _factors(n):
    """Some split of n into at most three passes, the last one the longest."""
    small = [a for a in range(1, MAX_COL + 1) if n % a == 0]
    have = set(small)
    for d in range(min(n, MAX_ROW), 0, -1):
        if n % d:
            continue
        c = n // d
        if any(c % a == 0 and c // a in have for a in small):
            return True
    return False


@pytest.mark.parametrize("n,factors", [(13 ** 7, [169, 169, 2197]), (7 ** 10, [343, 343, 2401]),
                                       (5 ** 13, [625, 625, 3125])])
@pytest.mark.parametrize("prec", [0, 1])
def test_longest_factor_may_be_a_row_pass(n, factors, prec):
    """Lengths whose three factors need one above the longest column pass: the
    contiguous axis takes it as its row pass."""
    steps = _sm100.plan_query([n], prec)["steps"]
    assert [s["kind"] for s in steps] == ["pass"] * 3
    assert [s["L"] for s in steps] == factors


@pytest.mark.parametrize("prec", [0, 1])
def test_smooth_lengths_with_factors_are_not_convolved(prec):
    """Every 13-smooth length up to 2^31 that three passes can make is made of passes."""
    for n in _smooth(1 << 31):
        if n <= MAX_ROW:
            continue
        steps = _sm100.plan_query([n], prec)["steps"]
        if all(s["kind"] == "pass" and not s["bs"] for s in steps):
            assert len(steps) <= 3, n
        else:
            assert not _factors(n), n


@pytest.mark.parametrize("dims,factors", [
    ((1 << 16,), [128, 512]), ((64, 1 << 15), [64, 512]), ((16, 1 << 16), [128, 512]), ((512, 1 << 16), [128, 512]),
    ((64, 1 << 17), [256, 512]), ((1 << 17, 64), [256, 512]), ((1 << 17,), [32, 32, 128]), ((1 << 14,), [128, 128])])
def test_complex128_axes_of_many_rows_take_two_passes(dims, factors):
    """Three short factors are for a lone 2^17 signal; many of them take two
    passes, the larger factor last."""
    steps = _sm100.plan_query(list(dims), 1)["steps"]
    lens = [s["L"] for s in steps]
    n = len(factors)
    assert any(lens[i:i + n] == factors for i in range(len(lens) - n + 1)), lens
    assert len(lens) == n + len(dims) - 1


def test_complex128_convolution_of_2p16():
    steps = _sm100.plan_query([22651], 1)["steps"]
    assert [s["L"] for s in steps if s["kind"] == "pass"] == [128, 512] * 2


@pytest.mark.parametrize("dims,L,tiles", [((353, 8), 353, 4), ((17, 277), 277, 9), ((6, 314), 314, 3),
                                          ((288, 269), 269, 144), ((337, 19, 13), 337, 124)])
def test_few_direct_columns_are_spread_over_tiles(dims, L, tiles):
    """complex64 direct-DFT passes of few columns: narrow tiles, so that more SMs share them."""
    steps = [s for s in _sm100.plan_query(list(dims), 0)["steps"] if s["L"] == L]
    assert len(steps) == 1 and steps[0]["tiles"] >= tiles, steps


@pytest.mark.parametrize("n,L,tiles,threads", [(1769625, 1287, 344, 256), (1279395, 1053, 304, 256),
                                               (1203125, 875, 344, 256), (1087515, 845, 322, 192)])
def test_resident_tiles_take_large_blocks(n, L, tiles, threads):
    """Generic complex64 passes whose tiles are all resident at once: many
    threads a tile, and narrow tiles, rather than few tiles of few threads."""
    step = next(s for s in _sm100.plan_query([n], 0)["steps"] if s["L"] == L)
    assert step["tiles"] >= tiles and step["threads"] >= threads, step
