"""The plan for a step's prompt portions (host code of the kernel library, no GPU): into how many parts the tcgen05 attention
kernel's (tile, head) units are cut, against a plain list scheduling of the same units."""
from __future__ import annotations

import ctypes
import heapq
import random

import pytest

SMS = 148


@pytest.fixture(scope="module")
def ops():
    from inferflux_b200.kernels import ops as o
    return o


def _tiles(entries, shortest, rows, window):
    """Key tiles of 64 that the query tiles go through, in the order of the list."""
    first = lambda p: 0 if window == 0 else max(0, p - window + 1) if window > 0 else p - p % -window
    return [(c + min(n, q0 + rows) - 1) // 64 - first(c + q0) // 64 + 1
            for n, c in entries if n >= shortest for q0 in range(0, n, rows)]


def _plan(ops, entries, heads, rows=256, window=0, shortest=1, max_keys=None):
    longest = max(n + c for n, c in entries)
    return ops.attn_prefill_plan([n for n, _ in entries], [c for _, c in entries], shortest, rows, heads, max_keys or longest,
                                 window, SMS)


@pytest.mark.parametrize("heads", [16, 28, 40])
@pytest.mark.parametrize("tokens", [4096, 8192, 16384])
def test_a_prompt_from_its_start_is_not_cut(ops, tokens, heads):
    """The units behind the last full round are the prompt's first tokens, which see next to nothing."""
    assert _plan(ops, [(tokens, 0)], heads)[0] == 1


@pytest.mark.parametrize("entries,heads,cut", [
    ([(2048, 0)], 28, False), ([(2048, 2048)], 28, False), ([(2048, 8192)], 28, True), ([(2048, 16384)], 28, True),
    ([(2048, 4096)], 40, True), ([(4096, 4096)], 28, True), ([(2048, 8192)], 37, False),        # (37 heads: 296 units, two full rounds)
    ([(16, 0), (2048, 8192)], 28, True), ([(1024, 0), (1500, 8192)], 40, False), ([(1024, 0), (1500, 8192)], 16, False)])
def test_the_cut_goes_by_the_units_that_are_cut(ops, entries, heads, cut):
    """A portion deep in a document is cut where its last round is far from full; a short prompt listed ahead of a long portion
    is not made to look like it."""
    assert (_plan(ops, entries, heads)[0] > 1) == cut


def _by_list_scheduling(tiles, heads):
    """(parts, microseconds): every unit to the SM that is free first, longest list first, as the GPU hands out blocks."""
    units = [k for k in reversed(tiles) for _ in range(heads)]
    whole = len(units) // SMS * SMS
    best = None
    for s in range(1, 7 if whole < len(units) else 2):
        jobs = [4.0 + k for k in units[:whole if s > 1 else len(units)]]
        for k in units[len(jobs):]:
            per = -(-k // s)
            jobs += [4.0 + min(per, k - p * per) if p * per < k else 0.3 for p in range(s)]
        free = [0.0] * SMS
        for j in jobs:
            heapq.heapreplace(free, free[0] + j)
        us = 3.0 + max(free) + (10.0 + 0.05 * (len(units) - whole) * s if s > 1 else 0.0)
        if best is None or us < (0.97 if best[0] == 1 else 1.0) * best[1] - 1e-3:
            best = (s, us)
    return best


@pytest.mark.parametrize("seed", range(40))
def test_plan_against_list_scheduling(ops, seed):
    rng = random.Random(seed)
    heads, window, shortest = rng.choice([1, 7, 16, 28, 40]), rng.choice([0, 0, 300, 4096, -512, -8192]), rng.choice([1, 2, 8])
    entries = [(rng.choice([1, 5, 40, 256, 257, 900, 3000]), rng.choice([0, 63, 1000, 9000])) for _ in range(rng.randint(1, 12))]
    while len(_tiles(entries, shortest, 256, window)) * heads <= SMS:
        entries.append((rng.randint(256, 6000), rng.randint(0, 9000)))
    parts, us, mma_us = _plan(ops, entries, heads, 256, window, shortest)
    want = _by_list_scheduling(_tiles(entries, shortest, 256, window), heads)
    assert us == pytest.approx(want[1], rel=1e-4) and parts == want[0]
    small = _tiles(entries, shortest, 64, window)
    assert mma_us == pytest.approx(5.1 + max(1.51 * max(small), 1.24 * sum(small) * heads / SMS), rel=1e-4)


@pytest.mark.parametrize("entries,heads,rows,parts", [([(64, 8000)], 28, 128, 5), ([(64, 300)], 28, 128, 1), ([(128, 40000)], 2, 128, 16),
                                                      ([(256, 2000)], 100, 256, 1), ([(1, 9000)], 8, 128, 1), ([(2048, 0)], 16, 256, 1)])
def test_fewer_units_than_sms(ops, entries, heads, rows, parts):
    """As many parts as give every block a place at once, each at least 8 key tiles; nothing to plan for single tokens."""
    assert _plan(ops, entries, heads, rows, shortest=2)[0] == parts


@pytest.mark.parametrize("entries,heads,window,tcgen05", [
    ([(2048, 0)], 28, -8192, True), ([(300, 0)], 28, 0, True), ([(64, 6000)], 28, 0, True), ([(512, 6000)], 40, -512, True),
    ([(8, 0)], 28, 0, False), ([(64, 0)], 16, 4096, False), ([(8, 300)] * 16, 28, 0, False), ([(8, 300)] * 4, 40, 256, False),
    ([(16, 1000)] * 16, 28, 256, False), ([(64, 1000)] * 32, 8, -512, False), ([(130, 0)] * 4, 40, 0, False)])
def test_which_kernel_takes_the_portions(ops, entries, heads, window, tcgen05):
    """Where one of the two prompt kernels was measured 10 % and more ahead of the other, the plan's two times say so."""
    blocks = sum((n + 255) // 256 for n, _ in entries) * heads
    longest = max(n + c for n, c in entries)
    _, us, mma_us = _plan(ops, entries, heads, 128 if 2 * blocks <= SMS else 256, window, 8, min(longest, abs(window) + 256) if window else longest)
    assert (us < mma_us) == tcgen05


@pytest.mark.parametrize("m,n,k,address,size", [
    (64, 2048, 2048, 256, 0), (65, 2048, 2048, 256, 6 * 65 * 2048), (301, 22016, 2052, 256, 6 * 301 * 2056),
    (4096, 255, 2048, 256, 0), (4096, 2048, 252, 256, 0), (4096, 2048, 2050, 256, 0), (4096, 2048, 2048, 260, 0),    # to the FFMA kernels
    (16384, 3584, 18944, 256, None), (100000, 256, 256, 256, None), (1 << 20, 151936, 4096, 256, None)])
def test_scratch_of_float32_products(ops, m, n, k, address, size):
    """None where none is used, six bytes a number of the rows, and never more than 64 MB."""
    got = ops.gemm_f32_scratch(address, m, n, k)
    assert got == size if size is not None else 32 << 20 < got <= 64 << 20


def test_a_samplers_list_takes_no_block_off_an_sm(ops):
    """Two blocks an SM (228 KB, of which each takes 1 KB besides its own) wherever two would fit without the list and are wanted; a list as
    long as possible otherwise; never more than 227 KB."""
    out = (ctypes.c_int * 3)()
    fit = lambda size: 228 * 1024 // (size + 1024)
    for vocab in [1, 1000, 8193, 32000, 100000, 152064, *range(160000, 176000, 500), 256000, 406400, 406464, 406912]:
        for rows in (1, 18, 19, 64, 1000):
            ops._lib().ifx_sample_shared(vocab, rows, SMS, out)
            blocks, bare, whole = out
            assert blocks and bare <= whole <= 227 * 1024
            if rows * blocks > SMS:
                assert min(2, fit(whole)) == min(2, fit(bare)), (vocab, rows)
            else:
                assert whole >= min(bare + 4096, 227 * 1024 - 128), (vocab, rows)
    ops._lib().ifx_sample_shared(406913, 1, SMS, out)
    assert out[0] == 0
