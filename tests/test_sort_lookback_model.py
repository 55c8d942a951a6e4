"""The onesweep digit passes (radix_onesweep in paratreet_b200/csrc/k_sort.cu)
with look-backs that give up, restated on the host.

A look-back cut short under-counts a digit's prefix: that pass writes inside
[0, n), but two keys can share a slot, and the slots nobody wrote keep what the
alternate buffer held before.  The passes after it then rank keys whose digits
no longer match the histograms, taken once from the original keys, and a digit
with more keys than its histogram says runs past the end.  The model counts such
destinations and restates the bound that keeps the kernel inside its buffers: a
tile's keys of a digit that would run past n go to the front, and the status bit
is set."""
import random
import re
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def sort_model(keys, alt, tile, cut, digits, bits):
    """The digit passes over keys; cut(pass, tile, digit) -> tiles a look-back
    sees before it gives up, or None for all of them.  Returns the last pass's
    keys, the number of destinations >= n and whether a look-back gave up."""
    n, radix = len(keys), 1 << bits
    starts = []
    for p in range(digits):  # the histograms of the original keys
        count = [0] * radix
        for k in keys:
            count[k >> bits * p & radix - 1] += 1
        starts.append([sum(count[:d]) for d in range(radix)])
    src, dst = list(keys), list(alt)
    past, status = 0, False
    for p in range(digits):
        tiles = [src[t:t + tile] for t in range(0, n, tile)]
        counts = []
        for q in tiles:
            count = [0] * radix
            for k in q:
                count[k >> bits * p & radix - 1] += 1
            counts.append(count)
        out = list(dst)
        for t, q in enumerate(tiles):
            at = [0] * radix
            for d in range(radix):
                seen = cut(p, t, d) if t else None
                lo = 0 if seen is None else max(0, t - seen)
                status |= lo > 0
                at[d] = starts[p][d] + sum(counts[u][d] for u in range(lo, t))
                if at[d] + counts[t][d] > n:
                    past += at[d] + counts[t][d] - n
                    status, at[d] = True, 0
            for k in q:
                d = k >> bits * p & radix - 1
                out[at[d]] = k  # IndexError past n
                at[d] += 1
        src, dst = out, src
    return src, past, status


def case(seed, n=600, tile=16, digits=6, bits=3):
    rng = random.Random(seed)
    keys = [rng.getrandbits(digits * bits) for _ in range(n)]
    alt = [rng.getrandbits(digits * bits) for _ in range(n)]  # an earlier sort's keys
    return rng, keys, alt, tile, digits, bits


@pytest.mark.parametrize("seed", range(4))
def test_complete_lookbacks_sort_and_stay_inside(seed):
    _, keys, alt, tile, digits, bits = case(seed)
    out, past, status = sort_model(keys, alt, tile, lambda p, t, d: None, digits, bits)
    assert out == sorted(keys) and past == 0 and not status


def test_later_passes_run_past_the_end_without_the_bound():
    """A few look-backs cut short are enough: whether a destination is past n then
    depends on the bound alone, in a pass behind the one whose look-back gave up."""
    total = 0
    for seed in range(40):
        rng, keys, alt, tile, digits, bits = case(seed)
        cuts = {(rng.randrange(digits - 1), rng.randrange(1, 600 // tile), rng.randrange(1 << bits)) for _ in range(4)}
        out, past, status = sort_model(keys, alt, tile, lambda p, t, d: 0 if (p, t, d) in cuts else None, digits, bits)
        assert status and out != sorted(keys)
        total += past
    assert total > 0


@pytest.mark.parametrize("seed", range(4))
def test_one_pass_cut_short_stays_inside(seed):
    """In the pass whose own look-back gives up, and in it alone, the histogram
    bounds the destinations."""
    rng, keys, alt, tile, _, bits = case(seed, digits=1)
    _, past, status = sort_model(keys, alt, tile, lambda p, t, d: rng.randrange(2), 1, bits)
    assert status and past == 0


def test_kernel_bounds_its_writes():
    """The kernel bounds a digit's first destination and its keys of the tile before
    the only two stores, which count from there."""
    src = open(os.path.join(ROOT, "paratreet_b200", "csrc", "k_sort.cu")).read()
    body = src[src.index("void __launch_bounds__(kSortThreads, 2) radix_onesweep"):src.index("// ---------------------------------------------------------------- small sort")]
    bound = re.search(r"uint32_t first = gofs\[d\] \+ excl;\s*if \(\(int64_t\)first \+ total > n\) \{"
                      r"\s*atomicOr\(status, kErrSort\);\s*first = 0;\s*\}\s*S\.gbase\[d\] = first;", body)
    assert bound, "radix_onesweep takes a digit's destination without the bound"
    assert body.count("S.gbase[") == 2 and "S.gbase[dd] + ((uint32_t)i - S.dstart[dd])" in body
    assert body.count("kout[") == 1 and body.count("vout[") == 1 and body.index("kout[") > bound.end()
