"""The device ensemble (energy sort, near-duplicate chain) at the edges of its tiles and segments,
against the same sort and chain on the host. Results are indices: they agree exactly."""
import numpy as np
import pytest

from flexaidds_gb300 import evaluator

pytestmark = pytest.mark.gpu

TILE, BLOCKS, SEGMENT, OWN_WALK = 2048, 4 * 152, 8192, 608


def _host(ic, e):
    order = np.argsort(e, kind="stable")     # NaN last, equal energies (and both zeros) in input order
    rows = ic[order].tolist()
    kept, last = [], None
    for p, r in enumerate(rows):
        if last is None or any(not abs(x - y) < 0.1 for x, y in zip(last, r)):
            kept.append(order[p])
            last = r
    return np.array(kept)


def _walk(n, ng, rng):
    """Chromosomes that in energy order take steps of none, less and more than the tolerance."""
    return np.cumsum(rng.choice([0.0, 0.0, 0.03, 0.06, 0.2], size=(n, ng), p=[0.4, 0.2, 0.2, 0.15, 0.05]), axis=0)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, TILE - 1, TILE, TILE + 1, SEGMENT - 1, SEGMENT + 1,
                               3 * SEGMENT + 5])
def test_ensemble_at_tile_and_segment_edges(n):
    rng = np.random.default_rng(n)
    e = rng.normal(-30.0, 8.0, n).round(2)                       # many ties
    special = [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-310, -1e300]
    e[rng.integers(0, n, min(n, 7))] = special[: min(n, 7)]
    ic = np.empty((n, 3))
    ic[np.argsort(e, kind="stable")] = _walk(n, 3, rng)
    r = evaluator.ensemble_dedup(ic, e)
    want = _host(ic, e)
    assert np.array_equal(r["index"], want)
    assert np.array_equal(r["energy"], e[want], equal_nan=True)


def test_ensemble_of_more_tiles_than_blocks():
    n = TILE * BLOCKS + 77
    rng = np.random.default_rng(5)
    e = rng.integers(-(1 << 40), 1 << 40, n).astype(np.float64)
    e[rng.integers(0, n, n // 3)] = 4.0
    ic = np.arange(n, dtype=np.float64)[:, None] % 1000.0
    order = np.argsort(e, kind="stable")
    keep = np.ones(n, bool)
    keep[1:] = ic[order[1:], 0] != ic[order[:-1], 0]             # whole numbers: within 0.1 means equal
    assert np.array_equal(evaluator.ensemble_dedup(ic, e)["index"], order[keep])


def test_one_chain_link_spans_segments():
    n = 3 * SEGMENT
    rng = np.random.default_rng(8)
    e = rng.permutation(n).astype(np.float64)
    ic = np.empty((n, 1))
    walk = 0.09 * (np.arange(n) % 2)                             # every head within 0.1 of the first
    walk[2 * SEGMENT + 3] = 5.0
    ic[np.argsort(e)] = walk[:, None]
    assert np.array_equal(evaluator.ensemble_dedup(ic, e)["index"], _host(ic, e))


@pytest.mark.parametrize("segments", [OWN_WALK - 1, OWN_WALK, OWN_WALK + 1, 2 * OWN_WALK + 1])
def test_chain_of_many_segments(segments):
    """Families within the tolerance of their first member, most of a few heads and some longer than a
    segment, so that the path enters segments at their first head, further in, or not at all."""
    n = segments * SEGMENT - 5
    rng = np.random.default_rng(segments)
    size = rng.integers(1, 40, n // 16)
    size[rng.integers(0, len(size), 40)] = rng.integers(SEGMENT // 2, 3 * SEGMENT, 40)
    first = np.concatenate([[0], np.cumsum(size)])
    first = first[first < n]
    family = np.zeros(n)
    family[first] = 1.0
    # (two values in turn: neighbours differ, so that every chromosome is a head)
    ic = np.cumsum(family) + 0.05 * (np.arange(n) % 2)
    order = rng.permutation(n)                                   # input index of each sorted place
    e, rows = np.empty(n), np.empty((n, 1))
    e[order] = np.arange(n) * 0.001 - 30.0
    rows[order, 0] = ic
    r = evaluator.ensemble_dedup(rows, e)
    assert np.array_equal(r["index"], order[first])
