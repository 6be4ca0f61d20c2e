"""The batched form by arcs (limits from 12,000 on) against the plain form,
which evaluates every Gaussian product: the smallest arc limit, the one below
it, the last row, low rows (shared primes and powers with most roots), heavy
rows of each parity, a limit with ragged last blocks, a call long enough to be
planned in two pieces, both CTA sizes and a captured graph.  And the no-alloc
form by arcs against the batched one, on two calls in a row."""
import pytest

import hss

FIELDS = ("pairs", "processed", "products", "candidates", "r16", "merged", "merged_products", "merged_candidates", "merged_r16")


@pytest.mark.gpu
@pytest.mark.parametrize("limit,first,last,opts", [
    (11_999, 11_400, 11_999, {}),
    (12_000, 1, 70, {}),
    (12_000, 11_400, 12_000, {}),
    (12_000, 5_000, 7_100, {}),
    (12_001, 5_515, 5_535, {"block_threads": 512}),
    (100_003, 32_032, 32_052, {}),
    (100_003, 64_080, 64_110, {"use_graph": 1}),
    (300_017, 160_215, 160_235, {}),
    (1_000_000, 801_120, 801_125, {}),
])
def test_batched_equals_plain(limit, first, last, opts):
    with hss.Search(limit, **opts) as s:
        plain = s.search(first, last, mode="plain", rows=True)
        batched = s.search(first, last, rows=True)
        again = s.search(first, last, rows=True)
    for got in (batched, again):
        assert {k: got.counts[k] for k in FIELDS} == {k: plain.counts[k] for k in FIELDS}
        assert got.row_candidates == plain.row_candidates
        assert got.hits == plain.hits


@pytest.mark.gpu
@pytest.mark.parametrize("limit,first,last", [
    (11_999, 11_990, 11_999),
    (12_000, 1, 64),
    (12_000, 11_937, 12_000),
    (300_017, 160_222, 160_228),
    (5_000_000, 1_185_665, 1_185_665),
])
def test_noalloc_equals_batched(limit, first, last):
    with hss.Search(limit) as s:
        want = s.search(first, last)
        for _ in range(2):
            got = s.search_noalloc(first, last)
            assert {k: got.counts[k] for k in FIELDS} == {k: want.counts[k] for k in FIELDS}
            assert got.hits == want.hits
