"""The batched form by arcs against the plain form, which evaluates every
Gaussian product: the smallest limit with the arc layout and the one below it,
calls of 64 and 65 rows below the limit from which long calls go by arcs, that
limit and the one below it, the last row, low rows (shared primes and powers with most roots), heavy
rows of each parity, a limit with ragged last blocks, a call long enough to be
planned in two pieces, both CTA sizes and a captured graph.  And the no-alloc
form by arcs against the batched one, on two calls in a row."""
import pytest

import hss

FIELDS = ("pairs", "processed", "products", "candidates", "r16", "merged", "merged_products", "merged_candidates", "merged_r16")


@pytest.mark.gpu
@pytest.mark.parametrize("limit,first,last,opts", [
    (999, 1, 64, {}),
    (1_000, 1, 64, {}),
    (5_000, 4_937, 5_000, {}),
    (5_000, 1, 65, {}),
    (9_999, 1_100, 1_163, {}),
    (9_999, 9_399, 9_999, {}),
    (10_000, 9_400, 10_000, {}),
    (12_000, 1, 70, {}),
    (12_000, 11_400, 12_000, {}),
    (12_000, 5_000, 7_100, {}),
    (12_001, 5_515, 5_535, {"block_threads": 512}),
    (100_003, 32_032, 32_052, {}),
    (100_003, 64_080, 64_110, {"use_graph": 1}),
    (300_017, 160_215, 160_235, {}),
    (1_000_000, 801_120, 801_125, {}),
    # calls with a hit (1853, 4380, 4427), (11789, 68104, 68595)
    (5_000, 1_850, 1_860, {}),
    (70_000, 11_789, 11_789, {}),
    (70_000, 11_750, 11_850, {"use_graph": 1}),
    # the largest limit: low roots with the longest shared-prime rows
    (30_000_000, 1_104, 1_105, {}),
    # item weights from the finest cut (2^17 items a launch) to one item per block; heavy rows over several items
    (100_003, 32_032, 32_052, {"item_target": 1}),
    (100_003, 32_032, 32_152, {"item_target": 1 << 31}),
    (300_017, 160_215, 160_235, {"item_target": 1 << 17, "block_threads": 512}),
    (1_000_000, 801_125, 801_125, {"item_target": 1 << 20, "block_threads": 512}),
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
    (999, 100, 163),
    (1_000, 937, 1_000),
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


@pytest.fixture(scope="module")
def plain_long():
    with hss.Search(100_000) as s:
        r = s.search(1, 30_000, mode="plain", rows=True)
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["stream", "graph", "serving"])
def test_queues_grow_from_their_first_size(plain_long, form):
    """A long call from low roots at LIMIT 100,000, whose shared-prime pairs outgrow the 2 M entries a queue starts
    with: by a handle, under a graph, and by a serving lane (one wave of up to 41,943 rows)."""
    torch = pytest.importorskip("torch")
    with hss.Search(100_000, use_graph=int(form == "graph")) as s:
        before = torch.cuda.mem_get_info()[0]
        if form == "serving":
            s.serve_start(wave_mpairs=4_000)
            before = torch.cuda.mem_get_info()[0]
            done = s.wait(s.submit(1, 30_000))
            counts, hits = done["counts"], done["hits"]
        else:
            got = s.search(1, 30_000, rows=True)
            counts, hits = got.counts, got.hits
            assert got.row_candidates == plain_long.row_candidates
        grown = before - torch.cuda.mem_get_info()[0]
    # the larger queue and its descriptors, 48 Mi entries of 16 bytes and 8 Mi of 192, in place of the first ones of
    # 2 Mi and 0.5 Mi; not 3 GB of descriptors, and the rows, items and values of the call beside them
    larger = 48 * 16 + 8 * 192 - (2 * 16 + 96)
    assert larger <= grown / 2 ** 20 < larger + 1024
    assert {k: counts[k] for k in FIELDS} == {k: plain_long.counts[k] for k in FIELDS}
    assert sorted(hits) == sorted(plain_long.hits)


@pytest.mark.gpu
def test_rest_list_equals_rows_at_the_largest_limit():
    """A call of 65 roots leaves the common parts with few roots to the shared-prime kernels; calls of 64 and of one root
    make rows of all of them."""
    with hss.Search(30_000_000) as s:
        whole = s.search(1_041, 1_105, rows=True)
        parts = [s.search(1_041, 1_104, rows=True), s.search(1_105, 1_105, rows=True)]
    for key in FIELDS:
        assert whole.counts[key] == sum(p.counts[key] for p in parts), key
    assert whole.row_candidates == parts[0].row_candidates + parts[1].row_candidates
    assert whole.counts["launches"] > parts[0].counts["launches"]


@pytest.mark.gpu
def test_root_of_the_most_values(built):
    """15,413,645 has the most values of all roots with its common parts (13.3 M at the largest limit; with itself it shares
    all five split primes).  Its pairs up to 15,420,000 against the oracle."""
    from oracle import Oracle
    limit, root = 15_420_000, 15_413_645
    with Oracle(limit) as o:
        want = o.search(root, root)
    with hss.Search(limit) as s:
        got = s.search(root, root, rows=True)
    for key in ("pairs", "processed", "products", "candidates", "r16"):
        assert got.counts[key] == want[key], key
    assert got.row_candidates == want["row_candidates"]
