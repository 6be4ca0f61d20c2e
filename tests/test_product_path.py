"""The product path, which calls of more than 64 roots below LIMIT 10,000 take: every compiled variant of its kernel, under a
graph, and as the autotuner leaves it, on roots with a hit (1853) against the plain form."""
import pytest

import hss

pytestmark = pytest.mark.gpu

FIELDS = ("pairs", "processed", "products", "candidates", "r16", "merged", "merged_products", "merged_candidates", "merged_r16")
LIMIT, FIRST, LAST = 5_000, 1_800, 1_900


@pytest.fixture(scope="module")
def plain():
    with hss.Search(LIMIT) as s:
        r = s.search(FIRST, LAST, mode="plain", rows=True)
    assert [h[:3] for h in r.hits] == [(1853, 4380, 4427)]
    return r


def check(got, plain):
    assert {k: got.counts[k] for k in FIELDS} == {k: plain.counts[k] for k in FIELDS}
    assert got.row_candidates == plain.row_candidates
    assert got.hits == plain.hits


@pytest.mark.parametrize("opts", [
    {"block_threads": 128, "ctas_per_sm": 4},
    {"block_threads": 128, "ctas_per_sm": 6},
    {"block_threads": 256, "ctas_per_sm": 2},
    {"block_threads": 256, "ctas_per_sm": 3},
    {"block_threads": 512, "ctas_per_sm": 1},
    {"use_graph": 1},
    {"use_graph": 1, "block_threads": 128},
    {"item_target": 1 << 14},
], ids=lambda o: "-".join(f"{k}{v}" for k, v in o.items()))
def test_variants(plain, opts):
    with hss.Search(LIMIT, **opts) as s:
        for _ in range(2):
            got = s.search(FIRST, LAST, rows=True)
            check(got, plain)
            assert (got.counts["graph_launches"] >= 1) == ("use_graph" in opts)


def test_autotuned(plain):
    with hss.Search(LIMIT) as s:
        chosen, trials = s.autotune(FIRST, LAST)
        assert len(trials) == len({t[:3] for t in trials}) and chosen["block_threads"] in (128, 256, 512)
        check(s.search(FIRST, LAST, rows=True), plain)


def test_graph_alternates_between_the_paths(plain):
    """One handle's graph, rebuilt or updated as calls go by products (101 roots) and by arcs (11 and 64 roots)."""
    with hss.Search(LIMIT, use_graph=1) as s, hss.Search(LIMIT) as streamed:
        for _ in range(2):
            check(s.search(FIRST, LAST, rows=True), plain)
            for first, last in ((1_850, 1_860), (1_801, 1_864)):
                got, want = s.search(first, last, rows=True), streamed.search(first, last, mode="plain", rows=True)
                check(got, want)
                assert got.counts["graph_launches"] >= 1


def test_handles_of_two_threads(plain):
    """Handles opened, searched by products, by arcs and by the plain form, and closed by two threads at a time, with rows of
    different weight: no launch meets the other thread's shared-memory limit."""
    import threading
    cases = [(LIMIT, 1_800, 1_900), (300_017, 160_225, 160_225)]
    want = {}
    for limit, first, last in cases:
        with hss.Search(limit) as s:
            want[limit] = s.search(first, last, mode="plain", rows=True)
    failures = []

    def work(limit, first, last):
        try:
            for _ in range(12):
                with hss.Search(limit) as s:
                    for mode in ("batched", "plain"):
                        check(s.search(first, last, mode=mode, rows=True), want[limit])
        except Exception as e:  # handed to the main thread
            failures.append(e)

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
