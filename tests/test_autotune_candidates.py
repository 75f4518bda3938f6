"""Which schedules the autotuner times, and on how many queries: no two that
run the same kernels, and a thread against a warp per query on all queries."""
import torch


def grid(rtd):
    return {"leaf_size": [2, 4, 8], "morton_bits": [42, 48],
            "radius_heuristic": [rtd.RADIUS_SAMPLED_NN, rtd.RADIUS_MORTON_WINDOW],
            "radius_param": [0.25, 0.5], "radius_increment_mult": [2.0, 4.0], "block_size": [128, 256],
            "mode": ["thread", "warp"]}


def test_exact_searches_do_not_sweep_the_radius(rtd):
    from rtdsl import autotune
    for k, n, threads in ((5, 1_000_000, True), (16, 1_000_000, True), (17, 1_000_000, False),
                          (2_048, 1_000_000, False), (5_000, 2_048, False)):
        cands = autotune._candidates(grid(rtd), k, n)
        assert len({(c["radius_heuristic"], c["radius_param"], c["radius_increment_mult"]) for c in cands}) == 1
        thread = [c for c in cands if c["lanes_per_query"] == 1]
        assert len(thread) == (3 * 2 * 2 if threads else 0)
        assert len(cands) - len(thread) == 3 * 2   # the collecting search takes no block size


def test_the_longest_lists_sweep_the_radius(rtd):
    from rtdsl import autotune
    cands = autotune._candidates(grid(rtd), 2_049, 5_000)
    assert {c["radius_heuristic"] for c in cands} == {rtd.RADIUS_SAMPLED_NN}
    assert len(cands) == 3 * 2 * 2 * 2 * 2 and {c["lanes_per_query"] for c in cands} == {32}


def test_batches_sweep_the_radius_for_long_lists_only(rtd):
    from rtdsl import autotune
    g = {"leaf_size": [8, 32], "radius_param": [0.5, 1.0, 2.0], "radius_increment_mult": [2.0, 4.0],
         "lanes_per_query": [0, 32]}
    assert len(autotune._batch_candidates(g, [(1_000, 10, 5), (9_000, 10, 512), (100, 10, 900), (9_000, 0, 900)])) == 4
    assert len(autotune._batch_candidates(g, [(1_000, 10, 5), (9_000, 10, 513)])) == 24


def test_modes_are_compared_on_all_queries(rtd):
    """A warp per query is ahead up to 50,000 queries, a thread per query
    beyond, as the searches are."""
    from rtdsl import autotune
    asked = []

    def time_fn(kw, m):
        asked.append((kw["lanes_per_query"], m))
        ms = 0.15 + kw["leaf_size"] * 1e-3 if kw["lanes_per_query"] == 1 else m * 2.5e-6 + kw["leaf_size"] * 1e-3
        return ms, torch.zeros(m, dtype=torch.int32)

    cands = autotune._candidates(grid(rtd), 5, 1_000_000)
    for nq, lanes in ((400_000, 1), (100_000, 1), (20_000, 32), (3_000, 32)):
        asked.clear()
        table = autotune._funnel(cands, nq, time_fn)
        assert len(table) == 1 and table[0][1]["lanes_per_query"] == lanes and table[0][1]["leaf_size"] == 2
        assert {x for x, m in asked if m == nq} == {1, 32}


def test_different_neighbours_are_refused_across_modes(rtd):
    import pytest
    from rtdsl import autotune

    def time_fn(kw, m):
        return 1.0, torch.full((m,), kw["lanes_per_query"], dtype=torch.int32)

    with pytest.raises(RuntimeError, match="different neighbours"):
        autotune._funnel(autotune._candidates(grid(rtd), 5, 1_000), 100, time_fn)
