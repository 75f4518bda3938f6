"""Which schedules the autotuner times: no two that run the same kernels."""


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
