"""Which way a plan's long pairs went: the path from the rows their sweeps kept,
or Myers-Miller divisions throughout (`Plan.path_counts`). Both give the same
results, so a test that is about one of them has to ask. Results are compared
with the oracle all the same, every field and cell count equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("fwd_score", "se1", "se2", "sb1", "sb2", "mm_score", "n_ident", "n_match")


def run(ctx, oracle_mod, seqs, matrix, params, pairs):
    """The pairs of kept rows and the frames left over of one checked run."""
    want = oracle_mod.align_pairs(seqs, matrix, params, pairs)
    ctx.set_matrix(matrix)
    ctx.set_params(params)
    ctx.upload_seqs(seqs)
    plan = ctx.plan(pairs)
    plan.launch()
    dist, stats = plan.results(stats=True)
    cells, route = plan.cell_counts(), plan.path_counts()
    plan.close()
    assert np.array_equal(dist, want["dist"])
    for f in FIELDS:
        assert np.array_equal(stats[f], want[f]), f
    assert cells == tuple(int(want[c].sum()) for c in ("cells_fwd", "cells_rev", "cells_diff"))
    return route


def test_route_is_reported(oracle_mod):
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("protein")
    longs, shorts = synth.protein_family(6, 420, 3), synth.protein_family(6, 90, 4)
    pairs = synth.all_pairs(6)
    with native.Context(0) as ctx:
        ctx.set_cta_tuning(max_pairs=0)
        assert run(ctx, oracle_mod, longs, matrix, params, pairs)[0] == len(pairs)
        assert run(ctx, oracle_mod, shorts, matrix, params, pairs) == (0, 0)  # the short-pair kernel divides
        free = dict(params, pw_gap_extend=0.0)
        assert run(ctx, oracle_mod, longs, matrix, free, pairs) == (0, 0)
