"""Which way a plan's long pairs went: the path from the rows their sweeps kept,
or Myers-Miller divisions throughout (`Plan.path_counts`). Both give the same
results, so a test that is about one of them has to ask. Results are compared
with the oracle all the same, every field and cell count equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("fwd_score", "se1", "se2", "sb1", "sb2", "mm_score", "n_ident", "n_match")


def run(ctx, oracle_mod, seqs, matrix, params, pairs, want=None):
    """The pairs of kept rows and the frames left over of one checked run."""
    if want is None:
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


def related(n, length, seed):
    """Copies of one sequence with a tenth of the residues replaced and a few lost."""
    rng = np.random.default_rng(seed)
    root = rng.integers(0, 20, size=length).astype(np.int8)
    out = []
    for _ in range(n):
        s = np.where(rng.random(length) < 0.1, rng.integers(0, 20, size=length), root).astype(np.int8)
        out.append(np.delete(s, rng.integers(0, length, size=3)))
    return out


def test_route_is_reported(oracle_mod):
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("protein")
    longs, shorts = related(6, 420, 3), related(6, 90, 4)
    pairs = synth.all_pairs(6)
    with native.Context(0) as ctx:
        ctx.set_cta_tuning(max_pairs=0)
        assert run(ctx, oracle_mod, longs, matrix, params, pairs)[0] == len(pairs)
        assert run(ctx, oracle_mod, shorts, matrix, params, pairs) == (0, 0)  # the short-pair kernel divides
        free = dict(params, pw_gap_extend=0.0)
        assert run(ctx, oracle_mod, longs, matrix, free, pairs) == (0, 0)


def gapped_pair(seed, head, middle, tail):
    """A sequence with `middle` letters that match nothing, and one without
    them; at the joint 17 letters that match on either side of the gap."""
    rng = np.random.default_rng(seed)
    a, b = (rng.integers(0, 4, size=k).astype(np.int8) for k in (head, tail))
    joint = rng.integers(4, 8, size=(3, 17)).astype(np.int8)
    return [np.concatenate([a, joint[0], np.full(middle, 8, np.int8), joint[1], b]), np.concatenate([a, joint[2], b])]


def scaled_scheme(match, mismatch, gap_open, gap_extend):
    """DNA rules (gap open 200, extension 100 per unit) over nine letters, of
    which 4 to 7 all match each other."""
    from clustalw_gb300 import load_matrix

    matrix, params = load_matrix("dna")
    matrix = np.full((32, 32), mismatch, dtype=np.int32)
    matrix[np.arange(4), np.arange(4)] = match
    matrix[4:8, 4:8] = match
    return matrix, dict(params, pw_gap_open=gap_open, pw_gap_extend=gap_extend)


@pytest.mark.parametrize("warps", [0, 16])  # one warp per pair, one CTA per pair
@pytest.mark.parametrize(
    "name, sizes, scheme, kept",
    [
        # A gap between two blocks of equal score that costs more than 2^28.
        ("costly gap", (9104, 8768, 16704), (32767, -32768, 0.5, 327.67), 0),
        # maxScore + gapOpen at 2^27: 4097 matches less the gap, and one more.
        ("largest score", (1500, 300, 2580), (32767, -32768, 1.0, 1.0), 1),
        ("score beyond", (1500, 300, 2581), (32767, -32768, 1.0, 1.0), 0),
        # gapExtend times the longer sequence at 2^28: 8192 residues, and 8193.
        ("largest gap", (4100, 7, 4051), (300, -300, 1.0, 327.67), 1),
        ("gap beyond", (4100, 7, 4052), (300, -300, 1.0, 327.67), 0),
    ],
)
def test_path_only_within_its_numbers(oracle_mod, warps, name, sizes, scheme, kept):
    from clustalw_gb300 import native

    matrix, params = scaled_scheme(*scheme)
    with native.Context(0) as ctx:
        if warps:
            ctx.set_cta_tuning(1 << 30, warps)
        else:
            ctx.set_cta_tuning(max_pairs=0)
        route = run(ctx, oracle_mod, gapped_pair(1, *sizes), matrix, params, np.array([[0, 1]], dtype=np.int32))
        assert route[0] == kept


def with_insertions(seed, parts, rows, columns):
    """A sequence of parts * rows letters, and one with `columns` random ones in
    the middle of each part: not at the rows diff() divides at down to the parts."""
    rng = np.random.default_rng(seed)
    halves = [rng.integers(0, 20, size=rows // 2).astype(np.int8) for _ in range(2 * parts)]
    second = []
    for a, b in zip(halves[::2], halves[1::2]):
        second += [a, rng.integers(0, 20, size=columns).astype(np.int8), b]
    return [np.concatenate(halves), np.concatenate(second)]


def test_many_frames_left_to_a_cta(oracle_mod):
    """Insertions wider than a box leave a frame each: more than the CTA takes
    from its list at a time, and, divided by the CTA down to two rows, more
    than its stack for one-warp frames holds."""
    from clustalw_gb300 import load_matrix, native

    matrix, params = load_matrix("dna")
    matrix = np.array(matrix)
    matrix[:20, :20] = np.where(np.eye(20, dtype=bool), 9, -4)
    params = dict(params, int_scale=1, pw_gap_open=10.0, pw_gap_extend=1.0)
    seqs, pairs = with_insertions(1, 64, 100, 430), np.array([[0, 1]], dtype=np.int32)
    want = oracle_mod.align_pairs(seqs, matrix, params, pairs)
    with native.Context(0) as ctx:
        for warps in (2, 4, 16):
            for large_rows in (2, 40, 0):
                ctx.set_cta_tuning(1 << 30, warps, large_rows)
                kept, left = run(ctx, oracle_mod, seqs, matrix, params, pairs, want)
                assert kept == 1 and left > 32


@pytest.mark.parametrize("warps", [0, 4])
def test_weak_alignments_are_divided(oracle_mod, warps):
    """Unrelated sequences leave nearly every column within a gap opening of the
    optimum, where kept rows cost more than divisions; so they do for boxes of few rows."""
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("protein")
    rng = np.random.default_rng(4)
    weak = [rng.integers(0, 20, size=600).astype(np.int8) for _ in range(8)]
    core = related(6, 60, 9)
    local = [np.concatenate([rng.integers(0, 20, size=250), c, rng.integers(0, 20, size=250)]).astype(np.int8) for c in core]
    strict, strict_params = load_matrix("dna")
    strict[:20, :20] = np.where(np.eye(20, dtype=bool), 9, -6)
    strict_params = dict(strict_params, int_scale=1, pw_gap_open=10.0, pw_gap_extend=1.0)
    with native.Context(0) as ctx:
        if warps:
            ctx.upload_seqs(synth.protein_family(60, 700, 1))
            ctx.set_matrix(matrix)
            ctx.set_params(params)
            ctx.align_pairs(np.array([[0, 1]], dtype=np.int32))  # memory for the kept rows of the small sets too
            ctx.set_cta_tuning(1 << 30, warps)
        else:
            ctx.set_cta_tuning(max_pairs=0)
        assert run(ctx, oracle_mod, weak, matrix, params, synth.all_pairs(8)) == (0, 0)
        assert run(ctx, oracle_mod, local, strict, strict_params, synth.all_pairs(6)) == (0, 0)
        assert run(ctx, oracle_mod, related(8, 600, 2), matrix, params, synth.all_pairs(8))[0] == 28


@pytest.mark.parametrize("warps", [0, 2])
def test_sets_of_one_stripe_are_divided(oracle_mod, warps):
    """Kept rows only in sets with more than 256 residues in some sequence."""
    from clustalw_gb300 import load_matrix, native

    matrix, params = load_matrix("protein")
    a, b = related(2, 303, 5)
    pairs = np.array([[0, 1], [1, 0]], dtype=np.int32)
    with native.Context(0) as ctx:
        if warps:
            ctx.set_cta_tuning(1 << 30, warps)
        else:
            ctx.set_cta_tuning(max_pairs=0)
        for n, kept in ((130, 0), (256, 0), (257, 2), (300, 2)):
            # More short sequences: a set of two would leave two warps too small a slice.
            seqs = [a[:n], b[:n]] + [b[:40]] * 8
            assert run(ctx, oracle_mod, seqs, matrix, params, pairs)[0] == kept


@pytest.mark.parametrize("warps", [0, 2, 4, 8, 16])
@pytest.mark.parametrize("n, length", [(3, 300), (4, 700), (10, 500), (6, 1523), (40, 300)])
def test_slices_fit_the_form_that_runs(oracle_mod, n, length, warps):
    """A new context's memory for kept rows is enough for a set's pairs, whichever
    form and width they run in; so the route does not depend on what the context
    held before."""
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("protein")
    pairs = synth.all_pairs(n)[-15:]
    with native.Context(0) as ctx:
        if warps:
            ctx.set_cta_tuning(1 << 30, warps)
        assert run(ctx, oracle_mod, related(n, length, 7), matrix, params, pairs)[0] == len(pairs)


def test_weak_pairs_among_related_ones_take_the_path(oracle_mod):
    """In a launch of mostly related pairs the weak ones go the same way; the
    longer ones here reach the choice after the others."""
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("protein")
    rng = np.random.default_rng(8)
    seqs = related(22, 300, 1) + [rng.integers(0, 20, size=600).astype(np.int8) for _ in range(8)]
    weak = synth.all_pairs(8) + 22
    pairs = np.concatenate([synth.all_pairs(22), weak, weak[:, ::-1]]).astype(np.int32)
    with native.Context(0) as ctx:
        ctx.set_cta_tuning(max_pairs=0)
        kept, left = run(ctx, oracle_mod, seqs, matrix, params, pairs)
        assert kept > 231 and left > 0


@pytest.mark.parametrize("n, length, ctas", [(20, 200, 1), (30, 250, 1), (38, 250, 0), (45, 200, 0), (45, 300, 1)])
def test_sets_of_one_stripe_run_as_many_ctas_as_fit(n, length, ctas):
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("protein")
    with native.Context(0) as ctx:
        ctx.set_matrix(matrix)
        ctx.set_params(params)
        ctx.upload_seqs(related(n, length, 3))
        plan = ctx.plan(synth.all_pairs(n))
        assert plan.pair_ctas() == bool(ctas)
        plan.close()


@pytest.mark.parametrize("warps", [2, 8, 16])
@pytest.mark.parametrize("scheme", ["protein", "dna"])
@pytest.mark.parametrize("kind", ["gaps", "close gaps", "wide gaps", "ties", "edges"])
def test_a_cta_walks_the_path(oracle_mod, kind, scheme, warps):
    """Rows, boxes and frames dealt over a CTA's warps, in a new context: gaps of
    two and more rows at every recursion level, gaps wider than a box, ties, and
    lengths around the rows kept and the rows of lanes and stripes."""
    from clustalw_gb300 import load_matrix, native, synth
    from test_gpu_path import sequences

    seqs = sequences(kind, 200 + len(kind))
    matrix, params = load_matrix(scheme)
    if scheme == "dna":
        seqs = [(s % 4).astype(np.int8) for s in seqs]
        matrix[:20, :20] = np.where(np.eye(20, dtype=bool), 9, -4)
        params = dict(params, int_scale=1, pw_gap_open=5.0, pw_gap_extend=2.0)
    up = synth.all_pairs(len(seqs))
    pairs = np.concatenate([up, up[:, ::-1]])
    with native.Context(0) as ctx:
        ctx.set_cta_tuning(1 << 30, warps)
        kept, left = run(ctx, oracle_mod, seqs, matrix, params, pairs)
    assert kept > 0
    if kind == "edges":
        assert (kept, left) == (len(pairs), 0)


@pytest.mark.parametrize("length, kept", [(1500, 1), (2200, 1), (3060, 1), (3200, 0)])
def test_rows_kept_further_apart_and_not_at_all(oracle_mod, length, kept):
    """With a slice for every warp of the long-pair kernel (sets of 56 sequences
    and more) one holds rows every 32 of 1500 residues, every 64 of 2200, every
    128 of 3060 and none of 3200."""
    from clustalw_gb300 import load_matrix, native

    matrix, params = load_matrix("protein")
    seqs = related(2, length + 3, 4) + related(62, 40, 5)
    with native.Context(0) as ctx:
        ctx.set_cta_tuning(max_pairs=0)
        assert run(ctx, oracle_mod, seqs, matrix, params, np.array([[0, 1]], dtype=np.int32))[0] == kept
