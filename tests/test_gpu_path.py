"""The path of the long-pair kernel (csrc/cwgpu_path.cuh): the rows the local
sweeps keep, the boxes between them, the walk over diff()'s frames and what is
left to Myers-Miller. Every distance, intermediate and cell count equal to the
oracle's, on sequences built for the places where it could go wrong: gaps of
two and more rows at every recursion level, gaps close together (horizontal
gaps at free corners), gaps wider than a box, ties, weak alignments, and sets
whose slices only hold the wider row spacings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("fwd_score", "se1", "se2", "sb1", "sb2", "mm_score", "n_ident", "n_match")


def mutate(rng, seq, letters, sub, spacing, longest):
    out = [int(c) if rng.random() >= sub else int(rng.integers(letters)) for c in seq]
    pos = int(rng.integers(2, 20))
    while pos < len(out) - 2:
        k = int(rng.integers(1, longest + 1))
        if rng.random() < 0.5:
            del out[pos : pos + k]
        else:
            out[pos:pos] = rng.integers(0, letters, size=k).tolist()
            pos += k
        pos += int(rng.integers(1, spacing + 1))
    return np.array(out or [0], dtype=np.int8)


def sequences(kind, seed):
    rng = np.random.default_rng(seed)
    root = rng.integers(0, 20, size=420).astype(np.int8)
    if kind == "gaps":
        return [mutate(rng, root, 20, 0.2, 60, 9) for _ in range(9)]
    if kind == "close gaps":
        return [mutate(rng, root, 20, 0.05, 12, 4) for _ in range(9)]
    if kind == "wide gaps":
        far = [np.concatenate([root[:150], rng.integers(0, 20, size=k).astype(np.int8), root[150:]])
               for k in (0, 60, 400, 900)]
        return far + [np.concatenate([root[:100], root[300:]]), root[40:].copy()]
    if kind == "ties":
        unit = root[:7]
        return [np.tile(unit, k) for k in (20, 31, 45)] + [np.zeros(n, np.int8) for n in (129, 160, 257)] + [root]
    if kind == "weak":
        return [rng.integers(0, 20, size=int(n)).astype(np.int8) for n in rng.integers(130, 600, size=8)]
    if kind == "edges":  # saved rows every 32, lanes of 8 rows, stripes of 256
        return [root[: n].copy() for n in (129, 136, 159, 160, 161, 191, 192, 193, 255, 256, 257, 288)]
    raise ValueError(kind)


def check(ctx, oracle_mod, seqs, matrix, params, pairs, cta_warps=0):
    want = oracle_mod.align_pairs(seqs, matrix, params, pairs)
    ctx.set_matrix(matrix)
    ctx.set_params(params)
    ctx.upload_seqs(seqs)
    if cta_warps:
        ctx.set_cta_tuning(1 << 30, cta_warps)  # one CTA of that many warps per pair
    else:
        ctx.set_cta_tuning(max_pairs=0)  # one warp per pair
    plan = ctx.plan(pairs)
    plan.launch()
    dist, stats = plan.results(stats=True)
    cells = plan.cell_counts()
    plan.close()
    assert np.array_equal(dist, want["dist"])
    for f in FIELDS:
        assert np.array_equal(stats[f], want[f]), f
    assert cells == tuple(int(want[c].sum()) for c in ("cells_fwd", "cells_rev", "cells_diff"))


@pytest.mark.parametrize("scheme", ["protein", "small extension", "cheap gaps", "free extension", "dna"])
@pytest.mark.parametrize("kind", ["gaps", "close gaps", "wide gaps", "ties", "weak", "edges"])
def test_path_matches_oracle(oracle_mod, kind, scheme):
    from clustalw_gb300 import load_matrix, native, synth

    seqs = sequences(kind, 100 + len(kind) + len(scheme))
    matrix, params = load_matrix("protein" if scheme == "protein" else "dna")
    if scheme != "protein":
        seqs = [(s % 4).astype(np.int8) if scheme == "dna" else s for s in seqs]
        matrix = np.array(matrix)
        matrix[:20, :20] = np.where(np.eye(20, dtype=bool), 9, -4)
        params["int_scale"] = 1
        params["pw_gap_open"], params["pw_gap_extend"] = {
            "small extension": (10.0, 1.0), "cheap gaps": (2.0, 1.0), "free extension": (6.0, 0.0), "dna": (5.0, 2.0)
        }[scheme]
    up = synth.all_pairs(len(seqs))
    with native.Context(0) as ctx:
        check(ctx, oracle_mod, seqs, matrix, params, np.concatenate([up, up[:, ::-1]]))


def test_path_wider_row_spacing(oracle_mod):
    """As many slices as the kernel has warps, in a set whose longest sequence
    leaves them room for rows every 64 or 128 only, or for none."""
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("protein")
    longs = [s for n in (700, 1500, 2200, 3000) for s in synth.protein_family(2, n, n)]
    seqs = longs + synth.protein_family(56, 40, 5)
    pairs = np.array([(i, j) for i in range(8) for j in range(8) if i != j], dtype=np.int32)
    with native.Context(0) as ctx:
        check(ctx, oracle_mod, seqs, matrix, params, pairs)


def test_path_free_corners_near_the_ends(oracle_mod):
    """Pairs in which diff() grants a free horizontal gap at a type 2 corner and
    ends along the box's edge before the next kept row: four found among the
    benchmark family's and another family's pairs."""
    from conftest import GOLDEN

    from clustalw_gb300 import load_matrix, native, synth

    z = np.load(f"{GOLDEN}/bench_protein_1000x1523.npz")
    offs = np.concatenate([[0], np.cumsum(z["lens"])[:-1]])
    seqs = [z["codes"][offs[i] : offs[i] + z["lens"][i]].astype(np.int8) for i in (417, 982, 475, 893, 723, 842)]
    matrix, params = load_matrix("protein")
    with native.Context(0) as ctx:
        check(ctx, oracle_mod, seqs, matrix, params, np.array([[0, 1], [2, 3], [4, 5]], dtype=np.int32))
        model = dict(synth.PROTEIN_MODEL, indel=0.02, depth=8.0)
        family = synth.family(600, 200, 6, model)
        params["pw_gap_open"], params["pw_gap_extend"] = 4.0, 0.2
        i, j = synth.all_pairs(600)[54841]
        check(ctx, oracle_mod, [family[i], family[j]], matrix, params, np.array([[0, 1], [1, 0]], dtype=np.int32))


@pytest.mark.parametrize("warps", [2, 8, 16])
@pytest.mark.parametrize("kind", ["gaps", "close gaps", "wide gaps", "ties", "weak", "edges"])
def test_path_shared_by_a_cta(oracle_mod, kind, warps):
    """The rows, the boxes and the walk's frames dealt over a CTA's warps."""
    from clustalw_gb300 import load_matrix, native, synth

    seqs = sequences(kind, 200 + len(kind))
    matrix, params = load_matrix("protein")
    up = synth.all_pairs(len(seqs))
    with native.Context(0) as ctx:
        check(ctx, oracle_mod, seqs, matrix, params, np.concatenate([up, up[:, ::-1]]), cta_warps=warps)
