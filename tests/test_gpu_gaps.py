"""The two forms of the pair kernels, chosen by the gap penalties: the usual one
pads a sweep's rows with a row of very low scores, which is sound for gap open
>= 0 and 0 <= extension <= 32767; other penalties take the general form. Both
against the oracle, every distance and intermediate equal (whole numbers), at
lengths around the rows per lane (4, 8), the lanes of a stripe and the
stripes, through every entry point that picks a form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = (1, 2, 3, 4, 5, 7, 8, 9, 31, 33, 63, 64, 65, 127, 128, 129, 191, 255, 256, 257, 264, 300)
FIELDS = ("fwd_score", "se1", "se2", "sb1", "sb2", "mm_score", "n_ident", "n_match")

# (gap open, gap extension) as the reference's floats; DNA rules: the integers
# are 2 * 100 * open and 100 * extension.
PENALTIES = {
    "no penalties": (0.0, 0.0),
    "free extension": (3.0, 0.0),
    "extension 1": (3.0, 0.01),
    "largest padded extension": (1.0, 327.67),
    "smallest general extension": (1.0, 327.68),
    "extension beyond every score": (2.0, 5000.0),
    "negative open": (-0.5, 0.2),
    "negative extension": (5.0, -0.03),
}


def sequences(seed):
    """One sequence of every length, mutated from one root so that they align."""
    rng = np.random.default_rng(seed)
    root = rng.integers(0, 4, size=max(LENGTHS)).astype(np.int8)
    out = []
    for n in LENGTHS:
        s = root[(max(LENGTHS) - n) // 2 :][:n].copy()
        hit = rng.random(n) < 0.2
        s[hit] = rng.integers(0, 4, size=int(hit.sum()))
        out.append(s)
    return out


@pytest.mark.parametrize("name", sorted(PENALTIES))
def test_gap_penalty_forms(oracle_mod, name):
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("dna")
    matrix = np.array(matrix)
    rng = np.random.default_rng(5)
    m4 = rng.integers(-900, 1200, size=(4, 4))
    matrix[:4, :4] = (m4 + m4.T) // 2 + 900 * np.eye(4, dtype=np.int64)
    params["pw_gap_open"], params["pw_gap_extend"] = PENALTIES[name]
    seqs = sequences(17)
    up = synth.all_pairs(len(seqs))
    pairs = np.concatenate([up, up[:, ::-1]])
    want = oracle_mod.align_pairs(seqs, matrix, params, pairs)

    def same(dist, stats):
        assert np.array_equal(dist, want["dist"])
        for f in FIELDS:
            assert np.array_equal(stats[f], want[f]), f

    with native.Context(0) as ctx:
        ctx.set_matrix(matrix)
        ctx.set_params(params)
        ctx.upload_seqs(seqs)
        same(*ctx.align_pairs(pairs, stats=True))  # few long pairs: one CTA per pair
        ctx.set_cta_tuning(max_pairs=0)
        same(*ctx.align_pairs(pairs, stats=True))  # one warp per pair
        ctx.set_tuning(0, 0, 300)  # every pair in the short-pair kernel, no tiny frames
        same(*ctx.align_pairs(pairs, stats=True))
        plan = ctx.plan(pairs)
        plan.launch()
        same(*plan.results(stats=True))
        plan.close()
