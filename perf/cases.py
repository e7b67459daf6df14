"""The work a ClustalW host program has this framework do, as timed cases.

Every case goes through the classes such a program calls: the full pairwise
distance stage (`FullPairwiseAlign.pairwiseAlign`), the quick k-tuple stage
(`FastPairwiseAlign.pairwiseAlign`), the guide tree (`NJTree.generateTree`) and
the serving loop (`Server`). All of them take host data (sequences, a packed
distance matrix) and leave host results, so a pass is the whole call.

Sequences are the seeded families of `clustalw_gb300.synth` with the shapes of
the repository's fixtures and benchmark workloads; distance matrices are
clustered, float32-valued and in [0, 1], as the pairwise stage stores them.
"""
import math
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cuda-clustalw_gb300"))

from clustalw_gb300 import load_matrix, native, pairwise, serve, synth, tree  # noqa: E402

# Cell updates (n * m summed over the pairs) of the largest listed case.
MOST_CELLS = 124750 * 1523 * 1523


def listed():
    return [
        # An interactive alignment of a handful of sequences: latency counts.
        full("full-protein-10x97", "protein", 10, 97),
        # The smallest shipped fixture, all pairs.
        full("full-protein-100x97", "protein", 100, 97),
        # The medium protein fixture.
        full("full-protein-100x498", "protein", 100, 498),
        # The headline family at half its number of sequences: throughput.
        full("full-protein-500x1523", "protein", 500, 1523),
        # DNA of a gene's length, the other alphabet and gap rule.
        full("full-dna-200x1002", "dna", 200, 1002),
        # A database extract: families of very different lengths in one set.
        full("full-uneven-200", "uneven", 200, 2000),
        # Adding one sequence to an alignment: a single column of the matrix.
        full("full-dna-column-100x1523", "dna", 100, 1523, column=True),
        # A few long proteins: far fewer pairs than the GPU has warps.
        full("full-protein-6x3000", "protein", 6, 3000),
        # The quick distances of a draft alignment.
        dict(name="quick-protein-200x1523", kind="quick", alphabet="protein", nseqs=200, length=1523),
        # Guide trees of a small and of a large set.
        dict(name="tree-100", kind="tree", nseqs=100),
        dict(name="tree-1000", kind="tree", nseqs=1000),
        # A service that aligns the sets of many users at once.
        dict(name="serve-24-jobs", kind="serve", jobs=24, nseqs=60, length=600),
    ]


def full(name, alphabet, nseqs, length, column=False):
    case = dict(kind="full", alphabet=alphabet, nseqs=nseqs, length=length, column=column)
    return dict(case, name=name) if name else case


def log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["full", "full", "full", "full", "column", "quick", "tree", "serve"])
    if kind in ("full", "column"):
        alphabet = rng.choice(["protein", "dna", "uneven"]) if kind == "full" else rng.choice(["protein", "dna"])
        length = log_int(rng, 30, 3000)
        most = 400 if kind == "column" else int(math.sqrt(0.25 * MOST_CELLS)) // length
        return full("", alphabet, log_int(rng, 4, max(5, min(400, most))), length, kind == "column")
    if kind == "quick":
        return dict(kind="quick", alphabet=rng.choice(["protein", "dna"]), nseqs=log_int(rng, 5, 200),
                    length=log_int(rng, 30, 2000))
    if kind == "tree":
        return dict(kind="tree", nseqs=log_int(rng, 5, 1000))
    return dict(kind="serve", jobs=rng.randint(2, 24), nseqs=log_int(rng, 10, 60), length=log_int(rng, 50, 600))


def sequences(case, seed):
    n, length = case["nseqs"], case["length"]
    if case["alphabet"] == "dna":
        return synth.dna_family(n, length, seed)
    if case["alphabet"] == "protein":
        return synth.protein_family(n, length, seed)
    # Families of log-uniform root lengths up to `length`, 25 sequences each.
    seqs = synth.uneven_protein(-(-n // 25), min(n, 25), min(30, length), length, seed)
    return seqs[:n]


def job_sets(case, seed):
    """Jobs of 4 to `nseqs` sequences of 30 to `length` residues: the sizes are
    the case's, the residues the seed's."""
    sizes = np.random.default_rng(case["jobs"])
    jobs = []
    for k in range(case["jobs"]):
        n = int(sizes.integers(4, case["nseqs"] + 1))
        length = int(sizes.integers(30, case["length"] + 1))
        jobs.append(synth.protein_family(n, length, seed * 1009 + k))
    return jobs


def distances(n, seed):
    """A packed DistMatrix of n sequences: clusters with noise, every distance
    of its own (float32 values in [0, 1], as the pairwise stage writes them)."""
    rng = np.random.default_rng(seed)
    centre = rng.normal(size=(max(2, n // 8), 4))
    pos = centre[rng.integers(0, len(centre), size=n)] + 0.3 * rng.normal(size=(n, 4))
    el = np.zeros((n + 1) * (n + 2) // 2)
    for a in range(1, n):
        v = np.linalg.norm(pos[:a] - pos[a], axis=1) / 8.0 + rng.uniform(0, 0.05, size=a)
        el[a * (a + 1) // 2 : a * (a + 1) // 2 + a] = np.minimum(v, 1.0).astype(np.float32)
    return el


def ranges(case):
    n = case["nseqs"]
    return (0, n, n - 2, n) if case["column"] else (0, n, 0, n)


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "tree":
        state.update(elements=distances(case["nseqs"], seed), matrix=pairwise.DistMatrix(case["nseqs"] + 1),
                     method=tree.NJTree(gpu=tree.NJGpu(0)), info=tree.SeqInfo(1, case["nseqs"], case["nseqs"]))
    elif kind == "serve":
        matrix, params = load_matrix("protein")
        state.update(jobs=job_sets(case, seed), server=serve.Server(matrix, params, memory_budget=1 << 30))
    else:
        state.update(alignment=pairwise.Alignment(sequences(case, seed)),
                     matrix=pairwise.DistMatrix(case["nseqs"] + 1))
        if kind == "full":
            matrix, params = load_matrix("dna" if case["alphabet"] == "dna" else "protein")
            state["method"] = pairwise.FullPairwiseAlign(pairwise.PairwiseSettings(matrix, params),
                                                         context=native.Context(0))
        else:
            state["method"] = pairwise.FastPairwiseAlign(dna=case["alphabet"] == "dna", context=native.Context(0))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "tree":
        # The tree joins its matrix in place, so every call starts from a copy.
        dist = state["matrix"]
        dist.getElements()[:] = state["elements"]
        phy = tree.PhyloTree()
        state["method"].generateTree(phy, dist, state["info"])
        return dict(left=phy.leftBranch, right=phy.rightBranch, desc=phy.treeDesc, joined=dist.getElements())
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(job) for job in state["jobs"]]
        out = []
        for job in ids:
            server.wait(job)
            out.append(server.result(job)[0])
            server.release(job)
        return out
    method, dist = state["method"], state["matrix"]
    if kind == "full":
        method.pairwiseAlign(state["alignment"], dist, *ranges(case))
        keys = ("fwd_score", "mm_score", "n_ident", "n_match")
    else:
        n = case["nseqs"]
        method.pairwiseAlign(state["alignment"], dist, 0, n, 0, n)
        keys = ("score", "frags")
    return dict(dist=dist.getElements(), **{k: method.last_stats[k] for k in keys})


def pair_total(case):
    return case["nseqs"] - 1 if case.get("column") else case["nseqs"] * (case["nseqs"] - 1) // 2


def work(case):
    """Bytes: residues (one byte each) or matrix in, results out. Operations:
    two sweeps of an alignment's cells (a score and its start) at 5 each; one
    per hit on a diagonal for the quick distances; 4 for each candidate pair of
    each join of the tree."""
    kind = case["kind"]
    n = case["nseqs"]
    if kind == "tree":
        return dict(bytes=16.0 * n * n / 2 + 4.0 * n * n, flops=4.0 * n**3 / 6)
    mean = case["length"]
    if kind == "serve":
        pairs = case["jobs"] * (n * n / 3.0) / 2
        cells = pairs * mean * mean / 3.0
        return dict(bytes=case["jobs"] * n * mean / 4.0 + 4.0 * pairs, flops=10.0 * cells)
    pairs = pair_total(case)
    cells = float(pairs) * mean * mean
    if kind == "quick":
        letters = 16 if case["alphabet"] == "dna" else 20
        return dict(bytes=n * mean + 24.0 * pairs, flops=cells / letters)
    if case["alphabet"] == "uneven":
        lo = min(30, mean)
        ratio = math.log(mean / lo) if mean > lo else 1.0
        cells = pairs * ((mean - lo) / ratio if mean > lo else mean) ** 2
        mean = math.sqrt(cells / pairs)
    return dict(bytes=n * mean + 40.0 * pairs, flops=10.0 * cells)


# ---------------------------------------------------------------- exact values


def gotoh_rows(a, b, sub, go, ge, top_h, top_e, left_h, left_f, corner, floor):
    """Yields row by row (H, E) of a global (or, with a floor, local) affine
    sweep over a x b. top_*: the row above, columns 1..m; left_h(r), left_f(r):
    column 0 of row r."""
    m = len(b)
    step = ge * np.arange(1, m + 1, dtype=np.int64)
    h, e, diag0 = top_h.copy(), top_e.copy(), corner
    for r, x in enumerate(a):
        e = np.maximum(e - ge, h - go - ge)
        diag = np.concatenate(([diag0], h[:-1])) + sub[x][b]
        best = np.maximum(diag, e)
        if floor is not None:
            best = np.maximum(best, floor)
        # F[c] = max(left F - c*ge, max over k < c of H[k] - go - (c - k)*ge)
        opened = np.concatenate(([left_h(r)], best[:-1] + step[:-1])) - go
        f = np.maximum(np.maximum.accumulate(opened), left_f(r)) - step
        h = np.maximum(best, f)
        diag0 = left_h(r)
        yield h, e


def exact_pair(a, b, sub, go, ge, len1, len2):
    """One pair's distance by the published algorithm of the reference's
    pairwise stage (local score, start cell, Myers-Miller), on whole numbers."""
    n, m = len(a), len(b)
    zero, cost = np.zeros(m, np.int64), 0
    end = (0, 0)
    for r, (h, _) in enumerate(gotoh_rows(a, b, sub, go, ge, zero, zero - go, lambda r: 0, lambda r: -go, 0, 0)):
        c = int(np.argmax(h))
        if h[c] > cost:
            cost, end = int(h[c]), (r + 1, c + 1)
    if cost == 0:
        return 1.0
    ar, br = a[: end[0]][::-1], b[: end[1]][::-1]
    minus = np.full(len(br), -1, np.int64)
    start = end
    for r, (h, _) in enumerate(gotoh_rows(ar, br, sub, go, ge, minus, minus, lambda r: -1, lambda r: -1, 0, None)):
        hit = np.flatnonzero(h >= cost)
        if len(hit):
            start = (end[0] - r, end[1] - int(hit[0]))
            break
    box_a, box_b = a[start[0] - 1 : end[0]], b[start[1] - 1 : end[1]]
    ident = myers_miller(box_a, box_b, sub, go, ge)
    mm = 100.0 * ident / min(len1, len2) if len1 and len2 else 0.0
    return (100.0 - mm) / 100.0


def myers_miller(a, b, sub, go, ge):
    """Identities on the path diff() chooses."""
    ident = 0
    stack = [(0, 0, len(a), len(b), 0, 0)]
    while stack:
        A, B, M, N, tb, te = stack.pop()
        if N <= 0 or M <= 0:
            continue
        x, y = a[A : A + M], b[B : B + N]
        j = np.arange(N + 1)
        if M == 1:
            k = j[1:]
            value = sub[x[0]][y]
            value = value - np.where(N - k > 0, te + ge * (N - k), 0) - np.where(k > 1, tb + ge * (k - 1), 0)
            at = int(np.argmax(value))
            if value[at] > max(-(tb + ge) - (te + ge * N), -(te + ge) - (tb + ge * N)):
                ident += int(x[0] == y[at] and x[0] < 30)
            continue
        mid = M // 2

        def last(rows, cols, open_):
            top = -open_ - ge * np.arange(1, N + 1, dtype=np.int64)
            edge = lambda r: -open_ - ge * (r + 1)  # noqa: E731
            for h, e in gotoh_rows(rows, cols, sub, go, ge, top, top - go, edge, lambda r: edge(r) - go, 0, None):
                pass
            side = edge(len(rows) - 1)
            return np.concatenate(([side], h)), np.concatenate(([side], e))

        hh, dd = last(x[:mid], y, tb)
        rr, ss = last(x[mid:][::-1], y[::-1], te)
        rr, ss = rr[::-1], ss[::-1]
        one, two = hh + rr, dd + ss + go
        best = int(one.max())
        ties = np.flatnonzero(one == best)
        later = ties[(hh[ties] != dd[ties]) & (rr[ties] == ss[ties])]
        col = int(later[-1]) if len(later) else int(ties[0])
        if two.max() > best:
            col = int(np.flatnonzero(two == two.max())[-1])
            stack += [(A + mid + 1, B + col, M - mid - 1, N - col, 0, te), (A, B, mid - 1, col, tb, 0)]
        else:
            stack += [(A + mid, B + col, M - mid, N - col, go, te), (A, B, mid, col, tb, go)]
    return ident


def exact_full(case, seed):
    seqs = [np.asarray(s).astype(np.int64) for s in sequences(case, seed)]
    matrix, p = load_matrix("dna" if case["alphabet"] == "dna" else "protein")
    sub = matrix.astype(np.int64)
    i0, i1, j0, j1 = ranges(case)
    out = np.zeros((case["nseqs"] + 1) * (case["nseqs"] + 2) // 2)
    for i in range(i0, i1):
        for j in range(max(i + 1, j0 + 1), j1):
            go, ge = native.gap_penalties(p, len(seqs[i]), len(seqs[j]))
            d = exact_pair(seqs[i], seqs[j], sub, go, ge, len(seqs[i]), len(seqs[j]))
            out[j * (j + 1) // 2 + i] = d
    return out


def exact_tree(n, el):
    """Neighbour joining (Saitou and Nei) with the reference's rules, in 64 bits."""
    lo = np.zeros((n, n))
    for a in range(1, n):
        lo[a, :a] = el[a * (a + 1) // 2 : a * (a + 1) // 2 + a]
    d = lo + lo.T
    live = np.ones(n, bool)
    av = np.zeros(n)
    left, right = np.zeros(n + 2), np.zeros(n + 2)
    small = lambda x: 0.0 if abs(x) < 0.0001 else x  # noqa: E731
    for nc in range(1, n - 2):
        k = np.flatnonzero(live)
        f = float(len(k) - 2)
        s = d[np.ix_(k, k)].sum(axis=1)
        t = f * d[np.ix_(k, k)] - s[:, None] - s[None, :]
        t[np.triu_indices(len(k))] = np.inf
        row, col = np.unravel_index(int(np.argmin(t)), t.shape)  # rows are the larger index
        i, j = k[col], k[row]
        dmin = d[i, j]
        bi = (dmin + (s[col] - dmin) / f - (s[row] - dmin) / f) * 0.5
        bj = dmin - bi
        left[nc], right[nc] = small(bi - av[i]), small(bj - av[j])
        av[i] = (dmin if dmin > 0 else 0.000001) * 0.5
        live[j] = False
        new = (d[i] + d[j]) * 0.5
        keep = live.copy()
        keep[i] = False
        d[i, keep] = d[keep, i] = new[keep]
        d[j, :] = d[:, j] = 0.0
    k = np.flatnonzero(live)
    b1 = (d[k[0], k[1]] + d[k[0], k[2]] - d[k[1], k[2]]) * 0.5
    for at, b, i in ((n - 2, b1, k[0]), (n - 1, d[k[0], k[1]] - b1, k[1]), (n, d[k[0], k[2]] - b1, k[2])):
        left[at] = small(b - av[i])
    joined = np.zeros_like(el)
    for a in range(1, n):
        joined[a * (a + 1) // 2 : a * (a + 1) // 2 + a] = d[a, :a]
    return left, right, joined


def exact(case, seed):
    """Distances of small sets and branch lengths in 64 bits. The quick
    distances and the served ones follow from whole numbers that are compared
    as such, and large sets take too long here."""
    if case["kind"] == "tree" and case["nseqs"] <= 500:
        left, right, joined = exact_tree(case["nseqs"], distances(case["nseqs"], seed))
        return dict(left=left, right=right, desc=None, joined=joined)
    if case["kind"] == "full" and pair_total(case) * case["length"] <= 20000:
        return dict(dist=exact_full(case, seed), fwd_score=None, mm_score=None, n_ident=None, n_match=None)
    return None
