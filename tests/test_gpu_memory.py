"""Device memory for kept rows is optional: with hardly any free, calls succeed
as far as their own buffers fit, plans made before stay good, and memory that
is free again is used again. The device is filled by one allocation, down to a
few hundred MB, and given back at once."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def device_full(leave):
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    block = torch.empty(free - leave, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del block
        torch.cuda.empty_cache()


def related(n, length, seed):
    rng = np.random.default_rng(seed)
    root = rng.integers(0, 20, size=length).astype(np.int8)
    return [np.where(rng.random(length) < 0.1, rng.integers(0, 20, size=length), root).astype(np.int8) for _ in range(n)]


@pytest.fixture()
def held():
    """A context that holds 1 GB for kept rows, and a plan of it that has run."""
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("protein")
    with native.Context(0) as ctx:
        ctx.set_matrix(matrix)
        ctx.set_params(params)
        for n in (6, 60):  # both forms of the kernel have run before memory is short
            ctx.upload_seqs(related(n, 700, 1))
            plan = ctx.plan(synth.all_pairs(n))
            plan.launch()
            want = plan.results(stats=True)
        yield ctx, plan, want
        plan.close()


def test_a_plan_takes_the_memory_and_an_older_one_still_runs(held):
    ctx, plan, want = held
    assert plan.path_counts()[0] == 1770
    pairs = np.zeros((8 << 20, 2), dtype=np.int32)  # 48 bytes each
    with device_full(leave=256 * MB):
        big = ctx.plan(pairs)
        plan.launch()
        got = plan.results(stats=True)
        kept = plan.path_counts()[0]
        big.close()
    assert kept == 0
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_a_longer_set_takes_the_memory(held, oracle_mod):
    from clustalw_gb300 import load_matrix

    ctx, _, _ = held
    matrix, params = load_matrix("protein")
    seqs, pairs = related(2, 9000, 2), np.array([[0, 1]], dtype=np.int32)
    want = oracle_mod.align_pairs(seqs, matrix, params, pairs)
    with device_full(leave=256 * MB):
        ctx.upload_seqs(seqs)  # boundary rows of 438 MB
        dist, stats = ctx.align_pairs(pairs, stats=True)
    assert np.array_equal(dist, want["dist"]) and stats["n_ident"][0] == want["n_ident"][0]


def test_memory_is_asked_for_again(held):
    from clustalw_gb300 import load_matrix, native, synth

    matrix, params = load_matrix("protein")
    seqs, pairs = related(56, 600, 3), synth.all_pairs(56)
    with native.Context(0) as ctx:
        ctx.set_matrix(matrix)
        ctx.set_params(params)
        kept = []
        for leave in (256 * MB, 0):
            with device_full(leave) if leave else contextlib.nullcontext():
                ctx.upload_seqs(seqs)
                plan = ctx.plan(pairs)
                plan.launch()
                dist = plan.results()
                kept.append((plan.path_counts()[0], dist))
                plan.close()
    assert kept[0][0] < kept[1][0] == len(pairs)
    assert np.array_equal(kept[0][1], kept[1][1])


def test_a_server_needs_only_its_own_buffers():
    """Created with room for the job memory and the boundary rows, but not for
    kept rows beside them, and with buffers of a first round to come."""
    from clustalw_gb300 import load_matrix, native, serve, synth

    matrix, params = load_matrix("protein")
    jobs = [related(40, 400, 5), related(300, 40, 6)]
    with native.Context(0) as ctx:  # kernels loaded and stacks taken before memory is short
        ctx.set_matrix(matrix)
        ctx.set_params(params)
        want = []
        for seqs in jobs:
            ctx.upload_seqs(seqs)
            ctx.set_cta_tuning(max_pairs=0)
            want.append(ctx.align_pairs(synth.all_pairs(len(seqs))))
    # 512 MB of job memory; rows: 2 rounds x 6,080 warps x 2 x 4,097 x 8 bytes = 797 MB;
    # one round's kept rows would be 1 GB more.
    with device_full(leave=2000 * MB):
        with serve.Server(matrix, params, memory_budget=512 * MB) as server:
            ids = [server.submit(seqs) for seqs in jobs]
            for job, w in zip(ids, want):
                server.wait(job)
                assert np.array_equal(server.result(job)[0], w)
                server.release(job)
