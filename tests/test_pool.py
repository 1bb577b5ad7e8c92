"""Blocks kept for the next session: size classes, the bound and what goes first, memory given back when an allocation fails (all on a
source that only counts), and on the GPU a session on a block that held something else, and a matrix that needs the idle blocks' memory."""
import importlib

import numpy as np
import pytest

import modelgen
from dflb import pkg

MB = 1 << 20


@pytest.mark.parametrize("host", [False, True])
def test_a_returned_block_serves_the_next_of_its_size(host):
    t = pkg.pool_selftest([3 * MB, -1, 3 * MB, -2, 3 * MB - 600, 3 * MB], 64 * MB, 1 << 40, host)
    assert t[:, 2].tolist() == [1, 1, 1, 1, 1, 2]     # the last one while its block is in use
    assert pkg.pool_selftest([0, 1, -1, 0], MB, MB, host)[:, 1].tolist() == [0, 512, 512, 0]


@pytest.mark.parametrize("host,classes,more", [(False, 16, 1 / 16), (True, 8, 1 / 8)])
def test_sizes_that_all_differ_share_a_few_blocks(host, classes, more):
    sizes = np.random.default_rng(3).permutation(np.arange(4 * MB, 8 * MB, 12345))
    ops = [x for i, n in enumerate(sizes) for x in (int(n), -i - 1)]
    t = pkg.pool_selftest(ops, 1 << 40, 1 << 40, host)
    assert t[-1, 2] <= classes + 1
    for n in sizes[:50]:
        assert n <= pkg.pool_selftest([int(n)], 0, 1 << 40, host)[0, 1] <= n * (1 + more) + 512


def test_the_block_returned_longest_ago_makes_room():
    sizes = [1 * MB << i for i in range(4)]                  # 1, 2, 4, 8 MB; room for 12
    ops = sizes + [-1, -2, -3, -4]
    t = pkg.pool_selftest(ops + [8 * MB, 4 * MB, 2 * MB], 12 * MB, 1 << 40)
    assert t[7, 1] == 12 * MB                                # 1 and 2 MB went, 4 and 8 stay
    assert t[8:, 2].tolist() == [4, 4, 5]
    # a process whose sizes never come again keeps the newest, not the first
    sizes = [(10 + i) * MB for i in range(0, 60, 3)]
    ops = [x for i, n in enumerate(sizes) for x in (n, -i - 1)]
    t = pkg.pool_selftest(ops + [sizes[-1]], 100 * MB, 1 << 40)
    assert t[-1, 2] == t[-2, 2] and t[:, 1].max() <= 100 * MB + max(sizes) * 17 // 16
    # larger than the bound: not kept
    assert pkg.pool_selftest([5 * MB, -1], 4 * MB, 1 << 40)[:, 1].tolist() == [5 * MB, 0]


def test_idle_blocks_are_given_back_when_memory_runs_out():
    t = pkg.pool_selftest([4 * MB, 4 * MB, -1, -2, 6 * MB, 6 * MB], 64 * MB, 10 * MB)
    assert t[:, 0].tolist() == [1, 1, 1, 1, 1, 0] and t[4, 1] == 6 * MB
    # what fits without the class's rounding is not refused, and goes back to the source when returned
    odd = 4 * MB + 512
    t = pkg.pool_selftest([odd, -1, odd], 64 * MB, odd)
    assert t[:, 0].all() and t[:, 1].tolist() == [odd, 0, odd]


def test_host_memory_without_a_device_is_refused():
    if pkg.device_count() == 0:
        assert pkg._result_f32((70000,)).base is None     # ordinary memory


@pytest.mark.gpu
def test_a_session_on_a_used_block_gives_the_bits_of_a_fresh_one():
    arch = modelgen.tiny_arch()
    gm = pkg.Model(arch, modelgen.target_tensors(arch, seed=3))
    cfg = modelgen.tiny_dflash_config(arch)
    gd = pkg.Drafter(gm, cfg, modelgen.drafter_tensors(arch, cfg, seed=4))
    rng = np.random.default_rng(2)

    def request(ids, n_slots, capacity, block):
        sess, scr, ds = pkg.Session(gm, capacity), pkg.Scratch(gm, 16, n_slots), pkg.DSession(gd, capacity)
        taps = gd.layer_ids()[:n_slots]
        logits, rows = pkg.prefill(gm, sess, scr, taps, ids, 0, feed_drafter=ds if n_slots == 2 else None, want_hidden=True)
        out = [logits.tobytes(), rows.tobytes(), pkg.packed_verify(gm, sess, scr, taps, block, ids.size, want_logits=True)[2].tobytes()]
        if n_slots == 2:
            out.append(ds.draft_block(3, ids.size, want_logits=True)[1].tobytes())
        for x in (sess, scr, ds):
            x.close()
        return out

    ids, block, other = rng.integers(0, 1000, 40), rng.integers(0, 1000, 16), rng.integers(0, 1000, 60)
    fresh = request(ids, 2, 128, block)
    request(other, 2, 128, block)
    request(other, 1, 124, block)        # other sizes of the same classes
    assert request(ids, 2, 128, block) == fresh
    gd.close(); gm.close()


@pytest.mark.gpu
def test_a_matrix_gets_the_memory_of_idle_blocks():
    import torch
    arch = modelgen.tiny_arch()
    gm = pkg.Model(arch, modelgen.target_tensors(arch, seed=3))
    pkg.Session(gm, 4 << 20).close()                     # one attention layer: two idle blocks of 1 GiB each
    rest = torch.cuda.mem_get_info(0)[0]
    filler = torch.empty(rest - (512 << 20), dtype=torch.uint8, device="cuda:0")
    try:
        assert torch.cuda.mem_get_info(0)[0] < (600 << 20)
        _, _, _, ptr, n_bytes = pkg.synth_tensor("w", pkg.Q4_K, 4096, 524288, 7, 0.02)   # 1.2 GB
        assert n_bytes > (1 << 30)
        pkg.device_free(ptr)
    finally:
        del filler
        torch.cuda.empty_cache()
    gm.close()


@pytest.mark.gpu
def test_results_beyond_the_pinned_bound_are_ordinary_arrays():
    kept = [pkg._result_f32((16, 151936)) for _ in range(30)]       # 9.7 MB each, 256 MiB in callers' hands
    pinned = [a.base is not None for a in kept]
    assert pinned[0] and not pinned[-1] and 20 <= sum(pinned) <= 27
    for i, a in enumerate(kept):
        a[:] = i
    assert all((a == i).all() for i, a in enumerate(kept))
    assert pkg._result_f32((17 << 20,)).base is None                # above 64 MiB
    del kept
    assert pkg._result_f32((16, 151936)).base is not None           # given back with the arrays


@pytest.mark.gpu
def test_two_matrix_pipelines_that_are_dropped_give_everything_back():
    import torch
    ms = []
    for n_in, n_out in ((1024, 1024), (1024, 32000)):
        _, _, _, ptr, n_bytes = pkg.synth_tensor("w", pkg.Q4_K, n_in, n_out, 3 + n_out, 0.02)
        ms.append(pkg.QMatrix(pkg.Q4_K, n_in, n_out, pkg.device_to_host(ptr, n_bytes)))
        pkg.device_free(ptr)
    x, draft = np.random.default_rng(0).standard_normal((16, 1024)).astype(np.float32), np.zeros(16, np.int32)
    first, held = None, []
    for _ in range(40):
        am, gap, _, _ = pkg.C1Pipeline(*ms).step(x, draft)      # no close
        first = first or (am.tobytes(), gap.tobytes())
        assert (am.tobytes(), gap.tobytes()) == first
        held.append(torch.cuda.mem_get_info(0)[0])
    assert held[-1] == held[1]
    last = pkg.C1Pipeline(*ms)
    last.step(x, draft)
    for m in ms:
        m.close()
    del last                                                    # after its matrices
