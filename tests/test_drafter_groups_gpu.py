"""Drafter context projected in groups of sixteen columns gives the bits of column-by-sixteen projection."""
import importlib

import numpy as np
import pytest

pkg = importlib.import_module("qwen-llm_b200")
syn = importlib.import_module("qwen-llm_b200.synthetic")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16, 17, 32, 33, 64, 65, 80, 200])
def test_grouped_context_projection_is_bitwise_the_sixteen_column_one(n):
    arch = syn.arch_9b()
    arch.n_layer, arch.vocab_size = 4, 4096
    ents = syn.target_entries(arch, seed=61, device=0)
    gm = syn.build_model(arch, ents)
    syn.free_entries(ents)
    cfg = syn.dflash_config_9b(arch)
    cfg.n_layer = 2
    dents = syn.drafter_entries(arch, cfg, device=0)
    gd = syn.build_drafter(gm, cfg, dents)
    syn.free_entries(dents)
    cols = np.random.default_rng(n).standard_normal((n, cfg.n_target_layers * arch.hidden_size)).astype(np.float32)
    at_once, by_sixteen = pkg.DSession(gd, 512), pkg.DSession(gd, 512)
    at_once.append_columns(cols, np.arange(n))
    want = None
    for c0 in range(0, n, 16):
        m = min(16, n - c0)
        by_sixteen.append_columns(cols[c0:c0 + m], np.arange(c0, c0 + m))
        _, want = by_sixteen.draft_block(7, c0 + m, want_logits=True)   # projects what is pending
    _, got = at_once.draft_block(7, n, want_logits=True)
    assert got.tobytes() == want.tobytes()
    for x in (at_once, by_sixteen, gd, gm):
        x.close()
