"""The many-row prompt pass against packed 16-row blocks of the same tokens (which the oracle tests pin): logits, captured rows,
K/V rows, recurrent and conv state, and the rollback of the prompt's last block, at the edges of its 128-token tiles, of its
512-token passes and of the packed remainder."""
import importlib

import numpy as np
import pytest

import modelgen
import orc
from dflb import pkg

syn = importlib.import_module("qwen-llm_b200.synthetic")
pytestmark = pytest.mark.gpu


def _state(arch, sess, n):
    n_attn = sum(modelgen.is_attn(arch, il) for il in range(arch.n_layer))
    kv = [np.concatenate(sess.read_kv(ai, p)) for ai in range(n_attn) for p in (0, n // 2, n - 1)]
    gdn = [np.concatenate(sess.read_gdn_state(gi)) for gi in range(arch.n_layer - n_attn)]
    return kv + gdn


def _check(arch, gm, n, start, layer_ids, kv_f16=True, capacity=None):
    rng = np.random.default_rng(n + start)
    capacity = capacity or start + n + 32
    ids = rng.integers(0, arch.vocab_size, size=start + n)
    a, b = pkg.Session(gm, capacity, kv_f16), pkg.Session(gm, capacity, kv_f16)
    sa, sb = pkg.Scratch(gm, 16, len(layer_ids)), pkg.Scratch(gm, 16, len(layer_ids))
    rows = []
    for off in range(0, start + n, 16):
        blk = ids[off:min(off + 16, start if off < start else start + n)]
        am, gap, lg = pkg.packed_verify(gm, b, sb, layer_ids, blk, off, want_logits=True)
        rows.append(sb.read_capture(blk.size))
    rows = np.concatenate(rows)[start:]
    if start:
        pkg.prefill(gm, a, sa, layer_ids, ids[:start], 0)
    logits, hidden = pkg.prefill(gm, a, sa, layer_ids, ids[start:], start, want_hidden=True)
    tol = dict(rtol=2e-3, atol=2e-4)
    np.testing.assert_allclose(logits, lg[-1], **tol)
    np.testing.assert_allclose(hidden, rows, rtol=2e-3, atol=2e-3)
    assert a.kv_n_pos == b.kv_n_pos == start + n
    for x, y in zip(_state(arch, a, start + n), _state(arch, b, start + n)):
        np.testing.assert_allclose(x, y, rtol=5e-3, atol=2e-3)
    # the last block can be undone in part, and the sequence goes on from there
    last = n % 16 or 16
    at = start + n - last
    np.testing.assert_allclose(sa.read_capture(last), rows[-last:], rtol=2e-3, atol=2e-3)
    keep = max(1, last - 3)
    for sess, scr in ((a, sa), (b, sb)):
        pkg.restore_partial(gm, sess, scr, keep, at)
    for x, y in zip(_state(arch, a, at + keep), _state(arch, b, at + keep)):
        np.testing.assert_allclose(x, y, rtol=5e-3, atol=2e-3)
    nxt = rng.integers(0, arch.vocab_size, size=5)
    la = pkg.packed_verify(gm, a, sa, layer_ids, nxt, at + keep, want_logits=True)[2]
    lb = pkg.packed_verify(gm, b, sb, layer_ids, nxt, at + keep, want_logits=True)[2]
    np.testing.assert_allclose(la, lb, **tol)
    for x in (a, b, sa, sb):
        x.close()


@pytest.fixture(scope="module")
def tiny():
    arch = modelgen.tiny_arch()
    gm = pkg.Model(arch, modelgen.target_tensors(arch, seed=3))
    yield arch, gm
    gm.close()


@pytest.mark.parametrize("n,start", [(17, 0), (32, 0), (127, 0), (128, 16), (129, 0), (512, 0), (513, 0), (529, 0), (700, 32)])
def test_prompt_pass_equals_packed_blocks(tiny, n, start):
    arch, gm = tiny
    _check(arch, gm, n, start, [0, 3, 3])


@pytest.mark.parametrize("n,kv_f16,capacity", [(77, True, None), (300, True, 16384), (300, False, None)])
def test_prompt_pass_at_dense_widths(n, kv_f16, capacity):
    arch = syn.arch_9b()
    arch.n_layer = 4
    ents = syn.target_entries(arch, seed=51, device=0)
    gm = syn.build_model(arch, ents)
    syn.free_entries(ents)
    _check(arch, gm, n, 0, [0, 1, 2, 3], kv_f16, capacity)
    gm.close()


@pytest.mark.parametrize("n,start", [(17, 0), (33, 16), (130, 0), (300, 0), (520, 0)])
def test_prompt_pass_with_routed_experts(n, start):
    arch = modelgen.tiny_arch(n_layer=4, expert_count=8, expert_used_count=3, expert_feed_forward_length=256, expert_shared_feed_forward_length=256,
                              intermediate_size=0)
    gm = pkg.Model(arch, modelgen.target_tensors(arch, seed=3))
    _check(arch, gm, n, start, [0, 3])
    gm.close()


@pytest.mark.parametrize("experts", [256, 257])
def test_prompt_routing_on_either_side_of_the_register_widths(experts):
    # a row's probabilities sit in 8 registers a lane up to 256 experts, in 32 beyond
    arch = modelgen.tiny_arch(n_layer=1, expert_count=experts, expert_used_count=5, expert_feed_forward_length=256, expert_shared_feed_forward_length=256,
                              intermediate_size=0)
    gm = pkg.Model(arch, modelgen.target_tensors(arch, seed=3))
    _check(arch, gm, 40, 0, [0])
    gm.close()


def test_prompt_pass_at_routed_widths():
    arch = syn.arch_35b_a3b()
    arch.n_layer = 4
    ents = syn.target_entries(arch, seed=53, device=0)
    gm = syn.build_model(arch, ents)
    syn.free_entries(ents)
    _check(arch, gm, 150, 0, [0, 3])
    gm.close()


@pytest.mark.parametrize("n", [18, 32, 33, 80, 81, 97, 160, 161])
def test_prompt_pass_at_tile_edges(n):
    # around the token counts at which a tile's capacity, its ring and its buffers change; several blocks and items a CTA
    arch = syn.arch_9b()
    arch.n_layer = 4
    arch.vocab_size = 8192
    ents = syn.target_entries(arch, seed=57, device=0)
    gm = syn.build_model(arch, ents)
    syn.free_entries(ents)
    _check(arch, gm, n, 0, [0, 3])
    gm.close()


@pytest.mark.parametrize("slots", [1, 3])
@pytest.mark.parametrize("n", [8, 40])
def test_feeding_a_drafter_of_another_slot_count_is_refused_before_the_first_pass(tiny, n, slots):
    arch, gm = tiny
    cfg = modelgen.tiny_dflash_config(arch)   # two tap layers
    gd = pkg.Drafter(gm, cfg, modelgen.drafter_tensors(arch, cfg, seed=4))
    sess, scr, ds = pkg.Session(gm, 64), pkg.Scratch(gm, 16, slots), pkg.DSession(gd, 64)
    with pytest.raises(pkg.DflError) as e:
        pkg.prefill(gm, sess, scr, [0, 1, 3][:slots], np.arange(n), 0, feed_drafter=ds)
    assert e.value.name == "BAD_SHAPE"
    assert sess.kv_n_pos == 0 and ds.ctx_len == 0 and not sess.poisoned
    for x in (sess, scr, ds, gd):
        x.close()


@pytest.mark.parametrize("n", [8, 40])
def test_feeding_a_drafter_of_another_model_is_refused_before_the_first_pass(tiny, n):
    arch, gm = tiny
    other = pkg.Model(arch, modelgen.target_tensors(arch, seed=9))
    cfg = modelgen.tiny_dflash_config(arch)
    gd = pkg.Drafter(other, cfg, modelgen.drafter_tensors(arch, cfg, seed=4))
    sess, scr, ds = pkg.Session(gm, 64), pkg.Scratch(gm, 16, 2), pkg.DSession(gd, 64)
    with pytest.raises(pkg.DflError) as e:
        pkg.prefill(gm, sess, scr, [1, 3], np.arange(n), 0, feed_drafter=ds)
    assert e.value.name == "BAD_ARG" and sess.kv_n_pos == 0 and ds.ctx_len == 0
    for x in (sess, scr, ds, gd, other):
        x.close()


def test_a_prompt_without_memory_for_its_workspace_takes_the_packed_path(tiny):
    import torch
    arch, gm = tiny
    rng = np.random.default_rng(5)
    ids, nxt = rng.integers(0, arch.vocab_size, 523), rng.integers(0, arch.vocab_size, 16)

    def packed(sess, scr):
        for off in range(0, ids.size, 16):
            logits, _ = pkg.prefill(gm, sess, scr, [1, 3], ids[off:off + 16], off)
        return logits

    a, b = pkg.Session(gm, 640), pkg.Session(gm, 640)
    sa, sb = pkg.Scratch(gm, 16, 2), pkg.Scratch(gm, 16, 2)
    want = packed(b, sb).copy()          # also loads every kernel that the packed path needs
    wnext = pkg.packed_verify(gm, b, sb, [1, 3], nxt, ids.size, want_logits=True)[2].copy()
    held = [torch.empty(torch.cuda.mem_get_info(0)[0] - (1 << 30), dtype=torch.uint8, device="cuda:0")]
    ptrs = []
    try:
        for kib in (1 << 18, 1 << 14, 1 << 11):          # 256, 16, 2 MiB until there is none left
            try:
                while True:
                    ptrs.append(pkg.synth_tensor("w", pkg.F32, 256, kib, 7, 0.02)[3])
            except pkg.DflError as e:
                assert e.name == "OOM"
        got, _ = pkg.prefill(gm, a, sa, [1, 3], ids, 0)
        gnext = pkg.packed_verify(gm, a, sa, [1, 3], nxt, ids.size, want_logits=True)[2].copy()
    finally:
        for p in ptrs:
            pkg.device_free(p)
        del held
        torch.cuda.empty_cache()
    assert a.kv_n_pos == ids.size + 16 and not a.poisoned
    assert got.tobytes() == want.tobytes() and gnext.tobytes() == wnext.tobytes()     # the packed path's own bits
    for x in (a, b, sa, sb):
        x.close()


@pytest.mark.parametrize("n", [8, 40, 520])
def test_capture_slots_without_a_layer_stay_untouched(tiny, n):
    arch, gm = tiny
    ids = np.random.default_rng(6).integers(0, arch.vocab_size, n)

    def run(layer_ids):
        sess, scr = pkg.Session(gm, 640), pkg.Scratch(gm, 16, 2)
        rows = pkg.prefill(gm, sess, scr, layer_ids, ids, 0, want_hidden=True)[1].copy()
        block = scr.read_capture(n % 16 or 16).copy()
        sess.close(); scr.close()
        return rows, block

    both = run([1, 3])              # fills both slots; its memory goes to the next scratch
    one = run([3])
    assert np.array_equal(one[0][:, 0], both[0][:, 1]) and not one[0][:, 1].any()
    assert np.array_equal(one[1][:, 0], both[1][:, 1]) and not one[1][:, 1].any()


# Four layers of the packed pass lie 4.5e-6 (9B widths) and 3.6e-6 (routed) of the float64 forward in the 2-norm of the captured rows, the
# many-row pass 4.3e-6 to 4.5e-6 and 3.4e-6.  Most of it is what the tensor-core sums drop, alike in both, so that the two differ by
# 2.5e-6 and 2.2e-6 only.  Sums of all a block's steps in one accumulator (1.56e-5 and 1.0e-5 of float64) or a lost lo plane (1e-4)
# lie above the bounds.  The cache is f32: one fp16 rounding that falls the other way outweighs all of it.
@pytest.mark.parametrize("routed,n,bound", [(False, 77, 4e-6), (False, 300, 4e-6), (True, 150, 3.5e-6)])
def test_prompt_pass_is_as_close_as_the_packed_one(routed, n, bound):
    arch = syn.arch_35b_a3b() if routed else syn.arch_9b()
    arch.n_layer, arch.vocab_size = 4, 8192
    ents = syn.target_entries(arch, seed=51, device=0)
    gm = syn.build_model(arch, ents)
    syn.free_entries(ents)
    ids = np.random.default_rng(n).integers(0, arch.vocab_size, n)
    taps = [0, 1, 2, 3]
    a, b = pkg.Session(gm, 512, False), pkg.Session(gm, 512, False)
    sa, sb = pkg.Scratch(gm, 16, 4), pkg.Scratch(gm, 16, 4)
    rows = []
    for off in range(0, n, 16):
        pkg.packed_verify(gm, b, sb, taps, ids[off:off + 16], off)
        rows.append(sb.read_capture(len(ids[off:off + 16])))
    got = pkg.prefill(gm, a, sa, taps, ids, 0, want_hidden=True)[1]

    def rel(x, y):
        return np.linalg.norm(x.astype(np.float64) - y) / np.linalg.norm(y.astype(np.float64))

    off = {"rows": rel(got, np.concatenate(rows))}
    off["kv"] = rel(np.stack([np.concatenate(a.read_kv(0, p)) for p in range(n)]), np.stack([np.concatenate(b.read_kv(0, p)) for p in range(n)]))
    off["state"] = rel(np.stack([np.concatenate(a.read_gdn_state(g)) for g in range(3)]), np.stack([np.concatenate(b.read_gdn_state(g)) for g in range(3)]))
    assert max(off.values()) < bound, off
    for x in (a, b, sa, sb, gm):
        x.close()


# The attention of a prompt pass keeps to the packed pass's spans (tiled cache) or merges chunk by chunk (row-major cache at the
# capacities where a packed span is one chunk), so over the same keys and values the two differ by what their queries do, some 1e-6, and
# by the f16 roundings (weights, the new rows' own keys and values) that this moves: 1.1e-5 to 1.5e-5 of the attention's output on average.
# One sum over the whole context differed by 1.4e-4 to 2e-4: weights rounded against another maximum, and an output short by what
# every further tensor-core step drops.
@pytest.mark.parametrize("n,capacity", [(900, 4096), (3000, 4096), (1500, 16384), (3000, 16384)])
def test_prompt_attention_is_the_packed_pass_s(n, capacity):
    arch = syn.arch_9b()
    arch.n_layer, arch.full_attention_interval, arch.vocab_size, arch.intermediate_size = 1, 1, 8192, 512
    ents = syn.target_entries(arch, seed=71, device=0)
    ents = [(nm, d, s, np.zeros(nb, np.uint8) if "ffn_down" in nm else data, nb) for nm, d, s, data, nb in ents]   # a layer of attention alone
    embd = next(e for e in ents if e[0] == "token_embd.weight")
    embd = orc.dequant(embd[1], pkg.device_to_host(embd[3], embd[4]), arch.hidden_size * arch.vocab_size).reshape(arch.vocab_size, -1)
    gm = syn.build_model(arch, ents)
    syn.free_entries([e for e in ents if isinstance(e[3], int)])
    ids = np.random.default_rng(n).integers(0, arch.vocab_size, n + 32)
    a, b = pkg.Session(gm, capacity, True), pkg.Session(gm, capacity, True)
    sa, sb = pkg.Scratch(gm, 16, 1), pkg.Scratch(gm, 16, 1)
    pkg.prefill(gm, a, sa, [0], ids[:n], 0)
    pkg.session_restore_snapshot(gm, b, None, pkg.session_snapshot(gm, a, None))
    got = pkg.prefill(gm, a, sa, [0], ids[n:], n, want_hidden=True)[1][:, 0]
    rows = []
    for off in (n, n + 16):
        pkg.packed_verify(gm, b, sb, [0], ids[off:off + 16], off)
        rows.append(sb.read_capture(16)[:, 0])
    rows = np.concatenate(rows).astype(np.float64)
    off = np.linalg.norm(got - rows, axis=1) / np.linalg.norm(rows - embd[ids[n:]], axis=1)
    assert off.mean() < 4e-5 and off.max() < 1e-4, off
    for x in (a, b, sa, sb, gm):
        x.close()


@pytest.mark.parametrize("n", [513, 540, 600])
def test_prompt_of_several_passes_at_routed_widths(n):
    # one pass of 512 rows (every expert chosen, segments of all sizes), then a packed remainder or a second pass
    arch = syn.arch_35b_a3b()
    arch.n_layer, arch.vocab_size = 2, 8192
    arch.full_attention_interval = 2
    ents = syn.target_entries(arch, seed=53, device=0)
    gm = syn.build_model(arch, ents)
    syn.free_entries(ents)
    _check(arch, gm, n, 0, [0, 1])
    gm.close()


def test_the_scalar_attention_switch_holds_for_prompts(monkeypatch):
    arch = modelgen.tiny_arch(n_q_heads=4)          # a group of four: the tensor-core kernel by default
    gm = pkg.Model(arch, modelgen.target_tensors(arch, seed=3))
    ids = np.random.default_rng(8).integers(0, arch.vocab_size, 100)
    out = []
    for value in (None, "0"):
        if value is not None:
            monkeypatch.setenv("DFL_ATTN_TC", value)
        sess, scr = pkg.Session(gm, 128), pkg.Scratch(gm, 16, 1)
        out.append(pkg.prefill(gm, sess, scr, [3], ids, 0, want_hidden=True)[1].copy())
        sess.close(); scr.close()
    assert out[0].tobytes() != out[1].tobytes()
    np.testing.assert_allclose(out[0], out[1], rtol=2e-3, atol=2e-3)
    gm.close()
