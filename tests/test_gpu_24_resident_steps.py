"""Single-token steps of up to eight sequences that run as one kernel (layers of more than 96 MB): every family and head size it takes, sizes
that no share of 148 divides, contexts around the edges of key tiles, pairs cut into pieces, sequences of different lengths - against
the oracle, with the tolerance of the other model tests; the replayed step against plain ones; and who takes the kernel."""
import ctypes

import numpy as np
import pytest
import torch

import util
from rai_b200 import _lib, configs, synth
from rai_b200.models import Model

pytestmark = pytest.mark.gpu

FAMILIES = {
    # heads of 64, one for keys and values, group 31 > 16 is not taken: 30 heads in two groups of 15; rows of 1920 = 148 * 13 - 4
    "qwen2-64": ("tiny-qwen2", dict(hidden_size=1920, num_attention_heads=30, num_key_value_heads=2, intermediate_size=8896)),
    "qwen2-128": ("tiny-qwen2", dict(hidden_size=1792, num_attention_heads=14, num_key_value_heads=2, intermediate_size=9536)),
    "qwen2-128-tied": ("tiny-qwen2-tied", dict(hidden_size=2560, num_attention_heads=20, num_key_value_heads=20, intermediate_size=6464)),
    "phi2-80": ("tiny-phi2", dict(hidden_size=2560, num_attention_heads=32, num_key_value_heads=32, intermediate_size=10304)),
    "phi3-96": ("tiny-phi3", dict(hidden_size=2304, num_attention_heads=24, num_key_value_heads=24, intermediate_size=7488)),
    "gemma-128": ("tiny-gemma", dict(hidden_size=2048, num_attention_heads=16, num_key_value_heads=1, head_dim=128, intermediate_size=8256)),
}


def _config(family, layers=2):
    name, sizes = FAMILIES[family]
    cfg = configs.get(name)
    cfg.update(sizes, num_hidden_layers=layers, vocab_size=1031, max_position_embeddings=1024)
    return cfg


@pytest.mark.parametrize("family", list(FAMILIES))
@pytest.mark.parametrize("lens", [[1], [63], [700], [64, 65], [2, 63, 200], [128] * 4, [5, 129, 64, 300, 1, 191, 66], [40] * 8])
def test_steps_match_the_oracle(cuda, family, lens):
    cfg = _config(family)
    w = synth.weights(cfg, 21)
    oracle = util.build_oracle(cfg, w)
    b, steps = len(lens), 3
    m = Model(cfg, _lib.BF16, cuda, b, 768, sum(lens) + 8 * b * max(lens))
    m.update_params(w)
    fed = synth.prompt(cfg, b, max(lens) + steps, 22).astype(np.int32)
    prompts = np.zeros((b, max(lens)), np.int32)
    for i, n in enumerate(lens):
        prompts[i, :n] = fed[i, :n]
    m.forward_ragged(prompts, lens)
    got = []
    for t in range(steps):
        ids = np.stack([fed[i, n + t:n + t + 1] for i, n in enumerate(lens)])
        before = cuda.launch_count()
        if len(set(lens)) == 1:
            got.append(m.forward(ids, lens[0] + t).reshape(b, -1).float().cpu())
        else:
            got.append(m.forward_rows(ids, None, range(b)).reshape(b, -1).float().cpu())
        assert cuda.launch_count() - before <= 6   # (a layer of kernels of its own would be seven)
    for i, n in enumerate(lens):
        oracle.clear_kv_cache()
        oracle.forward(torch.from_numpy(fed[i:i + 1, :n].astype(np.int64)), 0)
        for t in range(steps):
            want = oracle.forward(torch.from_numpy(fed[i:i + 1, n + t:n + t + 1].astype(np.int64)), n + t).reshape(-1)
            assert util.logit_error(got[t][i], want) <= 2e-2, (i, t)
    m.close()


@pytest.mark.parametrize("family", ["qwen2-128", "phi2-80"])
def test_replayed_steps_are_the_plain_ones_and_the_next_context_crosses_a_tile(cuda, family):
    """Eight replays of the captured step (from 60 keys over the edge of the tile) give the tokens and, in one more step, the bits of plain calls."""
    cfg = _config(family)
    b, n, steps = 3, 60, 8
    m = Model(cfg, _lib.BF16, cuda, b, 128, b * n)
    m.update_params(synth.weights(cfg, 23))
    ids = synth.prompt(cfg, b, n, 24).astype(np.int32)

    def best(logits):   # of equal logits (8 bits tell few of a thousand apart) the last, which is what the device's sampling takes
        logits = logits.reshape(b, -1).float().cpu()
        return np.array([[int((row == row.max()).nonzero()[-1])] for row in logits], np.int32)

    plain = [best(m.forward(ids, 0))]
    for t in range(steps):
        plain.append(best(m.forward(plain[-1], n + t)))
    last = m.forward(plain[-1], n + steps).float().cpu()
    m.clear_kv_cache()
    loop = m.decode_loop(torch.from_numpy(best(m.forward(ids, 0)).reshape(-1)).cuda(), n, steps).cpu().numpy()
    assert (loop == np.stack([p.reshape(-1) for p in plain[1:]])).all()
    again = m.forward(loop[-1].reshape(b, 1), n + steps).float().cpu()
    assert torch.equal(last, again)
    m.close()


@pytest.mark.parametrize("batch,context,one", [(8, 64, True), (9, 64, False), (8, 1450, True), (8, 1550, False)])
def test_who_takes_the_kernel(cuda, batch, context, one):
    """Up to eight sequences, and up to three quarters of a layer's weights (146 MB) in cached bytes (9.2 KB a token)."""
    cfg = _config("phi3-96")
    cfg["max_position_embeddings"] = 2048
    m = Model(cfg, _lib.BF16, cuda, batch, 1600, batch)
    m.update_params(synth.weights(cfg, 25))
    _lib.call("rb_kv_cache_set_len", _lib.lib().rb_model_kv_cache(m._m), batch, context)
    before = cuda.launch_count()
    m.forward(np.ones((batch, 1), np.int32), context)
    assert (cuda.launch_count() - before <= 6) == one
    m.close()


@pytest.mark.parametrize("family", ["qwen2-128", "phi2-80"])
def test_a_step_that_gives_up_says_so_and_the_next_ones_are_right(cuda, family):
    """Barriers that never open: every role stops waiting after the budget, the block stays until its copies have landed, the host learns of
    it, and the same step afterwards gives the same bits as ever."""
    cfg = _config(family)
    b, n = 3, 200
    m = Model(cfg, _lib.BF16, cuda, b, 256, b * n)
    m.update_params(synth.weights(cfg, 27))
    ids, token = synth.prompt(cfg, b, n, 28).astype(np.int32), np.array([[1], [2], [3]], np.int32)

    def prompt_and_step():
        m.clear_kv_cache()
        m.forward(ids, 0)
        return lambda: m.forward(token, n).float().cpu()

    want = prompt_and_step()()
    step = prompt_and_step()
    _lib.call("rb_set_wait_budget_us", cuda.ctx, 500)
    try:
        _lib.call("rb_selftest_spoil_step", m._m)
        with pytest.raises(_lib.RaiB200Error, match="0x57e9"):
            step()
    finally:
        _lib.call("rb_set_wait_budget_us", cuda.ctx, 1000000)
    assert torch.equal(prompt_and_step()(), want)
    m.close()


@pytest.mark.parametrize("captured", [False, True])
def test_a_refused_launch_falls_back_to_the_kernels_of_other_steps(cuda, captured):
    """All blocks or none: where the launch is refused, the step runs as launches of its own, and so do all later ones."""
    cfg = _config("phi3-96")
    b, n, steps = 2, 70, 5
    w = synth.weights(cfg, 31)
    m = Model(cfg, _lib.BF16, cuda, b, 128, b * n)
    m.update_params(w)
    ids = synth.prompt(cfg, b, n, 32).astype(np.int32)
    fed = synth.prompt(cfg, b, steps, 33).astype(np.int32)
    m.forward(ids, 0)
    if captured:   # (the captured step of before is not replayed)
        m.decode_loop(torch.from_numpy(fed[:, 0].copy()).cuda(), n, 4)
        m.clear_kv_cache()
        m.forward(ids, 0)
    _lib.call("rb_selftest_refuse_step", m._m)
    oracle = util.build_oracle(cfg, w)
    oracle.forward(torch.from_numpy(ids.astype(np.int64)), 0)
    for t in range(steps):
        before = cuda.launch_count()
        got = m.forward(fed[:, t:t + 1], n + t).reshape(b, -1).float().cpu()
        assert cuda.launch_count() - before > 6
        want = oracle.forward(torch.from_numpy(fed[:, t:t + 1].astype(np.int64)), n + t).reshape(b, -1)
        assert util.logit_error(got, want) <= 2e-2, t
    again = m.decode_loop(torch.from_numpy(fed[:, 0].copy()).cuda(), n + steps, 6)
    m.device.synchronize()
    assert again.shape == (6, b)
    with pytest.raises(_lib.RaiB200Error):
        _lib.call("rb_selftest_refuse_step", m._m)   # the plan is gone
    m.close()


@pytest.mark.parametrize("family", ["qwen2-128", "phi3-96"])
def test_rows_whose_squares_sum_past_float32(cuda, family):
    """RMSNorm divides by the root of the width before it squares (rai-nn/src/rms_norm.rs:18-22): a root mean square of 2^60 is in range, the
    sum of its squares is not.  What layers add to such a stream is nothing, so the logits are those of the embedding's norm."""
    cfg = _config(family)
    w = synth.weights(cfg, 35)
    embed = np.asarray(w["model.embed_tokens.weight"], np.float64)
    w["model.embed_tokens.weight"] = (embed * 2.0 ** 60 / np.sqrt((embed ** 2).mean())).astype(np.float32)
    m = Model(cfg, _lib.BF16, cuda, 3, 64, 3)
    m.update_params(w)
    ids = np.array([[5], [77], [1030]], np.int32)
    got = m.forward(ids, 0).reshape(3, -1).float().cpu()
    rows = torch.from_numpy(embed[ids[:, 0]])
    rows = rows / (rows ** 2).mean(-1, keepdim=True).sqrt() * torch.from_numpy(np.asarray(w["model.norm.weight"], np.float64))
    want = rows @ torch.from_numpy(np.asarray(w["lm_head.weight"], np.float64)).T
    for i in range(3):
        assert util.logit_error(got[i], want[i]) <= 2e-2, i
    m.close()


@pytest.mark.parametrize("family", ["phi3-96", "phi2-80"])
def test_a_profile_of_a_step_tells_its_classes_apart(cuda, family):
    """A launch belongs to one class of the per-launch profile, so a step under it runs as launches of its own; the next one does not."""
    cfg = _config(family)
    b, n = 2, 70
    m = Model(cfg, _lib.BF16, cuda, b, 128, b * n)
    m.update_params(synth.weights(cfg, 37))
    m.forward(synth.prompt(cfg, b, n, 38).astype(np.int32), 0)
    token = np.ones((b, 1), np.int32)
    _lib.call("rb_profile_start", cuda.ctx)
    m.forward(token, n)
    out, seen = (ctypes.c_double * 4)(), {}
    for i, name in enumerate(("gemm", "attention", "norm")):
        _lib.call("rb_profile_read", cuda.ctx, i, out)
        seen[name] = list(out)
    layers, kv = cfg["num_hidden_layers"], cfg["num_key_value_heads"]
    keys_values = 2 * 2 * b * (n + 1) * kv * configs.head_dim(cfg)
    assert seen["attention"][0] == layers and seen["attention"][2] >= layers * keys_values, seen
    assert seen["norm"][0] > layers and seen["gemm"][0] > 3 * layers, seen
    before = cuda.launch_count()
    m.forward(token, n + 1)
    assert cuda.launch_count() - before <= 6
    m.close()


@pytest.mark.parametrize("family", ["qwen2-128", "phi2-80"])
def test_a_step_that_gives_up_leaves_the_cache_alone(cuda, family):
    """No barrier opens, so no block has a key or value to append: the rows behind the cached ones stay as they are, zero in a new cache.  (Rows that are
    not numbers there would reach later sequences of the same pages, whose masked probabilities are zero times them.)"""
    cfg = _config(family)
    b, n = 3, 200
    m = Model(cfg, _lib.BF16, cuda, b, 256, b * n)
    m.update_params(synth.weights(cfg, 43))
    m.forward(synth.prompt(cfg, b, n, 44).astype(np.int32), 0)
    _lib.call("rb_set_wait_budget_us", cuda.ctx, 500)
    try:
        _lib.call("rb_selftest_spoil_step", m._m)
        with pytest.raises(_lib.RaiB200Error, match="0x57e9"):
            m.forward(np.array([[1], [2], [3]], np.int32), n)
    finally:
        _lib.call("rb_set_wait_budget_us", cuda.ctx, 1000000)
    for layer in range(cfg["num_hidden_layers"]):
        for seq in range(b):
            for head in range(cfg["num_key_value_heads"]):
                assert not any((x != 0).any() for x in m.kv_read(layer, seq, head, n, 1)), (layer, seq, head)
    m.close()


@pytest.mark.parametrize("batch,one", [(6, True), (7, False)])
def test_pairs_that_leave_blocks_idle_stay_on_launches(cuda, batch, one):
    """24 heads: 6 sequences are 144 pairs for 148 blocks, 7 are 168 (84 blocks would walk two pairs each, as long as 84 blocks alone can)."""
    cfg = _config("phi3-96")
    cfg["max_position_embeddings"] = 2048
    m = Model(cfg, _lib.BF16, cuda, batch, 1664, batch)
    m.update_params(synth.weights(cfg, 45))
    _lib.call("rb_kv_cache_set_len", _lib.lib().rb_model_kv_cache(m._m), batch, 1590)
    before = cuda.launch_count()
    m.forward(np.ones((batch, 1), np.int32), 1590)
    assert (cuda.launch_count() - before <= 6) == one
    m.close()


@pytest.mark.parametrize("family", ["qwen2-128", "phi2-80"])
@pytest.mark.parametrize("batch", [1, 8])
def test_a_vocabulary_that_takes_several_passes(cuda, family, batch):
    """40007 rows are three passes of 91 for each of 148 blocks: the last block has none, the one before it two."""
    cfg = _config(family)
    cfg["vocab_size"] = 40007
    w = synth.weights(cfg, 41)
    n = 65
    m = Model(cfg, _lib.BF16, cuda, batch, 128, batch * n)
    m.update_params(w)
    ids = synth.prompt(cfg, batch, n + 1, 42).astype(np.int32)
    m.forward(ids[:, :n], 0)
    before = cuda.launch_count()
    got = m.forward(ids[:, n:], n).reshape(batch, -1).float().cpu()
    assert cuda.launch_count() - before <= 6
    oracle = util.build_oracle(cfg, w)
    oracle.forward(torch.from_numpy(ids[:, :n].astype(np.int64)), 0)
    want = oracle.forward(torch.from_numpy(ids[:, n:].astype(np.int64)), n).reshape(batch, -1)
    for i in range(batch):
        assert util.logit_error(got[i], want[i]) <= 2e-2, i
    m.close()
