"""Steps and short prompts of at most eight rows, whose norms and residual sums are folded into the products: every family, with
as many rows as there are ways to share a row out among warps, against the oracle; and one row more, which is not folded."""
import numpy as np
import pytest
import torch

import util
from rai_b200 import _lib, configs, synth
from rai_b200.models import Model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tiny-qwen2", "tiny-qwen2-tied", "tiny-qwen2-narrow", "tiny-qwen2-g7", "tiny-qwen2-28h", "tiny-phi2",
                                  "tiny-phi3", "tiny-gemma"])
@pytest.mark.parametrize("batch,seq", [(1, 1), (1, 5), (2, 1), (2, 4), (3, 1), (4, 2), (5, 1), (6, 1), (7, 1), (8, 1), (9, 1)])
def test_few_rows_match_the_oracle(cuda, name, batch, seq):
    cfg = configs.get(name)
    w = synth.weights(cfg, 11)
    oracle = util.build_oracle(cfg, w)
    m = Model(cfg, _lib.BF16, cuda, batch, 64, batch * 16)
    m.update_params(w)
    pos = 0
    # (a later portion of a prompt, but for phi2: the oracle, like the reference, masks only whole prompts)
    for i, n in enumerate((seq, 1, 1, 1, 1) if name == "tiny-phi2" else (seq, 1, 1, 16, 1)):
        ids = synth.prompt(cfg, batch, n, 100 * i + batch).astype(np.int32)
        want = oracle.forward(torch.from_numpy(ids.astype(np.int64)), pos).reshape(batch, -1)
        got = m.forward(ids, pos).reshape(batch, -1).float().cpu()
        pos += n
        for b in range(batch):
            assert util.logit_error(got[b], want[b]) <= 2e-2, (i, b)
    m.close()


@pytest.mark.parametrize("hidden,rows,few", [(1024, 8, True), (1280, 8, False), (1280, 5, False), (1280, 4, True), (2048, 4, True), (2304, 4, False),
                                             (2304, 3, False), (2304, 2, True)])
def test_rows_that_few_warps_would_normalise_are_not_folded(cuda, hidden, rows, few):
    """Five launches a layer where a lane normalises at most four pieces of a row, seven and more otherwise; and the logits of each
    sequence alone up to rounding."""
    cfg = configs.get("tiny-qwen2")
    cfg.update(hidden_size=hidden, num_attention_heads=hidden // 128, num_key_value_heads=2, intermediate_size=512, num_hidden_layers=3)
    m = Model(cfg, _lib.BF16, cuda, rows, 64, rows * 8)
    m.update_params(synth.weights(cfg, 12))
    m.forward(synth.prompt(cfg, rows, 1, 3).astype(np.int32), 0)
    ids, before = synth.prompt(cfg, rows, 1, 4).astype(np.int32), cuda.launch_count()
    together = m.forward(ids, 1).reshape(rows, -1).float().cpu()
    launches = cuda.launch_count() - before
    assert (launches <= 5 * cfg["num_hidden_layers"] + 4) == few, launches
    m.clear_kv_cache()
    first = synth.prompt(cfg, rows, 1, 3).astype(np.int32)
    for r in (0, rows - 1):
        m.clear_kv_cache()
        m.forward(first[r:r + 1], 0)
        assert util.logit_error(m.forward(ids[r:r + 1], 1).reshape(-1).float().cpu(), together[r]) <= 2e-2
    m.close()
