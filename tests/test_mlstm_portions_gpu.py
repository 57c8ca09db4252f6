"""Portions of 48 - 127 tokens of the matrix memory in bf16 mode run chunk-parallel on pairs of bf16 values (recur_chunk.cu): lengths at
the rule's line and at the chunks' edges, batches, a second portion from the state the first one left, and single tokens behind it."""
import numpy as np
import pytest

import test_vupitar_gpu as vup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 256), (192, 128)])
@pytest.mark.parametrize("n,batch", [(47, 1), (48, 2), (64, 1), (65, 3), (127, 1)])
def test_portions(n, batch, dim, vdim):
    cfg = vup.config([vup.layer(r=vup.right(heads=2, dim=dim, vdim=vdim)), vup.layer(r=vup.right(heads=2, dim=dim, vdim=vdim), mlp=None)], width=128)
    total = 2 * n + 3
    m, o = vup.build(cfg, seed=n, dtype="bfloat16", max_seq_len=total + 1, max_batch_size=batch)
    ids = np.random.default_rng(n).integers(0, cfg["vocab"], (batch, total))
    got = [m.forward_rows(ids[:, s:e], s, list(range(batch * (e - s)))).reshape(batch, e - s, -1)
           for s, e in ((0, n), (n, 2 * n), (2 * n, 2 * n + 1), (2 * n + 1, 2 * n + 2), (2 * n + 2, total))]
    for b in range(batch):
        assert vup.err(np.concatenate([g[b] for g in got]), vup.fresh(o).run(ids[b])) < vup.BF16_BAR
    m.close()


@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 256)])
@pytest.mark.parametrize("n,bad", [(48, 30), (64, 40), (90, 60), (127, 100), (127, 60)])
def test_a_token_that_is_not_a_number_stays_behind_its_predecessors(n, bad, dim, vdim):
    """One token's embedding is NaN: the tokens ahead of it (all but the window layer's own neighbourhood of 12) keep their logits."""
    cfg = vup.config([vup.layer(r=vup.right(heads=2, dim=dim, vdim=vdim))], width=128)
    t = {k: np.array(v, np.float32) for k, v in vup.random_model(cfg, 3).items()}
    clean = dict(t)
    t["embed"] = t["embed"].copy()
    t["embed"][5] = np.nan
    m, _ = vup.build(cfg, dtype="bfloat16", max_seq_len=n + 2, tensors=t)
    o = vup.Oracle(cfg, clean)
    ids = np.random.default_rng(n).integers(6, cfg["vocab"], n)
    ids[bad] = 5
    got = m.forward_rows(ids[None], 0, list(range(n)))
    assert np.isnan(got[bad:]).any(1).all()
    assert vup.err(got[:bad - 12], o.run(ids[:bad - 12])) < vup.BF16_BAR
    m.close()
