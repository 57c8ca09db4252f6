"""Gated experts of many rows in groups, every expert over the rows that chose it (moe.cu, the grouped products of gemm_tc.cu): planted
routing that gives experts 0, 1, 127, 128, 129 and many rows, 1 - 3 chosen experts, with and without a shared one, weights on the input
(sigmoid scores) and on the output (softmax scores, gated shared expert).  Held to the float64 oracle at the families' bf16 bar, and
to the same model's portions of at most 128 tokens, which take the masked product over all experts: a lost, misplaced or
doubly counted pair is an error of the size of its row."""
import numpy as np
import pytest

import test_mabedra_gpu as mab
import test_vupitar_gpu as vup

pytestmark = pytest.mark.gpu
E, W, FF, V = 64, 1024, 256, 70


def _ids(n, seed):
    """tokens 0 - 4 so often that their first experts reach the edges of a 128-row tile, the rest spread; 60 and more never occur"""
    ids = [0] * 127 + [1] * 128 + [2] * 129 + [3] if n > 400 else [0] * 127 + [3]
    rng = np.random.default_rng(seed)
    return rng.permutation(np.concatenate([ids, rng.integers(8, 50, n - len(ids))]))


def _whole_and_portions(m, ids, cut):
    whole = m.forward_rows(ids[None], 0, list(range(len(ids))))
    parts = [m.forward_rows(ids[None, s:s + cut], s, list(range(len(ids[s:s + cut])))) for s in range(0, len(ids), cut)]
    return whole, np.concatenate(parts)


@pytest.mark.parametrize("n,top,shared", [(257, 1, 0), (600, 1, 264), (600, 2, 0), (431, 3, 128)])
def test_planted_routing(n, top, shared):
    cfg = mab.config([mab.attn(heads=2, kv_heads=1, dim=64, vdim=64, mlp=mab.moe(E, top, FF, shared))], width=W, vocab=V, taps=0)
    t = mab.random_model(cfg, 11)
    rng = np.random.default_rng(12)
    a = rng.standard_normal((E, W))
    a = np.linalg.qr(a.T)[0].T * np.sqrt(W)
    t["embed"] = sum((1.0 - 0.2 * k) * a[(np.arange(V) + k) % E] for k in range(top))  # a token's experts: itself and the next ones
    t["l0.mlp.router"] = a * (2.0 / W)
    t["l0.norm1"], t["l0.mix.o"] = np.ones(W), 0 * t["l0.mix.o"]
    t = {k: np.asarray(v, np.float32) for k, v in t.items()}
    t = {k: (v.view(np.uint32) + 0x8000 & 0xFFFF0000).astype(np.uint32).view(np.float32) for k, v in t.items()}  # values a bf16 holds
    m, o = mab.build(cfg, dtype="bfloat16", max_seq_len=n + 2, tensors=t)
    ids = _ids(n, n)
    whole, parts = _whole_and_portions(m, ids, 128)
    want = o.run(ids)
    assert mab.err(whole, want) < mab.BF16_BAR
    assert mab.err(whole, parts) < mab.BF16_BAR
    m.close()


@pytest.mark.parametrize("n,batch,shared", [(300, 1, 256), (150, 2, 0)])
def test_output_weights_and_gated_shared_expert(n, batch, shared):
    mlp = {"kind": "moe", "router": {"experts": E, "top": 2}, "expert": {"ff": FF}}
    if shared:
        mlp["shared"] = {"ff": shared}
    cfg = vup.config([vup.layer(l=vup.left(heads=2, kv_heads=1, dim=64, vdim=64, size=80), r=vup.right(heads=2, dim=64, vdim=64), mlp=mlp)], width=W, vocab=V)
    m, o = vup.build(cfg, seed=7, dtype="bfloat16", max_seq_len=n + 2, max_batch_size=batch)
    ids = np.random.default_rng(n).integers(0, V, (batch, n))
    whole = m.forward_rows(ids, 0, list(range(batch * n))).reshape(batch, n, -1)
    for b in range(batch):
        e = vup.row_errs(whole[b], vup.fresh(o).run(ids[b]))  # a rounded router input may turn a close choice
        assert np.quantile(e, 0.9) < vup.BF16_BAR and np.median(e) < vup.BF16_BAR / 3
    m.close()
