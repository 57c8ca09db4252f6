"""Gated experts of many rows in groups (moe.cu, layerlist.cu: ll_moe_groups), with the path asserted by its number of launches: order,
gather, two products and the sum - and two more products for a shared expert - where the masked form has two products and a pass over
the hidden values."""
import numpy as np
import pytest

import test_mabedra_gpu as mab

pytestmark = pytest.mark.gpu
E, W, FF, V = 64, 1024, 256, 70


def bf16_values(t):
    t = {k: np.asarray(v, np.float32) for k, v in t.items()}
    return {k: (v.view(np.uint32) + 0x8000 & 0xFFFF0000).astype(np.uint32).view(np.float32) for k, v in t.items()}


def run(m, ids):
    """all logits of one call, and its launches beyond those of a call of 128 rows, which takes the masked form"""
    b, n = ids.shape
    m.launch_count(reset=True)
    m.forward_rows(ids[:, :128 // b], 0, [0])
    few = m.launch_count(reset=True)
    got = m.forward_rows(ids, 0, list(range(b * n))).reshape(b, n, -1)
    return got, m.launch_count() - few


def sign_rows(rng):
    """embedding rows of +-1 that sum to zero, +1 at coordinate 0: a layer norm leaves them as they are"""
    e = np.empty((V, W), np.float32)
    for r in e:
        r[:] = 1
        r[rng.permutation(np.arange(1, W))[:W // 2]] = -1
    return e


@pytest.mark.parametrize("n", [300, 431])
def test_silu_of_a_shared_expert_keeps_its_tail(n):
    """As in the masked form: silu(-88) = -5e-37 and an up value of 2^120 decide the output."""
    cfg = mab.config([mab.attn(heads=2, kv_heads=1, dim=64, vdim=64, mlp=mab.moe(E, 1, FF, 264))], width=W, vocab=V, taps=0)
    rng = np.random.default_rng(n)
    t = mab.random_model(cfg, 3)
    t["embed"] = sign_rows(rng)
    t["l0.norm1"], t["l0.mix.o"], t["l0.ls2"] = np.ones(W), 0 * t["l0.mix.o"], np.ones(W)
    g, u, d = (t["l0.mlp.shared." + k] for k in ("gate", "up", "down"))
    g[0], u[0], d[:, 0] = 0, 0, 0
    g[0, 0], u[0, 0], d[1, 0] = -88, 2.0 ** 120, 64
    t = bf16_values(t)
    m, o = mab.build(cfg, dtype="bfloat16", max_seq_len=2048, tensors=t)
    ids = rng.integers(0, V, (1, n))
    got, more = run(m, ids)
    m.close()
    assert more == 4
    assert mab.err(got[0], o.run(ids[0])) < mab.BF16_BAR
