"""Gated experts of many rows in groups (moe.cu, layerlist.cu: ll_moe_groups), with the path asserted by its number of launches: order,
gather, two products and the sum - and two more products for a shared expert - where the masked form has two products and a pass over
the hidden values."""
import os
import subprocess
import sys

import numpy as np
import pytest

import test_mabedra_gpu as mab
import test_vupitar_gpu as vup

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


def planted_rows(top, rng):
    """64 directions at right angles; a token's embedding leans on its own and, less and less, on the next ones: its experts"""
    a = np.linalg.qr(rng.standard_normal((W, E)))[0].T * np.sqrt(W)
    return a, sum((1.0 - 0.2 * k) * a[(np.arange(V) + k) % E] for k in range(top))


def planted_ids(n, rng):
    """experts of 127, 128 and 129 first choices, one of one, the rest spread, some never chosen"""
    ids = [0] * 127 + [4] * 128 + [8] * 129 + [12] if n > 400 else [0] * 127 + [12]
    return rng.permutation(np.concatenate([ids, rng.integers(16, 50, n - len(ids))]))


def sigmoid_model(top, shared):
    cfg = mab.config([mab.attn(heads=2, kv_heads=1, dim=64, vdim=64, mlp=mab.moe(E, top, FF, shared))], width=W, vocab=V, taps=0)
    t = mab.random_model(cfg, 11)
    a, t["embed"] = planted_rows(top, np.random.default_rng(12))
    t["l0.mlp.router"] = a * (2.0 / W)
    t["l0.norm1"], t["l0.mix.o"] = np.ones(W), 0 * t["l0.mix.o"]
    return cfg, bf16_values(t)


@pytest.mark.parametrize("n,top,shared", [(257, 1, 0), (431, 3, 128), (600, 2, 264)])
@pytest.mark.parametrize("room", ["tight", "wide", "none"])
def test_the_form_does_not_hang_on_the_models_length(n, top, shared, room, monkeypatch):
    """A model made for just the prompt, one made for much longer ones, and - the masked form, where it needs one - without a workspace."""
    if room == "none":
        monkeypatch.setenv("L3_SCRATCH_MB", "0")
    cfg, t = sigmoid_model(top, shared)
    m, o = mab.build(cfg, dtype="bfloat16", max_seq_len=2048 if room == "wide" else n + 2, tensors=t)
    ids = planted_ids(n, np.random.default_rng(n))
    got, more = run(m, ids[None])
    m.close()
    if room != "none":
        assert more == (4 if shared else 2)
    elif n == 257:
        assert more == 0
    assert mab.err(got[0], o.run(ids)) < mab.BF16_BAR


@pytest.mark.parametrize("n,batch,top,shared", [(300, 1, 2, 256), (600, 1, 1, 64), (431, 1, 3, 128), (150, 2, 2, 0), (200, 3, 2, 264)])
def test_weights_on_outputs_and_a_gated_shared_expert(n, batch, top, shared):
    """Softmax scores over their sum on the experts' outputs, a sigmoid's on the shared one's, all added to the residual stream in
    place; planted routing, so that every row is held to the bar."""
    mlp = {"kind": "moe", "router": {"experts": E, "top": top}, "expert": {"ff": FF}}
    if shared:
        mlp["shared"] = {"ff": shared}
    cfg = vup.config([vup.layer(l=vup.left(heads=2, kv_heads=1, dim=64, vdim=64, size=80), r=vup.right(heads=2, dim=64, vdim=64), mlp=mlp)],
                     width=W, vocab=V, scale=1.0)
    t = vup.random_model(cfg, 7)
    rng = np.random.default_rng(13)
    a, t["embed"] = planted_rows(top, rng)
    t["l0.mlp.router"] = a * (4.0 / W)
    for k in ("left.o", "left.o.b", "right.o"):
        t["l0.mix." + k] = 0 * t["l0.mix." + k]
    t["l0.norm2"], t["l0.norm2.b"], t["l0.norm2.alpha"] = np.ones(W), np.zeros(W), np.array(0.7)
    t = bf16_values(t)
    m, o = vup.build(cfg, dtype="bfloat16", max_seq_len=n + 2, max_batch_size=batch, tensors=t)
    ids = np.stack([planted_ids(n, rng) for _ in range(batch)])
    got, more = run(m, ids)
    m.close()
    assert more == (4 if shared else 2)
    for b in range(batch):
        assert vup.err(got[b], vup.fresh(o).run(ids[b])) < vup.BF16_BAR


def test_the_fused_form_still_answers_to_its_switch():
    """L3_MOE_EPI=1 (read once per process) takes prompts of any length to the one product with weights in its epilogue."""
    code = ("import numpy as np, test_moe_group_paths_gpu as t\n"
            "cfg, w = t.sigmoid_model(2, 264)\n"
            "m, o = t.mab.build(cfg, dtype='bfloat16', max_seq_len=2048, tensors=w)\n"
            "ids = t.planted_ids(300, np.random.default_rng(1))\n"
            "got, more = t.run(m, ids[None])\n"
            "assert more == 0 and t.mab.err(got[0], o.run(ids)) < t.mab.BF16_BAR")
    here = os.path.dirname(os.path.abspath(__file__))
    path = os.pathsep.join([here, os.path.dirname(here)] + [p for p in [os.environ.get("PYTHONPATH")] if p])
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, L3_MOE_EPI="1", PYTHONPATH=path), cwd=os.path.dirname(here),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
