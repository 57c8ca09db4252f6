"""bf16 projections of 9 - 128 rows (gemm_swap.cu) inside a whole model: equal bits from call to call where the K slices of a residual
projection are few, and the gated epilogue in full fp32."""
import os

import numpy as np
import pytest

from llama3_np_b200 import Llama, ModelArgs
from llama3_np_b200.synth import make_weights

pytestmark = pytest.mark.gpu


def _model(tmp_path, hidden, w=None, dim=256, layers=2, max_seq_len=64):
    args = ModelArgs(dim=dim, n_layers=layers, n_heads=8, n_kv_heads=4, vocab_size=1024, max_seq_len=max_seq_len, max_batch_size=4)
    args.dtype = "bfloat16"
    path = os.path.join(str(tmp_path), "model.npz")
    np.savez(path, **(w or make_weights(args, hidden, seed=5)))
    return Llama(path, args), args


@pytest.mark.parametrize("hidden", [448, 512, 704, 960])
def test_a_prompt_gives_equal_bits_every_time(tmp_path, hidden):
    m, _ = _model(tmp_path, hidden)
    ids = np.random.default_rng(3).integers(3, 1024, (4, 9))
    want = m.forward_f32(ids, 0)
    for _ in range(40):
        m.reset_cache()
        assert np.array_equal(m.forward_f32(ids, 0).view(np.uint32), want.view(np.uint32))
    m.close()


@pytest.mark.parametrize("batch,tokens", [(3, 3), (4, 5), (4, 10), (4, 25)])
def test_silu_keeps_its_tail(tmp_path, batch, tokens):
    """A gate of -88 leaves silu(g) = -88 exp(-88) = -5e-37, a number that fp32 and bf16 hold; with an up value of 2^120 it decides the
    output.  (A reciprocal that gives 0 from 2^126 on loses it.)  Bound: operands and results in bf16, 2^-9 each, over one layer."""
    args = ModelArgs(dim=256, n_layers=1, n_heads=8, n_kv_heads=4, vocab_size=1024, max_seq_len=64, max_batch_size=4)
    w = make_weights(args, 512, seed=6)
    rng = np.random.default_rng(7)
    p = "model.layers.0."
    w["model.embed_tokens.weight"] = rng.choice([-1.0, 1.0], (1024, 256)).astype(np.float32)
    w["model.embed_tokens.weight"][:, 0] = 1
    w[p + "self_attn.o_proj.weight"] *= 0
    w[p + "post_attention_layernorm.weight"] = np.ones(256, np.float32)
    gate, up, down = (w[p + "mlp.%s_proj.weight" % k] for k in ("gate", "up", "down"))
    gate[0], up[0], down[:, 0] = 0, 0, 0
    gate[0, 0], up[0, 0], down[1, 0] = -88, 2.0 ** 120, 16
    m, _ = _model(tmp_path, 512, w, layers=1)
    ids = rng.integers(0, 1024, (batch, tokens))
    got = m.forward_f32(ids, 0).reshape(batch, -1)
    m.close()
    x = w["model.embed_tokens.weight"][ids[:, -1]].astype(np.float64)
    rms = lambda v: v / np.sqrt((v * v).mean(-1, keepdims=True) + args.norm_eps)   # noqa: E731
    g, u = rms(x) @ gate.T.astype(np.float64), rms(x) @ up.T.astype(np.float64)
    x = x + (g / (1 + np.exp(-g)) * u) @ down.T.astype(np.float64)
    want = (rms(x) * w["model.norm.weight"]) @ w["lm_head.weight"].T.astype(np.float64)
    assert np.abs(x[:, 1]).min() > 8   # the planted unit's share
    assert np.sqrt(((got - want) ** 2).mean(-1)).max() < 2e-2 * np.sqrt((want ** 2).mean())
