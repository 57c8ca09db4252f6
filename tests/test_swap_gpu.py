"""bf16 projections of 9 - 128 rows (gemm_swap.cu) inside a whole model: equal bits from call to call where the K slices of a residual
projection are few."""
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
