"""Two fp32 handles whose head sizes share an attention kernel (attn_f32.cu: 64 and 48, 93 and 74 KB of shared memory) run prompts from two
threads: the limit of shared memory belongs to the kernel, so a call that set its own size could take it from the other one between its
setting and its launch.  Every call succeeds and gives the bits of a run on its own."""
import threading

import numpy as np
import pytest

from llama3_np_b200 import Llama, ModelArgs
from llama3_np_b200.synth import make_weights

pytestmark = pytest.mark.gpu


def test_head_sizes_that_share_a_kernel():
    ids = np.random.default_rng(0).integers(0, 128, (1, 70))
    models, want, failed = [], [], []
    for dim in (256, 192):
        args = ModelArgs(dim=dim, n_layers=6, n_heads=4, n_kv_heads=4, vocab_size=128, max_seq_len=80, max_batch_size=1)
        models.append(Llama(make_weights(args, 128, seed=dim), args))
        want.append(np.array(models[-1](ids, 0)))

    def prompts(i):
        try:
            for _ in range(400):
                assert np.array_equal(np.asarray(models[i](ids, 0)), want[i])
        except Exception as e:  # noqa: BLE001 - reported by the thread that started this one
            failed.append((i, repr(e)))

    threads = [threading.Thread(target=prompts, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for m in models:
        m.close()
    assert not failed
