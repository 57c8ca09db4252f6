"""bf16 tensor-core projections of more than 128 rows (gemm_tc.cu) over every way of cutting them: tiles of one CTA and of pairs, every
width in steps of 32, one round of tiles and several, K whole and in slices.  test_gemm_plan_cpu.py holds that SHAPES reach them all."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# remainders of rows and columns in all of them
SHAPES = [
    (324, 41, 88), (574, 1880, 536), (166, 34, 2328), (414, 1242, 72), (939, 2346, 352), (260, 3149, 72), (995, 3515, 264), (133, 7315, 88),
    (989, 4730, 80), (282, 7000, 72), (513, 7742, 80), (523, 4646, 72), (833, 6814, 72), (523, 5645, 72), (1036, 6688, 72), (870, 4716, 72),
    (1076, 7278, 72), (129, 4764, 1768), (395, 6196, 840), (131, 7422, 1344), (416, 8398, 784), (396, 5086, 928), (551, 7559, 776),
    (404, 6369, 1000), (1202, 4655, 784), (417, 7406, 1096), (1185, 5680, 784), (406, 8416, 3168), (1213, 7111, 800),
    # K in slices: pairs in one round and in two, single CTAs in two
    (434, 1000, 8192), (556, 1021, 8200), (1166, 1024, 8192), (1288, 1021, 14336), (312, 4000, 14336), (130, 200, 4104)]


def _bf16(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


def _linear(x, w):
    from llama3_np_b200 import _cabi
    out = np.empty((len(x), len(w)), np.float32)
    _cabi.check(_cabi.lib().l3_op_linear(0, _cabi.f32p(x), _cabi.f32p(w), len(x), len(w), x.shape[1], 3, 1, _cabi.f32p(out)))
    return out


@pytest.mark.parametrize("rows,n,k", SHAPES)
def test_every_cut(rows, n, k):
    """Products of bf16 values are exact; the accumulator loses at most 2^-23 of its value per instruction of 16 terms, half of that on
    average, and fp32 results their last half bit.  Entries are N(0, 1): 6 sigma bounds all of them."""
    rng = np.random.default_rng(rows + n + k)
    x, w = _bf16(rng.standard_normal((rows, k))), _bf16(rng.standard_normal((n, k)) / np.sqrt(k))
    out = _linear(x, w)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert np.abs(out - want).max() < 6 * (k / 16 + 2) * 2.0 ** -24
    assert np.linalg.norm(out - want) < (k / 16 + 2) * 2.0 ** -24 * np.linalg.norm(want)
    assert np.array_equal(out, _linear(x, w))   # slices are added in their order


def test_timeline_is_left_where_it_was_asked_for():
    from llama3_np_b200 import _cabi
    lib, buf = _cabi.lib(), (C.c_uint64 * 64)()
    x = np.ones((300, 256), np.float32)
    for on in (1, 0):
        assert lib.l3_debug_tc_timeline(0, on, None) == 0
        _linear(x, x)
        assert lib.l3_debug_tc_timeline(0, 0, buf) == 0
        assert any(buf) == bool(on)


@pytest.mark.parametrize("batch", [130, 200])
def test_pairs_inside_a_captured_decode_step(batch):
    """More than 128 sequences decode through these products, replayed from a graph: the tokens of the same steps launched one by one."""
    from llama3_np_b200 import Llama, ModelArgs, _cabi
    from llama3_np_b200.synth import make_weights
    args = ModelArgs(dim=512, n_layers=2, n_heads=8, n_kv_heads=4, vocab_size=1024, max_seq_len=32, max_batch_size=batch)
    args.dtype = "bfloat16"
    w = make_weights(args, 1536, seed=4)
    ids = np.random.default_rng(5).integers(3, 1024, (batch, 6))
    got = []
    for flags in (0, _cabi.FLAG_NO_GRAPH):
        m = Llama(w, args, flags=flags)
        tokens = m.generate_all(ids, 24)
        m.reset_cache()
        got.append((tokens, m.forward_f32(ids, 0)))
        m.close()
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1].view(np.uint32), got[1][1].view(np.uint32))
