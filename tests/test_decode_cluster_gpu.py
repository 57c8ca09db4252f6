"""The decode step in one cluster (decode_cluster.cu) against the oracle and against the path of a kernel per product: every batch slot
count, rows that do not divide evenly over the CTAs, heads of 16 to 128, shared KV heads, the first and the last position of a cache and
contexts of more keys than one turn of the attention takes."""
import numpy as np
import pytest

from llama3_np_b200 import Llama, ModelArgs, _cabi
from llama3_np_b200.synth import make_weights
from oracle import ref_llama3 as orc

pytestmark = pytest.mark.gpu

SHAPES = {
    # name: (dim, layers, heads, kv_heads, hidden, vocab, max_seq)
    "hd48": (288, 3, 6, 6, 768, 1001, 72),     # 4 or 5 fours of rows per CTA, three pieces of K
    "hd16": (64, 2, 4, 2, 160, 96, 40),        # one four per CTA, K below a warp's turn, idle attention CTAs
    "hd96": (192, 1, 2, 1, 200, 130, 24),      # K = 192 and 200: last turns of 16 and 18 lanes; 32 lanes per key
    "hd128": (256, 2, 2, 1, 392, 200, 300),    # 16 keys per row of threads: several turns over 300 positions
    "hd32": (128, 1, 4, 1, 264, 64, 512),      # eight lanes of 16 per key, the longest cache it takes
}


def _args(name, B):
    d, nl, hn, kv, hid, vs, msl = SHAPES[name]
    args = ModelArgs(dim=d, n_layers=nl, n_heads=hn, n_kv_heads=kv, vocab_size=vs, max_seq_len=msl, max_batch_size=B)
    return args, make_weights(args, hid, seed=5)


@pytest.mark.parametrize("B", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("name", list(SHAPES))
def test_steps_match_the_oracle(name, B):
    """Forward steps at position 0, at the edges of the attention's turns and at the last position; fp32 against the fp32 oracle: sums
    of K <= 768 terms differ by their order only, K eps / 2 = 5e-5 of the largest value at the worst."""
    args, w = _args(name, B)
    M = args.max_seq_len
    rng = np.random.default_rng(B)
    ids = rng.integers(0, args.vocab_size, (B, M))
    m, o, m2 = Llama(w, args), orc.OracleLlama(w, args), Llama(w, args, flags=_cabi.FLAG_NO_MEGA)
    for model in (m, m2):      # the layers are one launch here and five or more each there
        model.launch_count(reset=True)
        model(ids[:, :1], 0)
    assert m.launch_count() < 6 and m2.launch_count() >= 5 * args.n_layers
    tol = lambda want: 5e-5 * np.abs(want).max()

    def check(lo, hi):
        want = np.asarray(o(ids[:, lo:hi], lo))
        got, ref = np.asarray(m(ids[:, lo:hi], lo)), np.asarray(m2(ids[:, lo:hi], lo))
        np.testing.assert_allclose(got, want, rtol=0, atol=tol(want))
        np.testing.assert_allclose(got, ref, rtol=0, atol=tol(want))

    edges = sorted({p for p in (1, 31, 32, 33, 63, 64, 127, 128, 129, 255, 256, 257, M - 2, M - 1) if p < M})
    check(0, 1)
    at = 1
    for p in edges:
        if p < at:
            continue
        if p > at:
            check(at, p)
        check(p, p + 1)
        at = p + 1
    for li in range(args.n_layers):
        for a, b in zip(m.read_cache(li), m2.read_cache(li)):
            np.testing.assert_allclose(a, b, rtol=0, atol=tol(b))
    m.close()
    m2.close()


@pytest.mark.parametrize("B", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("name", ["hd48", "hd16", "hd96"])
def test_greedy_tokens_match_the_oracle(name, B):
    args, w = _args(name, B)
    ids = np.random.default_rng(3).integers(0, args.vocab_size, (B, 5))
    cap = args.max_seq_len
    want = np.concatenate(list(orc.OracleLlama(w, args).generate(ids, cap)), axis=1)
    m = Llama(w, args)
    counts = []
    for n in (cap, cap, cap - 10):  # the head's counters are back at zero behind a run
        m.launch_count(reset=True)
        assert np.array_equal(m.generate_all(ids, n), want[:, :n - 5])
        counts.append(m.launch_count())
        m.reset_cache()
    assert counts[1] - counts[2] == 2 * 10  # layers, LM head: the step is the cluster's
    assert np.array_equal(np.concatenate(list(m.generate(ids, cap)), axis=1), want)
    m.close()


def test_a_wait_that_ran_out_is_reported():
    """The host side of the cluster step's error word, which the test sets in the kernel's place: the call that finds it fails, the next one
    is whole again.  The same word serves the layer-list kernels."""
    import test_risalix_gpu as ris
    args, w = _args("hd48", 2)
    ids = np.random.default_rng(3).integers(0, args.vocab_size, (2, 5))
    m = Llama(w, args)
    want = m.generate_all(ids, 20)
    step = m(ids[:, :1], 0).copy()
    calls = [lambda: m.generate_all(ids, 20), lambda: m(ids[:, :1], 0), lambda: list(m.generate(ids, 20))]
    for call in calls:
        _cabi.check(_cabi.lib().l3_debug_fail_wait(m._h), m._h)
        with pytest.raises(RuntimeError, match="gave up waiting"):
            call()
        assert np.array_equal(m.generate_all(ids, 20), want) and np.array_equal(m(ids[:, :1], 0), step)
    m.close()
    cfg = ris.config([ris.lightning()])
    m, _ = ris.build(cfg)
    ids = ids[:1] % cfg["vocab"]
    want = m.forward_rows(ids, 0, [4])
    _cabi.check(_cabi.lib().l3_debug_fail_wait(m._h), m._h)
    with pytest.raises(RuntimeError, match="gave up waiting"):
        m.forward_rows(ids, 0, [4])
    assert np.array_equal(m.forward_rows(ids, 0, [4]), want)
    m.close()
    m = Llama(w, args, flags=_cabi.FLAG_NO_MEGA)   # no kernel of this handle has such a wait
    assert _cabi.lib().l3_debug_fail_wait(m._h) == -1
    m.close()


@pytest.mark.parametrize("B", [1, 3, 8])
@pytest.mark.parametrize("vocab", [5, 531, 26003])
def test_head_of_every_vocabulary_size(vocab, B):
    """The LM head behind the layers: fewer rows than CTAs, a few rows each, and more rows than shared memory holds (26003 x 288 x 4 bytes
    over 132 CTAs: 220 KB); logits of a forward step and greedy tokens.  Bound as above."""
    args = ModelArgs(dim=288, n_layers=1, n_heads=6, n_kv_heads=6, vocab_size=vocab, max_seq_len=40, max_batch_size=B)
    w = make_weights(args, 768, seed=7)
    ids = np.random.default_rng(vocab).integers(0, vocab, (B, 9))
    m, o = Llama(w, args), orc.OracleLlama(w, args)
    for p, q in ((0, 8), (8, 9)):
        want = np.asarray(o(ids[:, p:q], p))
        np.testing.assert_allclose(np.asarray(m(ids[:, p:q], p)), want, rtol=0, atol=5e-5 * np.abs(want).max())
    m.reset_cache()
    got = np.concatenate(list(m.generate(ids, 30)), axis=1)
    want = np.concatenate(list(orc.OracleLlama(w, args).generate(ids, 30)), axis=1)
    m.close()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("B", [1, 8])
def test_logits_are_as_exact_as_short_chains_of_sums(B):
    """Layers that add nothing: the logits are norm(embedding) W^T.  An fp32 rounding is 2.5e-8 of its value in the mean square, so 288
    products as 32 chains of nine that meet in five steps (1440 + 5 x 288 partial sums of unit variance, and two roundings of the normed
    row) are sqrt(12) of them or 8.8e-8 away from 64 bits; chains of 36 sqrt(23.5) or 1.23e-7.  The one factor of the norm is left out."""
    args = ModelArgs(dim=288, n_layers=1, n_heads=6, n_kv_heads=6, vocab_size=32000, max_seq_len=8, max_batch_size=B)
    w = make_weights(args, 768, seed=3)
    w["model.layers.0.self_attn.o_proj.weight"][:] = 0
    w["model.layers.0.mlp.down_proj.weight"][:] = 0
    ids = np.arange(7, 7 + B)[:, None]
    m = Llama(w, args)
    got = np.asarray(m(ids, 0), np.float64).reshape(B, -1)
    m.close()
    x = w["model.embed_tokens.weight"][ids[:, 0]].astype(np.float64)
    x = x / np.sqrt((x * x).mean(-1, keepdims=True) + args.norm_eps) * w["model.norm.weight"]
    want = x @ w["lm_head.weight"].astype(np.float64).T
    want *= (got * want).sum(-1, keepdims=True) / (want * want).sum(-1, keepdims=True)
    err = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
    assert err.max() < 1.05e-7, err
