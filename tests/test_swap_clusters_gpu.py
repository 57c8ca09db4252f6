"""Products of 9 - 128 rows whose K slices are a cluster (gemm_swap.cu): shapes for which the plan chooses one (asserted; 9 and 16 bf16 rows
of 6144 x 4096 are the ones beside them that it publishes), rows that do not divide over the slices, tiles' edges and a ragged K, in both
operand kinds; against float64, and bit for bit the same from run to run and as slices that meet in device memory.  All other epilogues -
rotation, residual, gated units, arg-max - through models whose every product is such a cluster.
Bounds: bf16 operands are exact, sums of K terms in fp32 accumulators that truncate, K / 16 * 2^-24 of the accumulated size at the worst,
4096 / 16 * 2^-24 = 1.5e-5; three TF32 products leave 2^-22 of each term and truncate likewise."""
import numpy as np
import pytest

from llama3_np_b200 import Llama, ModelArgs, _cabi
from llama3_np_b200.synth import make_weights
from oracle import ref_llama3 as orc
from test_gemm_plan_cpu import GATED, RESID, STORE, plan

pytestmark = pytest.mark.gpu


def _product(x, w, bf16, path=4):
    out = np.empty((len(x), len(w)), np.float32)
    _cabi.check(_cabi.lib().l3_op_linear(0, _cabi.f32p(x), _cabi.f32p(w), len(x), len(w), x.shape[1], path, int(bf16), _cabi.f32p(out)))
    return out


@pytest.mark.parametrize("bf16", [True, False])
@pytest.mark.parametrize("n,k", [(128, 2048), (389, 4096), (3072, 2056), (6144, 4096), (9336, 2048)])
@pytest.mark.parametrize("rows", [9, 16, 19, 33, 64, 127])
def test_slices_in_a_cluster(rows, n, k, bf16):
    import torch
    rng = np.random.default_rng(rows + n)
    x, w = (torch.from_numpy(rng.standard_normal(s).astype(np.float32)) for s in ((rows, k), (n, k)))
    if bf16:
        x, w = x.bfloat16().float(), w.bfloat16().float()
    x, w = x.numpy(), w.numpy()
    got = _product(x, w, bf16)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert np.linalg.norm(got - want) < 1.5e-5 * np.linalg.norm(want)
    assert np.array_equal(got, _product(x, w, bf16))
    p = plan(rows, n, k, STORE, int(not bf16))
    assert p["slices"] > 1 and (p["ctas"] == p["slices"]) == (not (bf16 and n == 6144 and rows <= 16))
    assert np.array_equal(got, _product(x, w, bf16, path=7))


# rows = sequences that the 4 and 8 slices do not divide; the residual products of bf16 mode are shorter than the ones that may
# be added in place.  fp32: greedy tokens identical to the oracle's, logits at K eps / 2 of the largest (1376 terms); bf16 at the bar of the
# other bf16 steps
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("B", [9, 19, 33, 70, 127])
def test_every_epilogue(B, bf16):
    dim, ff, kv = (960, 960, 15) if bf16 else (512, 1376, 2)
    heads = dim // 64
    args = ModelArgs(dim=dim, n_layers=2, n_heads=heads, n_kv_heads=kv, vocab_size=1000, max_seq_len=24, max_batch_size=B, dtype="bfloat16" if bf16 else "float32")
    for n, k, epi in (((heads + 2 * kv) * 64, dim, STORE), (dim, dim, RESID), (2 * ff, dim, GATED), (dim, ff, RESID), (1000, dim, STORE)):
        p = plan(B, n, k, epi, int(not bf16))
        assert p["ctas"] == p["slices"] > 1 and not p["any_order"] and B % p["slices"], (n, k, epi, p)
    w = make_weights(args, ff, seed=B)
    ids = np.random.default_rng(B).integers(0, 1000, (B, 6))
    m, o = Llama(w, args), orc.OracleLlama(w, args)
    want = np.asarray(o(ids, 0)), np.asarray(o(ids[:, :1], 6))
    got = np.asarray(m(ids, 0)), np.asarray(m(ids[:, :1], 6))
    for g, t in zip(got, want):
        assert orc.scaled_max_err(g, t) < (3e-2 if bf16 else 8.2e-5)
    if not bf16:
        m.reset_cache()
        assert np.array_equal(m.generate_all(ids, 18), np.concatenate(list(orc.OracleLlama(w, args).generate(ids, 18)), axis=1))
    else:   # the fused arg-max takes the token that the step's logits name
        m.reset_cache()
        tokens = m.generate_all(ids, 8)
        m.reset_cache()
        m(ids, 0)
        assert np.array_equal(tokens[:, -1], np.asarray(m(tokens[:, :1], 7)).reshape(B, -1).argmax(-1))
    m.close()
