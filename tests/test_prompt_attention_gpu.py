"""Softmax, differential, sigmoid and keep-first attention of prompts on the tensor cores (bf16 mode, heads of 64 and more):
lengths at the edges of the 128-query tiles and 64-key blocks, heads that are no multiple of a 64-entry slice, windows smaller
than a block, kept tokens within and beyond one block, a second portion that starts inside a block - each against the float64
oracle row by row at the families' bf16 bar, 6e-2: a wrong mask, head or slice changes rows by order one."""
import numpy as np
import pytest

import test_debuzen_gpu as deb
import test_gifudra_gpu as gif
import test_mabedra_gpu as mab
import test_risalix_gpu as ris

pytestmark = pytest.mark.gpu

# prompt length, length of a second portion behind it
LENGTHS = [(9, 9), (64, 65), (129, 63), (200, 130)]


def _run(m, o, n, more, vocab, run):
    ids = np.random.default_rng(n).integers(0, vocab, n + more)
    want = run(o, ids)
    got = m.forward_rows(ids[None, :n], 0, list(range(n)))
    got2 = m.forward_rows(ids[None, n:], n, list(range(more)))
    m.close()
    return np.concatenate([got, got2]), want


@pytest.mark.parametrize("n,more", LENGTHS)
@pytest.mark.parametrize("heads,kv,dim", [(4, 1, 64), (2, 2, 72), (2, 1, 128)])
def test_softmax(n, more, heads, kv, dim):
    cfg = ris.config([ris.attn(heads, kv, dim, dim ** -0.5, ff=128), ris.attn(heads, kv, dim, 2.0 * dim ** -0.5)], width=128)
    m, o = ris.build(cfg, 3, "bfloat16", max_seq_len=n + more + 3)
    got, want = _run(m, o, n, more, cfg["vocab"], lambda o, ids: o.run(ids))
    assert ris.err(got, want) < 6e-2


@pytest.mark.parametrize("n,more", LENGTHS)
@pytest.mark.parametrize("heads,kv,dim,vdim,window", [(4, 1, 64, 128, 100), (2, 2, 72, 64, 5), (2, 1, 128, 192, 0)])
def test_differential(n, more, heads, kv, dim, vdim, window):
    a = mab.attn(heads, kv, dim, vdim, window=window, scale=dim ** -0.5, mlp=mab.dense(128))
    cfg = mab.config([a, a], width=128)
    m, o = mab.build(cfg, 4, "bfloat16", max_seq_len=n + more + 3)
    got, want = _run(m, o, n, more, cfg["vocab"], lambda o, ids: (mab.fresh(o), o.run(ids))[1])
    assert mab.err(got, want) < 6e-2


@pytest.mark.parametrize("n,more", LENGTHS)
@pytest.mark.parametrize("kind", ["sigmoid", "sink"])
@pytest.mark.parametrize("heads,kv,dim,vdim,size,keep", [(4, 1, 64, 64, 40, 3), (2, 2, 72, 128, 5, 70), (2, 1, 128, 192, 1000, 2)])
def test_windows_with_kept_tokens(n, more, kind, heads, kv, dim, vdim, size, keep):
    left = deb.attn(heads, kv, dim, vdim, size=size, keep_first=keep, dims=dim - dim % 16, scale=dim ** -0.5)
    lc = deb.par(left=left, mlp={"kind": "dense", "ff": 128}) if kind == "sigmoid" else deb.par2(left=left, mlp={"kind": "dense", "ff": 128})
    cfg = deb.config([lc, lc], width=120 if heads % 2 else 96)
    m, o = deb.build(cfg, 5, "bfloat16", max_seq_len=n + more + 3)
    got, want = _run(m, o, n, more, cfg["vocab"], lambda o, ids: (deb.fresh(o), o.run(ids))[1])
    assert deb.err(got, want) < 6e-2


def _family(kind):
    """test module of the family, configuration, its random weights, an oracle run from a fresh state"""
    if kind == "softmax":
        return ris, ris.config([ris.attn(4, 2, 64, 0.125), ris.attn(2, 1, 72, 0.2)], width=128, side=0), ris.random_model, lambda o, ids: o.run(ids)
    if kind == "differential":
        cfg = mab.config([mab.attn(2, 1, 64, 128, window=70, scale=0.125, mlp=mab.dense(128))] * 2, width=128)
        return mab, cfg, mab.random_model, lambda o, ids: (mab.fresh(o), o.run(ids))[1]
    if kind == "latent":
        cfg = gif.config([gif.latent(heads=2, dim=64, rot_dim=16, vdim=72, kv_rank=64, scale=0.125, ff=64)], width=128)
        return gif, cfg, gif.random_model, lambda o, ids: (o.reset(), o.run(ids))[1]
    left = deb.attn(4, 2, 64, 64, size=23, keep_first=None if kind == "window" else 3, dims=32, scale=0.125)
    mlp = {"kind": "dense", "ff": 128}
    layer = deb.par(left=left, mlp=mlp) if kind == "sigmoid" else deb.par2(left=left, mlp=mlp)
    return deb, deb.config([layer, layer], width=96), deb.random_tensors, lambda o, ids: (deb.fresh(o), o.run(ids))[1]


@pytest.mark.parametrize("kind", ["softmax", "differential", "sigmoid", "sink", "window", "latent"])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_rows_that_no_query_sees_do_not_count(kind, value):
    """Infinities and NaN in cache rows behind a sequence's own: left by an earlier, longer request of the slot, and in the rows of the
    next head and the next sequence, which the last key block of a full cache reaches into (100 rows are no multiple of 64)."""
    M = 100
    fam, cfg, tensors, run = _family(kind)
    t = tensors(cfg, 12)
    big = cfg["vocab"] - 1
    t["embed"][big] = value
    m, o = fam.build(cfg, dtype="bfloat16", max_seq_len=M, max_batch_size=2, tensors=t)
    rng = np.random.default_rng(11)
    ids = rng.integers(0, big, (2, M))
    spoiled = ids.copy()
    spoiled[:, [25, 40, 70]] = big
    assert not np.isfinite(m.forward_rows(spoiled[:, :90], 0, [70, 160])).any()
    # the slots again, shorter, the second portion with kept tokens in a block of their own
    got = np.concatenate([m.forward_rows(ids[:, :20], 0, list(range(40))).reshape(2, 20, -1),
                          m.forward_rows(ids[:, 20:34], 20, list(range(28))).reshape(2, 14, -1)], 1)
    for b in range(2):
        assert ris.err(got[b][:, :big], run(o, ids[b, :34])[:, :big]) < 6e-2   # (a tied output projection has the token's row, too)
    # a sequence that fills its cache, ahead of one that is spoiled
    ids[1, [5, 20]] = big
    got = m.forward_rows(ids, 0, list(range(M)))
    assert ris.err(got[:, :big], run(o, ids[0])[:, :big]) < 6e-2
    m.close()


def _against_portions_of_8(m, vocab, batch, n):
    """Several sequences at once against portions of 8 tokens, which run the FFMA kernels on fp32 queries and the same bf16 caches."""
    ids = np.random.default_rng(n).integers(0, vocab, (batch, n))
    whole = m.forward_rows(ids, 0, list(range(batch * n))).reshape(batch, n, -1)
    parts = np.concatenate([m.forward_rows(ids[:, p:p + 8], p, list(range(batch * len(ids[0, p:p + 8])))).reshape(batch, -1, whole.shape[-1])
                            for p in range(0, n, 8)], 1)
    m.close()
    return max(ris.err(whole[b], parts[b]) for b in range(batch))


@pytest.mark.parametrize("n,batch", [(65, 3), (129, 2)])
def test_packed_queries_of_softmax_layers(n, batch):
    """Scores of a few hundred: queries rounded to 16 bits would move the logits by 5e-2 (restated in 64 bits), their pairs move them
    by 1e-4."""
    cfg = ris.config([ris.attn(4, 2, 64, 16.0, ff=128)], width=128, side=0)
    m, _ = ris.build(cfg, 3, "bfloat16", max_seq_len=n + 3, max_batch_size=batch)
    assert _against_portions_of_8(m, cfg["vocab"], batch, n) < 1e-2


@pytest.mark.parametrize("n,batch", [(65, 3), (129, 2)])
def test_two_maps_that_nearly_cancel(n, batch):
    """lambda = 1 and queries of the second map 1 % from the first's: the head norm lifts what is left of a1 - a2, so that queries of 16
    bits would move the logits by 0.18 and weights of 16 bits by 5e-2 (restated in 64 bits), pairs by 6e-4."""
    a = mab.attn(2, 1, 64, 128, window=0, diff=0.3, scale=0.5, scaling=None, mlp=mab.dense(128))
    cfg = mab.config([a], width=128)
    t = mab.random_model(cfg, 4)
    rng = np.random.default_rng(0)
    for name, heads, off in (("q", 2, 0.01), ("k", 1, 0.0)):
        for key in (f"l0.mix.{name}", f"l0.mix.{name}.b"):
            w = t[key].reshape((heads, 2, 64) + t[key].shape[1:])
            w[:, 1] = w[:, 0] * (1.0 + off * rng.standard_normal(w[:, 0].shape))
            t[key] = w.reshape(t[key].shape)
    for key in ("lq1", "lk1", "lq2"):
        t[f"l0.mix.{key}"][:] = 0.0
    t["l0.mix.lq1"][0], t["l0.mix.lk1"][0] = 1.0, np.log(1.7)    # lambda = 1.7 - 1 + 0.3
    m, _ = mab.build(cfg, dtype="bfloat16", max_seq_len=n + 3, max_batch_size=batch, tensors=t)
    assert _against_portions_of_8(m, cfg["vocab"], batch, n) < 2e-2
