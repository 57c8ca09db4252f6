"""Softmax, differential, sigmoid and keep-first attention of prompts on the tensor cores (bf16 mode, heads of 64 and more):
lengths at the edges of the 128-query tiles and 64-key blocks, heads that are no multiple of a 64-entry slice, windows smaller
than a block, kept tokens within and beyond one block, a second portion that starts inside a block - each against the float64
oracle row by row at the families' bf16 bar, 6e-2: a wrong mask, head or slice changes rows by order one."""
import numpy as np
import pytest

import test_debuzen_gpu as deb
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
