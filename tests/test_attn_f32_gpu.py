"""fp32 prompt attention in tiles of 32 rows x 64 keys (attn_f32.cu): lengths at the edges of tiles and of a warp's 8 rows, both ways of
walking the keys (one and two groups of warps), row pieces of every head size, portions that start inside a tile, and the masks."""
import numpy as np
import pytest

import test_debuzen_gpu as deb
from llama3_np_b200 import _cabi
from oracle import ref_llama3 as orc

pytestmark = pytest.mark.gpu


def _attend(q, k, v, start):
    B, L, H, HD = q.shape
    G = k.shape[2]
    out = np.empty((B, L, H * HD), np.float32)
    assert _cabi.lib().l3_op_attention(0, _cabi.f32p(q), _cabi.f32p(k), _cabi.f32p(v), B, L, H, G, HD, start, 0, 1, _cabi.f32p(out)) == 0
    return out


def _inputs(B, L, H, G, HD, start, seed):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal((B, n, h, HD)).astype(np.float32) for n, h in ((L, H), (start + L, G), (start + L, G))]


# the last two: more CTAs than two per SM (one group of warps), and short prompts of many sequences
@pytest.mark.parametrize("B,L,H,G,HD,start", [
    (1, 33, 4, 4, 48, 0), (1, 63, 6, 2, 16, 1), (1, 64, 4, 1, 96, 64), (2, 65, 8, 1, 128, 31), (1, 97, 4, 4, 32, 100), (1, 130, 3, 1, 64, 7),
    (2, 300, 16, 16, 128, 0), (250, 7, 4, 4, 48, 60)])
def test_softmax(B, L, H, G, HD, start):
    q, k, v = _inputs(B, L, H, G, HD, start, B + L + HD)
    got = _attend(q, k, v, start)
    kk, vv = (np.repeat(x.astype(np.float64), H // G, axis=2).transpose(0, 2, 1, 3) for x in (k, v))
    s = q.astype(np.float64).transpose(0, 2, 1, 3) @ kk.transpose(0, 1, 3, 2) / np.sqrt(HD)
    s = np.where(np.arange(start + L)[None] <= start + np.arange(L)[:, None], s, -np.inf)
    want = (orc.softmax_lastdim(s) @ vv).transpose(0, 2, 1, 3).reshape(B, L, -1)
    assert orc.scaled_max_err(got, want) < 3e-6   # the bar of the other fp32 attention kernels


# short prompts of many sequences, which run the same kernel by the count of their tiles; beside them the ones that keep the 16-row tiles
@pytest.mark.parametrize("B,L,H,G,HD,start", [
    (64, 33, 6, 6, 48, 0), (250, 7, 6, 2, 48, 60), (129, 17, 8, 8, 64, 3), (48, 2, 16, 4, 128, 40), (64, 15, 8, 8, 96, 0),
    (1, 47, 16, 16, 128, 0), (250, 5, 4, 4, 48, 9), (64, 33, 8, 8, 32, 0)])
def test_softmax_of_many_short_prompts(B, L, H, G, HD, start):
    test_softmax(B, L, H, G, HD, start)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_later_token_does_not_reach_rows_ahead_of_its_eight(bad):
    q, k, v = _inputs(1, 100, 2, 2, 64, 0, 5)
    clean = _attend(q, k, v, 0)
    k[0, 64], v[0, 64] = bad, bad
    got = _attend(q, k, v, 0)
    assert np.array_equal(got[0, :64], clean[0, :64])
    assert not np.isfinite(got[0, 64]).any()


# fp32 bar of the families' tests: 1e-4 of the logits' scale; a wrong mask, head or slice changes rows by order one
@pytest.mark.parametrize("n,more", [(33, 31), (65, 64), (130, 70)])
@pytest.mark.parametrize("kind", ["sigmoid", "sink"])
@pytest.mark.parametrize("heads,kv,dim,vdim,size,keep", [(4, 1, 64, 64, 40, 3), (2, 2, 72, 128, 5, 70), (2, 1, 16, 196, 1000, 2)])
def test_windows_with_kept_tokens(n, more, kind, heads, kv, dim, vdim, size, keep):
    left = deb.attn(heads, kv, dim, vdim, size=size, keep_first=keep, dims=dim - dim % 16, scale=dim ** -0.5)
    lc = (deb.par if kind == "sigmoid" else deb.par2)(left=left, mlp={"kind": "dense", "ff": 128})
    cfg = deb.config([lc, lc], width=120 if heads % 2 else 96)
    m, o = deb.build(cfg, 5, "float32", max_seq_len=n + more + 3)
    ids = np.random.default_rng(n).integers(0, cfg["vocab"], n + more)
    got = np.concatenate([m.forward_rows(ids[None, :n], 0, list(range(n))), m.forward_rows(ids[None, n:], n, list(range(more)))])
    m.close()
    deb.fresh(o)
    assert deb.err(got, o.run(ids)) < 1e-4
