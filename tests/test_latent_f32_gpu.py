"""Latent attention of prompts in fp32 mode over expanded cache rows: portions of 64 tokens and more, at the edges of the rule, of the
64-key tiles and of the 128-row expansion, with and without rotated part, sinks, both gates, a cache shared with a later layer,
several sequences, a second portion behind the first.  Against the float64 oracle at the families' fp32 bar (1e-4 of the logit scale),
and against portions of 40 tokens, which attend in the folded form: both are chains of fp32 sums over the same values, a few hundred
roundings of 2^-24 each: 2e-5."""
import numpy as np
import pytest

import test_gifudra_gpu as gif
import test_rakelorn_gpu as rak

pytestmark = pytest.mark.gpu


def _check(m, o, vocab, n, batch):
    ids = np.random.default_rng(n).integers(0, vocab, (batch, n))
    whole = m.forward_rows(ids, 0, list(range(batch * n))).reshape(batch, n, -1)
    for b in range(batch):
        o.reset()
        assert gif.err(whole[b], o.run(ids[b])) < 1e-4
    parts = gif.in_portions(m, ids[0], [40])
    assert gif.err(whole[0], parts) < 2e-5
    if n >= 130:
        two = gif.in_portions(m, ids[0], [65, 65, 9])
        assert gif.err(whole[0], two) < 2e-5
    m.close()


@pytest.mark.parametrize("n,batch", [(63, 1), (64, 2), (65, 1), (128, 3), (200, 1)])
@pytest.mark.parametrize("heads,dim,rot,vdim,rank", [(3, 16, 8, 24, 56), (2, 128, 64, 128, 512), (1, 40, 24, 136, 72)])
def test_sinks_wide_gates_and_shared_caches(n, batch, heads, dim, rot, vdim, rank):
    a = dict(heads=heads, dim=dim, rot_dim=rot, vdim=vdim, kv_rank=rank, scale=(dim + rot) ** -0.5)
    cfg = gif.config([gif.latent(**a, ff=40), gif.latent(**a, kv_from=0)], width=72)
    m, o = gif.build(cfg, 6, max_seq_len=n + 3, max_batch_size=batch)
    _check(m, o, cfg["vocab"], n, batch)


@pytest.mark.parametrize("n,batch", [(64, 1), (150, 2)])
def test_head_gates_and_rotary_pairs(n, batch):
    cfg = rak.config([rak.latent(4, 32, 16, 40, kv_rank=64, dims=8), rak.latent(2, 64, 16, 64, kv_rank=48)], width=72)
    m, o = rak.build(cfg, 7, max_seq_len=n + 3, max_batch_size=batch)
    _check(m, o, cfg["vocab"], n, batch)


def test_short_portions_behind_long_prefixes_keep_the_folded_form():
    """A portion expands its whole prefix again: 64 tokens do it at the start of a sequence and behind up to twice their number, not behind
    a longer prefix, 256 tokens of eight heads behind any (the launches of a call tell the two forms apart)."""
    cfg = gif.config([gif.latent(heads=8, dim=16, rot_dim=8, vdim=24, kv_rank=64, scale=0.2, ff=40)], width=72)
    m, o = gif.build(cfg, 8, max_seq_len=900, max_batch_size=3)
    ids = np.random.default_rng(5).integers(0, cfg["vocab"], (3, 900))
    at, count, got = 0, {}, []
    for n in (64, 64, 64, 300, 64, 40, 256, 48):
        m.launch_count(reset=True)
        got.append(m.forward_rows(ids[:, at:at + n], at, list(range(3 * n))).reshape(3, n, -1))
        count[at, n] = m.launch_count()
        at += n
    for b in range(3):
        o.reset()
        assert gif.err(np.concatenate([g[b] for g in got]), o.run(ids[b, :at])) < 1e-4
    m.close()
    expanded = count[0, 64]   # a GEMM per sequence
    assert [count[64, 64], count[128, 64], count[192, 300], count[596, 256]] == [expanded] * 4
    assert all(count[k] < expanded for k in ((492, 64), (556, 40), (852, 48)))
