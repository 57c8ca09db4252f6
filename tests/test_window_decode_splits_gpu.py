"""Window attention of single tokens with the keys of a head spread over 2, 3, 8 (a cluster that merges) and 10 CTAs (a launch that merges):
positions at which the last splits are empty, hold one key and are full, in both dtypes, against the oracle row by row at the families'
bars; the splits follow from the cache's length, in tiles of 64 keys."""
import numpy as np
import pytest

import test_debuzen_gpu as deb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cache", [128, 190, 512, 640])
@pytest.mark.parametrize("kind,heads,kv,dim,vdim,size,keep", [("sigmoid", 4, 1, 64, 64, 1000, 3), ("sink", 4, 2, 72, 128, 1000, 2), ("sink", 8, 1, 32, 64, 40, 4)])
def test_steps_match_the_oracle(kind, heads, kv, dim, vdim, size, keep, cache, dtype):
    left = deb.attn(heads, kv, dim, vdim, size=size, keep_first=keep, dims=dim - dim % 16, scale=dim ** -0.5)
    cfg = deb.config([(deb.par if kind == "sigmoid" else deb.par2)(left=left, mlp={"kind": "dense", "ff": 128})], width=96)
    m, o = deb.build(cfg, 6, dtype, max_seq_len=cache)
    ids = np.random.default_rng(cache).integers(0, cfg["vocab"], 110)
    got = [m.forward_rows(ids[None, :1], 0, [0])]
    at = 1
    for p in (1, 8, 63, 64, 65, 107, 109):   # the token at p alone, what lies before it as a portion
        if p > at:
            got.append(m.forward_rows(ids[None, at:p], at, list(range(p - at))))
        got.append(m.forward_rows(ids[None, p:p + 1], p, [0]))
        at = p + 1
    m.close()
    deb.fresh(o)
    assert deb.err(np.concatenate(got), o.run(ids)) < (deb.FP32_BAR if dtype == "float32" else deb.BF16_BAR)
