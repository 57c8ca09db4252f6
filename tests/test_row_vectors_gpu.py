"""Row kernels that hold rows, or eight tokens of four channels, in registers as 16-byte vectors (rowvec.cuh): norms, the residual's
norm, output stages, convolutions with their preparations, combinations - at the shapes that reach them, with token counts at the edges
of the eight, batches, and a second portion that reads the first one's convolution tail.  fp32 mode against the float64 oracle at
the families' fp32 bars: a value that is lost or misplaced is an error of the size of the logits."""
import numpy as np
import pytest

import test_debuzen_gpu as deb
import test_mabedra_gpu as mab
import test_risalix_gpu as ris

pytestmark = pytest.mark.gpu


def _check(fam, cfg, n, batch, bar, seed=5):
    m, o = fam.build(cfg, seed=seed, max_seq_len=n + 2, max_batch_size=batch)
    ids = np.random.default_rng(n).integers(0, cfg["vocab"], (batch, n))
    whole = m.forward_rows(ids, 0, list(range(batch * n))).reshape(batch, n, -1)
    cut = n // 2 + 1
    a, b = (m.forward_rows(ids[:, s:e], s, list(range(batch * (e - s)))).reshape(batch, e - s, -1) for s, e in ((0, cut), (cut, n)))
    for i in range(batch):
        if hasattr(o, "reset"):
            o.reset()
        want = o.run(ids[i])
        assert fam.err(whole[i], want) < bar
        assert fam.err(np.concatenate([a[i], b[i]]), want) < bar
    m.close()


@pytest.mark.parametrize("n,batch", [(9, 1), (16, 2), (17, 1), (40, 3)])
@pytest.mark.parametrize("width,heads", [(128, 1), (640, 2), (1536, 3)])
def test_post_norm_rows(n, batch, width, heads):
    layers = [ris.lightning(heads, 128, 128, tuple(np.linspace(0.7, 0.98, heads))), ris.delta(heads, heads, 128, 128, 4), ris.attn(2 * heads, heads, 128, 0.1, ff=256)]
    _check(ris, ris.config(layers, width=width), n, batch, ris.FP32_BAR)


@pytest.mark.parametrize("n,batch", [(9, 1), (24, 2), (66, 1), (67, 2)])
@pytest.mark.parametrize("width,dim,dims,ff", [(128, 64, 64, 256), (516, 64, 16, 1028), (1152, 128, 64, 8192)])
def test_parallel_rows(n, batch, width, dim, dims, ff):
    layers = [mab.attn(2, 1, dim, 128, 9, dims=dims, mlp=mab.dense(ff)), mab.attn(2, 2, dim, 64, 0, dims=dim, mlp=mab.dense(72))]
    _check(mab, mab.config(layers, width=width, taps=4), n, batch, mab.FP32_BAR)


@pytest.mark.parametrize("n,batch", [(9, 1), (16, 2), (33, 1), (23, 3)])
@pytest.mark.parametrize("width,groups,heads", [(128, 1, 1), (512, 4, 2), (1536, 3, 3), (2048, 4, 2)])
def test_pre_norm_rows(n, batch, width, groups, heads):
    layers = [deb.par(heads=heads, kv_heads=heads, dim=128, vdim=256, conv=4), deb.par2(heads=16, groups=2, state=64, vdim=64, conv=4, norm_groups=2),
              deb.gla(heads, 128, 128)]
    _check(deb, deb.config(layers, width=width, groups=groups), n, batch, deb.FP32_BAR)
