"""Gated units whose activation runs in a product's epilogue without routing weights: GELU (Risalix) and the clamped unit (Vupitar), at the
row counts where the product changes its kernel (8 | 9, 128 | 129) and with rows and hidden values that do not fill a tile; against the
oracles, at the families' bars.  In fp32 mode the gate's weights are eight times as large, so that both of GELU's tails and both clamps
are reached."""
import numpy as np
import pytest

import test_risalix_gpu as risalix
import test_vupitar_gpu as vupitar

pytestmark = pytest.mark.gpu

ROWS = [1, 8, 9, 31, 128, 129, 300]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("ff", [72, 296])
@pytest.mark.parametrize("family", ["gelu", "clamp"])
def test_gated_units_over_rows(family, ff, dtype):
    f = risalix if family == "gelu" else vupitar
    cfg = f.config([f.attn(ff=ff)]) if family == "gelu" else f.config([f.layer(mlp={"kind": "dense", "ff": ff, "limit": 0.6})])
    t = f.random_model(cfg, 3)
    if dtype == "float32":
        for k in t:
            if k.endswith("mlp.gate"):
                t[k] = t[k] * 8
    m, o = f.build(cfg, dtype=dtype, max_seq_len=max(ROWS), tensors=t)
    ids = f.toks(max(ROWS), cfg["vocab"])
    want = o.run(ids)
    for n in ROWS:
        got = m.forward_rows(ids[None, :n], 0, list(range(n)))
        assert f.err(got, want[:n]) < (f.FP32_BAR if dtype == "float32" else f.BF16_BAR), n
    m.close()
