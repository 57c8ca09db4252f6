"""Programmatic dependent launches: whether a chunk's kernels are launched as dependents of one another (by rows and layer size; everywhere and
nowhere with L3_PDL=1 and 0; nowhere with L3_FLAG_NO_PDL) changes no bit of a result and no count of launches, and the switches belong to
the handle that was made with them."""
import numpy as np
import pytest

import test_debuzen_gpu as deb
import test_gifudra_gpu as gif
import test_mabedra_gpu as mab
import test_rakelorn_gpu as rak
import test_risalix_gpu as ris
import test_vupitar_gpu as vup
from llama3_np_b200 import Llama, ModelArgs, _cabi
from llama3_np_b200.debuzen import Debuzen
from llama3_np_b200.gifudra import Gifudra
from llama3_np_b200.mabedra import Mabedra
from llama3_np_b200.rakelorn import Rakelorn
from llama3_np_b200.risalix import Risalix
from llama3_np_b200.synth import make_weights
from llama3_np_b200.vupitar import Vupitar

pytestmark = pytest.mark.gpu


def _llama(dtype, B, flags, dim=288, heads=6, ff=768, layers=2):
    args = ModelArgs(dim=dim, n_layers=layers, n_heads=heads, n_kv_heads=heads, vocab_size=600, max_seq_len=96, max_batch_size=B, dtype=dtype)
    return Llama(make_weights(args, ff, seed=3), args, flags=flags), 600


FAMILIES = {
    "debuzen": (Debuzen, lambda: deb.config([deb.par(), deb.par2(), deb.gla()]), deb.random_tensors),
    "gifudra": (Gifudra, lambda: gif.config([gif.latent(ff=96), gif.latent(kv_from=0, ff=96)]), gif.random_model),
    "mabedra": (Mabedra, lambda: mab.config([mab.attn(mlp=mab.moe()), mab.attn(mlp=mab.dense(128))]), mab.random_model),
    "rakelorn": (Rakelorn, lambda: rak.config([rak.latent(), rak.gru()]), rak.random_model),
    "risalix": (Risalix, lambda: ris.config([ris.attn(ff=128), ris.lightning()]), ris.random_model),
    "vupitar": (Vupitar, lambda: vup.config([vup.layer()]), vup.random_model),
}


def _family(name, dtype, B, flags):
    cls, config, tensors = FAMILIES[name]
    cfg = config()
    return cls(cfg, tensors(cfg, 3), dtype=dtype, max_seq_len=96, max_batch_size=B, flags=flags), cfg["vocab"]


def _outputs(m, vocab, B, llama):
    ids = np.random.default_rng(B).integers(0, vocab, (B, 50))
    m.launch_count(reset=True)
    if llama:
        out = [np.array(m(ids[:, :40], 0)), np.array(m(ids[:, 40:41], 40)), np.array(m(ids[:, 41:44], 41))]
        m.reset_cache()
        out.append(np.array(m.generate_all(ids[:, :9], 20)))
    else:
        rows = [b * 40 + t for b in range(B) for t in (0, 39)]
        out = [np.array(m.forward_rows(ids[:, :40], 0, rows)), np.array(m.forward_rows(ids[:, 40:41], 40, list(range(B)))), np.array(m.generate_all(ids[:, :9], 8))]
    n = m.launch_count()
    m.close()
    return out, n


@pytest.mark.parametrize("B", [1, 6, 12, 20, 40])
@pytest.mark.parametrize("name,dtype", [("llama", "float32"), ("llama", "bfloat16")] + [(f, d) for f in sorted(FAMILIES) for d in ("float32", "bfloat16")])
def test_every_switch_gives_the_same_bits(name, dtype, B, monkeypatch):
    if name != "llama" and B > 12:
        B = B // 20 + 2
    make = (lambda flags: _llama(dtype, B, flags)) if name == "llama" else (lambda flags: _family(name, dtype, B, flags))
    want, n = _outputs(*make(0), B, name == "llama")
    for env, flags in (("0", 0), ("1", 0), (None, _cabi.FLAG_NO_PDL)):
        monkeypatch.delenv("L3_PDL", raising=False)
        if env:
            monkeypatch.setenv("L3_PDL", env)
        got, k = _outputs(*make(flags), B, name == "llama")
        assert k == n
        for a, b in zip(got, want):
            assert np.array_equal(a, b, equal_nan=True), (env, flags)


def _dependent(m, B, L):
    return _cabi.lib().l3_debug_pdl(m._h, B, L)


def test_the_switches_belong_to_a_handle(monkeypatch):
    plain, _ = _llama("float32", 12, 0)
    quiet, _ = _llama("float32", 12, _cabi.FLAG_NO_PDL)
    assert [_dependent(plain, 12, L) for L in (1, 5)] == [1, 1] and [_dependent(quiet, 12, L) for L in (1, 5)] == [0, 0]
    monkeypatch.setenv("L3_PDL", "0")     # heard by the handles that are made from now on
    off, _ = _llama("float32", 12, 0)
    assert _dependent(off, 12, 5) == 0 and _dependent(plain, 12, 5) == 1
    monkeypatch.setenv("L3_PDL", "1")
    on, _ = _llama("float32", 32, 0)
    assert _dependent(on, 30, 1) == 1 and _dependent(off, 12, 5) == 0
    for m in (plain, quiet, off, on):
        m.close()


def test_the_rule():
    m, _ = _llama("float32", 64, 0)
    assert [_dependent(m, b, 1) for b in (1, 8, 9, 16, 17, 32, 33, 64)] == [0, 0, 1, 1, 0, 0, 1, 1]    # steps by sequences
    assert all(_dependent(m, 1, n) for n in (2, 8, 9, 32, 33, 90))                                      # prompts
    m.close()
    for name in FAMILIES:
        for dtype in ("float32", "bfloat16"):
            m, _ = _family(name, dtype, 36, 0)
            rows = (1, 4, 5, 8, 9, 32, 33)
            want = [1, 1, 0, 0, 1, 1, 1] if name == "mabedra" else [1, 1, 1, 1, 0, 0, 1] if dtype == "float32" else [1] * 7
            assert [_dependent(m, b, 1) for b in rows] == want, (name, dtype)
            assert [_dependent(m, 1, n) for n in rows[1:]] == ([1, 0, 0, 1, 1, 1] if name == "mabedra" else [1] * 6), (name, dtype)
            m.close()
