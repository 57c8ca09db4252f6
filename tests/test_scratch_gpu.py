"""Models whose prompts find no room for the workspaces of the faster paths (L3_SCRATCH_MB): the paths beside them take the calls, with the
same results within the families' bars, and nothing is refused."""
import numpy as np
import pytest

import test_debuzen_gpu as deb
import test_gifudra_gpu as gif
import test_mabedra_gpu as mab
import test_risalix_gpu as ris

pytestmark = pytest.mark.gpu

CASES = {
    "recurrences": (deb, lambda: deb.config([deb.gla(2, 64, 64, mlp={"kind": "dense", "ff": 96}), deb.par(heads=2, kv_heads=2, dim=64, vdim=64)], width=96), deb.random_tensors),
    "softmax": (ris, lambda: ris.config([ris.attn(2, 1, 64, 0.125, ff=128), ris.lightning(2, 64, 64)], width=128), ris.random_model),
    "differential": (mab, lambda: mab.config([mab.attn(2, 1, 64, 64, scale=0.125, mlp=mab.dense(128))], width=128), mab.random_model),
    "windows": (deb, lambda: deb.config([deb.par2(left=deb.attn(2, 1, 64, 64, size=40, dims=32, scale=0.125))], width=96), deb.random_tensors),
    "latent": (gif, lambda: gif.config([gif.latent(heads=2, dim=64, rot_dim=16, vdim=64, kv_rank=64, scale=0.125, ff=128)], width=128), gif.random_model),
}


@pytest.mark.parametrize("room", ["0", "1", None])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_any_room_will_do(name, dtype, room, monkeypatch):
    fam, config, tensors = CASES[name]
    if room is not None:
        monkeypatch.setenv("L3_SCRATCH_MB", room)
    cfg = config()
    m, o = fam.build(cfg, dtype=dtype, max_seq_len=210, max_batch_size=3, tensors=tensors(cfg, 3))
    ids = np.random.default_rng(2).integers(0, cfg["vocab"], (3, 200))
    m.launch_count(reset=True)
    got = m.forward_rows(ids, 0, list(range(600))).reshape(3, 200, -1)
    n = m.launch_count()
    for b in range(3):
        if hasattr(o, "reset"):
            o.reset()
        assert ris.err(got[b], o.run(ids[b])) < (1e-4 if dtype == "float32" else 6e-2)
    m.close()
    if room == "0" and (name, dtype) in (("differential", "bfloat16"), ("latent", "float32")):
        monkeypatch.delenv("L3_SCRATCH_MB")
        m, _ = fam.build(cfg, dtype=dtype, max_seq_len=210, max_batch_size=3, tensors=tensors(cfg, 3))
        m.launch_count(reset=True)
        m.forward_rows(ids, 0, [0])
        assert m.launch_count() != n    # with room, another path (where the number of launches tells them apart)
        m.close()
