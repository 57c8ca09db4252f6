"""fp32 prompts of layer lists over operands cut into bf16 parts beforehand (layerlist.cu ll_cut_operands), through whole models: matrices that
lie inside a fused one, strided inputs, plain, residual and gated epilogues, the expansion of latent rows, experts.  Where L3_SCRATCH_MB
leaves no room for the parts the kernel cuts its operands itself, with the same parts, products and order of sums: the same bits."""
import numpy as np
import pytest

import test_debuzen_gpu as deb
import test_gifudra_gpu as gif
import test_mabedra_gpu as mab
import test_risalix_gpu as ris

pytestmark = pytest.mark.gpu

N = 400   # tokens of the prompt: matrices of a million values and more are cut
MLP = {"kind": "dense", "ff": 2048}
MODELS = {   # a parallel mixer's halves in one input matrix; streams and latent rows; GELU; experts beside a dense layer
    "parallel": (deb, lambda: deb.config([deb.par(left=deb.attn(8, 2, 64, 64, size=300, dims=32, scale=0.125), heads=8, kv_heads=8, dim=64, vdim=64, mlp=MLP),
                                          deb.par2(left=deb.attn(8, 8, 64, 64, size=100, dims=32, scale=0.125), mlp=MLP)], width=512, groups=4), deb.random_tensors),
    "latent": (gif, lambda: gif.config([gif.latent(heads=8, dim=128, rot_dim=32, vdim=128, q_rank=768, kv_rank=512, scale=160 ** -0.5, ff=2048),
                                        gif.latent(heads=8, dim=128, rot_dim=32, vdim=128, q_rank=768, kv_rank=512, scale=160 ** -0.5, kv_from=0, ff=2048)], width=512), gif.random_model),
    "gelu": (ris, lambda: ris.config([ris.attn(8, 2, 64, 0.125, ff=2048), ris.lightning(8, 64, 64, decay=(0.7, 0.8, 0.9, 0.92, 0.95, 0.97, 0.98, 0.99), ff=2048)], width=512), ris.random_model),
    "experts": (mab, lambda: mab.config([mab.attn(8, 2, 64, 64, scale=0.125, window=300, mlp={"kind": "moe", "expert": {"ff": 512}, "router": {"experts": 8, "top": 2}, "shared": {"ff": 512}}),
                                         mab.attn(8, 2, 64, 64, scale=0.125, window=300, mlp=mab.dense(2048))], width=512), mab.random_model),
}


def _build(name, cap):
    fam, config, tensors = MODELS[name]
    cfg = config()
    return fam.build(cfg, dtype="float32", max_seq_len=cap, tensors=tensors(cfg, 3))[0], cfg


@pytest.mark.parametrize("name", sorted(MODELS))
def test_the_same_bits_without_room_for_them(name, monkeypatch):
    got, launches = [], []
    for room in (None, "33"):   # 32 MB for the partial sums of the K split, which both have
        if room:
            monkeypatch.setenv("L3_SCRATCH_MB", room)
        m, cfg = _build(name, N + 130)
        ids = np.random.default_rng(1).integers(0, cfg["vocab"], (1, N + 129))
        m.launch_count(reset=True)
        out = [m.forward_rows(ids[:, :N], 0, [0, 127, 128, N - 1])]
        launches.append(m.launch_count())
        out.append(m.forward_rows(ids[:, N:], N, [0, 128]))   # 129 rows: the expansion still has all of them
        m.close()
        got.append(np.concatenate(out))
    assert launches[0] > launches[1]      # a launch for the parts of each cut input
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("cap", [128, N])
def test_only_handles_whose_prompts_can_use_them_hold_them(cap, monkeypatch):
    import torch
    used = []
    for room in (None, "33"):
        if room:
            monkeypatch.setenv("L3_SCRATCH_MB", room)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        m, _ = _build("gelu", cap)
        used.append(free - torch.cuda.mem_get_info()[0])
        m.close()
    parts = 6 * 2 * 3 * 2048 * 512        # gate, up and down projections of both layers
    assert (used[0] - used[1] >= parts - (4 << 20)) if cap == N else (used[0] - used[1] < 8 << 20), used
