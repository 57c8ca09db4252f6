"""The prompt kernels of bf16 mode whose operands are pairs hi + lo of bf16 values, one launch at a time against 64-bit restatements on the
same inputs: a lost, doubled or misplaced low part is an error of 2^-9 to 2^-10 of the result, which a whole model's bar cannot see."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SINK, SIGMOID, SOFTMAX = 0, 1, 2


def _bf16(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


def _call(name, *args):
    from llama3_np_b200 import _cabi
    _cabi.check(getattr(_cabi.lib(), name)(0, *[_cabi.f32p(a) if isinstance(a, np.ndarray) else a for a in args]))


@pytest.mark.parametrize("B,L,start,M", [(1, 9, 0, 16), (3, 64, 0, 100), (2, 129, 0, 130), (2, 65, 63, 150), (3, 10, 190, 201)])
@pytest.mark.parametrize("H,G,DK,DV", [(4, 2, 64, 64), (3, 3, 72, 128), (2, 1, 128, 192)])
@pytest.mark.parametrize("kind,window,chunked,keep", [(SOFTMAX, 0, 0, 0), (SINK, 40, 0, 0), (SIGMOID, 23, 0, 3), (SINK, 7, 0, 70), (SOFTMAX, 48, 1, 0)])
def test_attention(B, L, start, M, H, G, DK, DV, kind, window, chunked, keep):
    """fp32 queries against bf16 caches whose unwritten rows are NaN.  Bound: a query's pair is right to 2^-18 of each entry and a weight's
    to 2^-18, both independent from entry to entry; the exponential to 2^-21; the accumulator drops at most 2^-23 per instruction of 16
    keys and part, (T / 16) 2^-23 = 1.5e-6 for 200 keys: 2^-15 leaves room for the scores' size, and is a twentieth of a lost part."""
    rng = np.random.default_rng(B * 1000 + L + DK)
    T = start + L
    q, k, v = (rng.standard_normal((B, T, n, d)).astype(np.float32) for n, d in ((H, DK), (G, DK), (G, DV)))
    hv = rng.standard_normal(H).astype(np.float32)
    scale = np.float32(DK ** -0.5)
    qkv = np.concatenate([a.reshape(B, T, -1) for a in (q, k, v)], -1)
    out = np.empty((B, L, H, DV), np.float32)
    _call("l3_op_prompt_attention", np.ascontiguousarray(qkv), hv, B, L, H, G, DK, DV, start, M, kind, window, chunked, keep, float(scale), out)
    i, j = np.arange(T)[start:, None], np.arange(T)[None]
    seen = j <= i
    if window:
        seen &= (i // window == j // window) if chunked else ((i - j < window) | (j < keep))
    kb, vb = (np.repeat(_bf16(a).astype(np.float64), H // G, 2) for a in (k, v))
    z = np.einsum("bihd,bjhd->bhij", q[:, start:].astype(np.float64), kb) * float(scale)
    if kind == SIGMOID:
        p = np.where(seen, 1.0 / (1.0 + np.exp(-(z + hv[:, None, None]))), 0.0)
    else:
        z = np.where(seen, z, -np.inf)
        m = z.max(-1, keepdims=True)
        p = np.exp(z - m)
        p = p / (p.sum(-1, keepdims=True) + (np.exp(hv[:, None, None] - m) if kind == SINK else 0.0))
    want = np.einsum("bhij,bjhd->bihd", p, vb)
    err = np.linalg.norm(out - want, axis=-1) / np.linalg.norm(want, axis=-1)
    assert err.max() < 2.0 ** -15 * 4 and np.linalg.norm(out - want) < 2.0 ** -15 * np.linalg.norm(want), (err.max(), np.linalg.norm(out - want) / np.linalg.norm(want))


def _recur(q, k, v, lg, beta, S):
    q, k, v, g, S = (a.astype(np.float64) for a in (q, k, v, np.exp(lg.astype(np.float64)), S))
    out = np.empty(v.shape)
    for t in range(q.shape[1]):
        S = S * g[:, t, :, :, None]
        u = v[:, t]
        if beta is not None:
            u = beta[:, t, :, None] * (u - np.einsum("bhkv,bhk->bhv", S, k[:, t]))
        S = S + k[:, t, :, :, None] * u[:, :, None]
        out[:, t] = np.einsum("bhkv,bhk->bhv", S, q[:, t])
    return out, S


@pytest.mark.parametrize("B,L,chunks", [(1, 128, 9), (2, 129, 1), (1, 191, 2), (3, 200, 9), (1, 320, 3)])
@pytest.mark.parametrize("H,DK,DV", [(2, 64, 16), (1, 128, 48), (3, 128, 256)])
@pytest.mark.parametrize("delta", [False, True])
@pytest.mark.parametrize("rate", [0.02, 0.5, 6.0])
def test_recurrences(B, L, chunks, H, DK, DV, delta, rate):
    """Outputs and the state left behind, from a state that is not empty, in one segment and in segments of a small workspace.  Bound: every
    operand is right to 2^-18 and the product of two low parts (2^-18) is left out, the decays to 2^-18 (running sums of up to 16 x 6):
    2^-15 of the result's 2-norm, a lost low part is 2^-10 and more.  The chain is held to 2^-19."""
    rng = np.random.default_rng(L + DK)
    shape = lambda d: (B, L, H, d) if d else (B, L, H)  # noqa: E731
    q, k, v = (rng.standard_normal(shape(d)).astype(np.float32) for d in (DK, DK, DV))
    q *= np.float32(DK ** -0.5)
    k /= np.linalg.norm(k, axis=-1, keepdims=True)
    lg = (-rate * rng.random(shape(DK))).astype(np.float32)
    beta = rng.random(shape(0)).astype(np.float32) if delta else None
    S0 = rng.standard_normal((B, H, DK, DV)).astype(np.float32)
    want, end = _recur(q, k, v, lg, beta, S0)
    for ws, bar in ((chunks, 2.0 ** -15), (0, 2.0 ** -19)):
        out, S = np.empty(shape(DV), np.float32), S0.copy()
        _call("l3_op_recurrence", q, k, v, lg, beta, S, B, L, H, DK, DV, ws, out)
        errs = [np.linalg.norm(a - b) / np.linalg.norm(b) for a, b in ((out, want), (S, end))]
        assert max(errs) < bar, (ws, errs)


@pytest.mark.parametrize("delta,B,H,least", [(True, 1, 2, 128), (True, 3, 21, 128), (True, 4, 16, 64), (False, 1, 7, 72), (False, 4, 2, 48)])
def test_which_portions_run_in_chunks(delta, B, H, least):
    """The chunk-parallel form takes the lengths from which it is the faster one, and no shorter ones."""
    def run(L):
        q, k, lg, v = (np.full((B, L, H, d), -0.1, np.float32) for d in (64, 64, 64, 16))
        beta = np.full((B, L, H), 0.5, np.float32) if delta else None
        _call("l3_op_recurrence", q, k, v, lg, beta, np.zeros((B, H, 64, 16), np.float32), B, L, H, 64, 16, 9, np.empty_like(v))

    run(least)
    with pytest.raises(ValueError):
        run(least - 1)
