"""The CUDA-core kernels for head dims 17 to 128: tile edges, unaligned rows, unequal head dims, masks
over more tiles than are classified at a time, split query ranges; against the float64 oracle at the
float32 bound of the other parity tests (every sum here has fewer terms than theirs)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.util import check_close, to_dev

pytestmark = pytest.mark.gpu


def ra():
    import ring_attention_b200

    return ring_attention_b200


def _check(b, lq, lk, h, dk, dv, mask, dtype=torch.float32, pack=False):
    rng = np.random.default_rng(lq + 3 * lk + dk)
    mk = lambda *s: to_dev(rng.standard_normal(s), dtype)
    q, k, v, do = mk(b, lq, h, dk), mk(b, lk, h, dk), mk(b, lk, h, dv), mk(b, lq, h, dv)
    if pack:  # rows that are not on 16-byte boundaries
        q, k = (torch.cat([t, t[..., :1]], -1)[..., :dk] for t in (q, k))
    kw, bias = {}, None
    if mask != "none":
        # queries at the end of the keys, so that every row sees one
        qpos = np.broadcast_to(np.arange(lq) + max(lk - lq, 0), (b, lq)).astype(np.int32)
        kpos = np.broadcast_to(np.arange(lk), (b, lk)).astype(np.int32)
        causal, window, slopes = "causal" in mask, 90 if "window" in mask else 0, O.alibi_slopes(h) if "alibi" in mask else None
        bias = O.score_mod_bias(b, h, qpos, kpos, None, None, None, None, causal, slopes, window)
        sm = ra().ScoreMod(causal=causal, window=window, alibi_slopes=None if slopes is None else to_dev(slopes))
        kw = dict(bias_fn=sm, bias_q_kwargs={"q_positions": to_dev(qpos, torch.int32)},
                  bias_kv_kwargs={"kv_positions": to_dev(kpos, torch.int32)})
        if mask == "dense":
            kw["bias_fn"] = lambda q_positions, kv_positions: to_dev(bias)
    t = [x.detach().requires_grad_(True) for x in (q, k, v)]
    out = ra().ring_attention(*t, "sp", block_impl="simt", **kw)
    grads = torch.autograd.grad(out, t, do)
    n = [x.detach().double().cpu().numpy() for x in (q, k, v, do)]
    check_close(out, O.mha(*n[:3], bias), dtype, "out")
    for name, got, want in zip(("dq", "dk", "dv"), grads, O.mha_grads(*n, bias)):
        check_close(got, want, dtype, name, 2e-5)


@pytest.mark.parametrize("lq,lk", [(1, 1), (64, 64), (63, 65), (65, 129), (1, 300), (300, 1)])
@pytest.mark.parametrize("dk,dv", [(17, 17), (64, 64), (65, 65), (128, 128), (40, 100), (128, 24)])
def test_edges(lq, lk, dk, dv):
    _check(2, lq, lk, 2, dk, dv, "none")


@pytest.mark.parametrize("mask", ["causal", "causal+window", "alibi", "dense"])
@pytest.mark.parametrize("dk", [32, 96])
def test_masks(mask, dk):
    _check(2, 200, 333, 3, dk, dk, mask)


@pytest.mark.parametrize("mask", ["none", "causal+window"])
def test_many_tiles(mask):
    """More than 256 key tiles (the forward's classes) and query tiles (the backward's)."""
    _check(1, 70, 64 * 256 + 70, 1, 32, 32, mask)
    if mask == "none":
        _check(1, 64 * 256 + 70, 70, 1, 32, 32, mask)


def test_full_grid_takes_the_wide_tile():
    _check(2, 640, 640, 16, 64, 64, "causal")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_unaligned_rows(dtype):
    _check(2, 100, 150, 2, 33, 33, "none", dtype, pack=True)
    _check(2, 100, 150, 2, 64, 64, "causal", dtype, pack=True)
