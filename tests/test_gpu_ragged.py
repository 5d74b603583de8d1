"""Lengths that are not multiples of 128 on the tensor-core kernels (a ring of one, bf16): tile edges,
single rows, every mask family, strided inputs; against the CUDA-core kernels, which hold P and dS in
float32, and through them against the float64 oracle of the other parity tests."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.util import check_close, make_inputs, to_dev

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
IMPL_SIMT, IMPL_TCGEN05 = 1, 2


def ra():
    import ring_attention_b200

    return ring_attention_b200


def _both(q, k, v, do, bias_fn=None, bias_q_kwargs=None, bias_kv_kwargs=None):
    """(out, dq, dk, dv) of the tensor-core and of the CUDA-core kernels.  Both backward passes read the
    first one's out and L: a bf16 step between two outs would move delta, and with it whole rows."""
    from ring_attention_b200 import ring as R
    from ring_attention_b200._lib import lib

    ring, scale = R.resolve_axis("sp"), q.shape[-1] ** -0.5
    mod = (bias_fn, bias_q_kwargs or {}, bias_kv_kwargs or {})
    results, saved = [], None
    for name, code in (("cuda", IMPL_TCGEN05), ("simt", IMPL_SIMT)):
        R._set_impl(name)
        out, lse = R._fused_fwd(ring, q, k, v, scale, *mod)
        assert lib.ra_last_impl() == code
        saved = saved or (out, lse)
        results.append((out, *R._fused_bwd(ring, q, k, v, *saved, do, scale, *mod)))
        assert lib.ra_last_impl() == code
        bits = C.c_uint32(0)
        assert lib.ra_device_status(C.byref(bits)) == 0, hex(bits.value)
    R._set_impl("cuda")
    return results


def _agree(got, want, what):
    """Both round to bf16 what differs by the 2^-17 of a two-part P or dS: at most one bf16 step apart
    (2^-7 of the value), plus 2^-17 of the summed terms, whose absolute sum stays below 32 here."""
    got, want = got.double(), want.double()
    assert torch.equal(got.isnan(), want.isnan()), f"{what}: NaN pattern"
    bad = (got - want).abs() > 2.0**-7 * want.abs() + 32 * 2.0**-17
    assert not (bad & ~want.isnan()).any(), f"{what}: {(got - want).abs().nan_to_num().max():.3e}"


SIZES = [(1, 1), (1, 300), (300, 1), (127, 129), (129, 127), (128, 200), (200, 128), (255, 385), (448, 1500), (1025, 1025),
         # tiles in a row at which sums start to move out: dK and dV from 17 query tiles, O from 33 key tiles
         (2048, 100), (2049, 100), (4100, 70), (100, 4096), (70, 4097), (70, 8200)]


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("lq,lk", SIZES)
def test_lengths(lq, lk, d):
    q, k, v, do, _ = make_inputs(lq + lk, 2, lq, lk, 3, d, BF)
    t = [to_dev(x, BF) for x in (q, k, v, do)]
    got, want = _both(*t)
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        _agree(a, b, name)
    check_close(got[0], O.mha(q, k, v), BF, "out")
    for name, a, b in zip(("dq", "dk", "dv"), got[1:], O.mha_grads(q, k, v, do)):
        check_close(a, b, BF, name)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("mask", ["causal", "causal+docs", "docs", "prefix", "alibi+window", "alibi", "no key"])
@pytest.mark.parametrize("order", ["contiguous", "shuffled"])
def test_masks(mask, order, d):
    """Masks whose last tiles are cut; positions in order and scattered; rows that see no key (NaN
    results, zero gradient contributions).  Inputs are slices of one packed projection."""
    b, h, n = 2, 2, 333
    rng = np.random.default_rng(5)
    packed = torch.from_numpy(rng.standard_normal((b, n, 3, h, d))).to("cuda", BF)
    q, k, v = (packed[:, :, i] for i in range(3))
    do = torch.from_numpy(rng.standard_normal((b, n, h, d))).to("cuda", BF)
    pos = np.stack([np.arange(n)] * b) if order == "contiguous" else np.stack([rng.permutation(n) for _ in range(b)])
    pos = to_dev(pos, torch.int32)
    qkw, kkw = {"q_positions": pos}, {"kv_positions": pos}
    sm = dict(causal="causal" in mask)
    if "docs" in mask or mask == "no key":
        seg = to_dev(np.sort(rng.integers(0, 5, (b, n)), axis=1), torch.int32)
        qkw["q_segment_ids"], kkw["kv_segment_ids"] = seg, seg
        if mask == "no key":
            kkw["kv_segment_ids"] = torch.where(seg == 2, 7, seg)
    if mask == "prefix":
        pre = to_dev(rng.integers(0, 2, (b, n)), torch.bool)
        qkw["q_prefix_mask"], kkw["kv_prefix_mask"] = pre, pre
    if "alibi" in mask:
        sm["alibi_slopes"] = to_dev(O.alibi_slopes(h), torch.float32)
    if "window" in mask:
        sm.update(causal=True, window=70)
    kw = dict(bias_fn=ra().ScoreMod(**sm), bias_q_kwargs=qkw, bias_kv_kwargs=kkw)
    for name, a, b_ in zip(("out", "dq", "dk", "dv"), *_both(q, k, v, do, **kw)):
        _agree(a, b_, name)


@pytest.mark.parametrize("d", [64, 128])
def test_long_sums_are_not_truncated(d):
    """The tensor pipe cuts every sum it accumulates towards zero, so a long sum in tensor memory comes out too
    small by a common factor; the kernels therefore move O, dK and dV to float32 sums every 32 (16) tiles.
    The factor is measured against 64 bits over every element of the results.  Bound: 16 sums a tile, each cut by
    2^-24 on average, over the tiles of one move; sums of one sign pattern grow from zero, half of that; plus
    four standard deviations of what rounding the results to bf16 leaves in the factor."""
    n, h = 16061, 2
    g = torch.Generator("cuda").manual_seed(d)
    q, k, v, do = (torch.randn((1, n, h, d), generator=g, device="cuda").to(BF) for _ in range(4))
    t = [x.requires_grad_(True) for x in (q, k, v)]
    out = ra().ring_attention(*t, "sp")
    _, dk, dv = torch.autograd.grad(out, t, do)
    got = [x.detach()[0].double() for x in (out, dk, dv)]
    sums = torch.zeros((3, 3), dtype=torch.float64, device="cuda")
    for hh in range(h):
        Q, K, V, G = (x.detach()[0, :, hh].double() for x in (q, k, v, do))
        O64, dK, dV = torch.empty_like(Q), torch.zeros_like(K), torch.zeros_like(V)
        for r in (slice(i, min(i + 2048, n)) for i in range(0, n, 2048)):
            P = (Q[r] @ K.T / d**0.5).softmax(-1)
            O64[r] = P @ V
            delta = (got[0][r, hh] * G[r]).sum(-1)  # from the rounded out, as the backward has it
            dK += (P * (G[r] @ V.T - delta[:, None])).T @ Q[r] / d**0.5
            dV += P.T @ G[r]
        for i, want in enumerate((O64, dK, dV)):
            err = got[i][:, hh] - want
            sums[i] += torch.stack([(err * want).sum(), (want * want).sum(), (err * want).pow(2).sum()])
    for name, tiles, (a, b, c) in zip(("out", "dk", "dv"), (32, 16, 16), sums.tolist()):
        assert abs(a / b) < tiles * 16 * 2.0**-25 + 4 * c**0.5 / b, f"{name}: factor 1 {a / b:+.2e}"


def test_named_implementation_still_refuses():
    q = torch.zeros((1, 100, 1, 64), dtype=BF, device="cuda")
    with pytest.raises(RuntimeError):
        ra().ring_attention(q, q, q, "sp", block_impl="tcgen05")
