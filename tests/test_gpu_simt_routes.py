"""What the CUDA-core kernels' routing by head dim owes its callers: a call pays for its own head dims and
types and not for a larger template's (ratios of device times of two calls of one process, far from what
a wrong route shows), and dK, dV of repeated calls are the same bits."""
import pytest
import torch

from oracle import oracle as O
from tests.util import check_close, make_inputs, to_dev

pytestmark = pytest.mark.gpu


def ra():
    import ring_attention_b200

    return ring_attention_b200


def _qkv(b, h, n, dk, dv, dtype):
    g = torch.Generator("cuda").manual_seed(dk + dv)
    return [torch.randn((b, n, h, d), generator=g, device="cuda").to(dtype) for d in (dk, dk, dv)]


def _forward_ms(b, h, n, dk, dv, dtype=torch.float32):
    q, k, v = _qkv(b, h, n, dk, dv, dtype)
    best = float("inf")
    with torch.no_grad():
        for _ in range(4):
            ra().ring_attention(q, k, v, "sp", block_impl="simt")
            a, b_ = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(4_000_000)  # the host enqueues the calls under it
            a.record()
            for _ in range(4):
                ra().ring_attention(q, k, v, "sp", block_impl="simt")
            b_.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b_) / 4)
    return best


@pytest.mark.parametrize("dk,dv", [(160, 32), (256, 64), (192, 128)])
def test_a_forward_pays_for_its_own_value_columns(dk, dv):
    # the kernel with 256 value columns instead of 64 or 128: equal times; with its own: 0.49 to 0.6 of them
    assert _forward_ms(2, 4, 1500, dk, dv) < 0.8 * _forward_ms(2, 4, 1500, dk, 256)


def test_a_forward_pays_for_its_own_key_columns():
    # Q K^T over 128 padded columns instead of 16: equal times
    assert _forward_ms(2, 4, 1500, 8, 128) < 0.85 * _forward_ms(2, 4, 1500, 128, 128)


@pytest.mark.parametrize("d", [80, 128])
def test_a_forward_on_bf16_inputs_costs_no_more_than_on_float32(d):
    # staged element by element, bf16 tiles took 1.5 times the time of float32 ones
    assert _forward_ms(1, 8, 1000, d, d, torch.bfloat16) < 1.25 * _forward_ms(1, 8, 1000, d, d)


@pytest.mark.parametrize("dk,dv", [(160, 32), (256, 64), (192, 128), (8, 128), (20, 100)])
def test_those_head_dims_against_the_oracle(dk, dv):
    q, k, v, do, _ = make_inputs(dk, 2, 130, 200, 2, dk, torch.float32, dv=dv)
    t = [to_dev(x).requires_grad_(True) for x in (q, k, v)]
    out = ra().ring_attention(*t, "sp")
    grads = torch.autograd.grad(out, t, to_dev(do))
    check_close(out, O.mha(q, k, v), torch.float32, "out")
    for name, got, want in zip(("dq", "dk", "dv"), grads, O.mha_grads(q, k, v, do)):
        check_close(got, want, torch.float32, name, 2e-5)


@pytest.mark.parametrize("b,h,lq,lk,d,dtype,mask", [
    (1, 4, 1024, 1024, 64, torch.float32, True), (2, 4, 777, 1000, 64, torch.float32, False),
    (1, 2, 300, 500, 33, torch.float32, False), (1, 4, 1000, 1000, 128, torch.float32, True),
    (1, 4, 1000, 1000, 96, torch.bfloat16, True), (1, 1, 8192, 64, 64, torch.float32, False)])
def test_repeated_calls_repeat_dk_and_dv(b, h, lq, lk, d, dtype, mask):
    """Few key tiles: the query range is split over CTAs, whose sums are added in a fixed order."""
    q, k, v = _qkv(b, h, max(lq, lk), d, d, dtype)
    t = [x[:, :n].contiguous().requires_grad_(True) for x, n in ((q, lq), (k, lk), (v, lk))]
    do = torch.randn_like(t[0])
    kw = {}
    if mask:
        pos = torch.arange(lq, dtype=torch.int32, device="cuda").expand(b, lq).contiguous()
        kw = dict(bias_fn=ra().ScoreMod(causal=True, window=lq // 3), bias_q_kwargs={"q_positions": pos},
                  bias_kv_kwargs={"kv_positions": pos})
    out = ra().ring_attention(*t, "sp", block_impl="simt", **kw)
    first = torch.autograd.grad(out, t, do, retain_graph=True)
    for _ in range(5):
        again = torch.autograd.grad(out, t, do, retain_graph=True)
        assert torch.equal(first[1], again[1]) and torch.equal(first[2], again[2])
