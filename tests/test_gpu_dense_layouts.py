"""The layouts a `bias_fn` callable may return its tile in: broadcast axes, slices of a larger table,
transposed and misaligned views.  Every layout that the tensor-core kernels take must give the bits that
a dense tile of the same values gives; a contiguous tile whose base is off 16 bytes goes to the CUDA-core
kernels, as it always did."""
import pytest
import torch

pytestmark = pytest.mark.gpu
B, H, N = 2, 3, 256  # two key tiles: dQ has two contributions, whose order does not change their sum
IMPL_SIMT, IMPL_TCGEN05 = 1, 2


def _table(*shape):
    return torch.randn(shape, generator=torch.Generator("cuda").manual_seed(7), device="cuda")


def _misaligned():
    return _table(B * H * N * N + 1)[1:].view(B, H, N, N)


LAYOUTS = {
    "heads": lambda: _table(B, 1, N, N).expand(B, H, N, N),
    "one head": lambda: _table(B, 1, N, N),
    "queries": lambda: _table(B, H, 1, N).expand(B, H, N, N),
    "batch": lambda: _table(1, H, N, N).expand(B, H, N, N),
    "batch and heads": lambda: _table(N, N).expand(B, H, N, N),
    "keys": lambda: _table(B, H, N, 1).expand(B, H, N, N),
    "rows of a wider table": lambda: _table(B, H, N, N + 64)[..., 32 : 32 + N],
    "rows of a taller table": lambda: _table(B, H, N + 5, N)[:, :, 3 : 3 + N],
    "heads outermost": lambda: _table(H, B, N, N).transpose(0, 1),
    "transposed": lambda: _table(B, H, N, N).transpose(2, 3),
    "odd pitch": lambda: _table(B, H, N, N + 1)[..., :N],
    "misaligned view": lambda: _table(B, H, N, N + 64)[..., 1 : 1 + N],
}


def _run(bias, d, block_impl="cuda"):
    import ring_attention_b200 as ra
    from ring_attention_b200._lib import lib

    g = torch.Generator("cuda").manual_seed(3)
    q, k, v, do = (torch.randn((B, N, H, d), generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    t = [x.requires_grad_(True) for x in (q, k, v)]
    out = ra.ring_attention(*t, "sp", bias_fn=lambda: bias, block_impl=block_impl)
    impl = [lib.ra_last_impl()]
    grads = torch.autograd.grad(out, t, do)
    impl.append(lib.ra_last_impl())
    return (out, *grads), impl


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_a_layout_gives_the_bits_of_the_dense_tile(layout, d):
    bias = LAYOUTS[layout]()
    dense = bias.expand(B, H, N, N).clone(memory_format=torch.contiguous_format)
    got, impl = _run(bias, d)
    want, _ = _run(dense, d)
    assert impl == [IMPL_TCGEN05] * 2
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        assert torch.equal(a, b), f"{layout}: {name}"


@pytest.mark.parametrize("d", [64, 128])
def test_a_misaligned_contiguous_tile_stays_on_the_cuda_cores(d):
    bias = _misaligned()
    assert bias.data_ptr() % 16 and bias.is_contiguous()
    got, impl = _run(bias, d)
    want, _ = _run(bias.clone(), d, "simt")
    assert impl == [IMPL_SIMT] * 2
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        if name != "dq":  # added to atomically by the splits of four query tiles
            assert torch.equal(a, b), name
    with pytest.raises(RuntimeError):
        _run(bias, d, "tcgen05")
