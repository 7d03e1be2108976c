"""Router logits (csrc/moe_router.cu) against float64: token and output tiles full and not, one CTA and clusters along k, a last step of k that is short.  An fp32
sum of K products in any order is within K 2^-24 of the sum of their magnitudes; sqrt(K) of the 2-norms is what random signs leave: 2e-6 of the result."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,E,K", [(1, 16, 1024), (64, 33, 2048), (33, 40, 2048), (31, 17, 136), (300, 20, 1024), (5000, 40, 512), (6500, 40, 2048), (6401, 17, 264), (2, 41, 264), (70, 100, 768), (4, 16, 640), (2, 40, 1152), (3, 1, 8)])
@pytest.mark.parametrize("bias", [False, True])
def test_against_float64(dtype, n, E, K, bias):
    from nanovllm import mixops as mx
    g = torch.Generator(device="cuda").manual_seed(n + E)
    x = torch.randn(n, K + 8, device="cuda", generator=g).to(dtype)[:, :K]
    w = torch.randn(E, K, device="cuda", generator=g)
    b = torch.randn(E, device="cuda", generator=g) if bias else None
    want = x.double() @ w.double().t() + (b.double() if bias else 0)
    got = mx.moe_logits(x, w, b)
    assert got.shape == (n, E) and (got - want).norm() <= 2e-6 * want.norm()


def test_other_sizes_go_to_the_library():
    from nanovllm import mixops as mx
    x, w = torch.randn(5, 20, device="cuda"), torch.randn(3, 20, device="cuda")
    assert torch.allclose(mx.moe_logits(x, w), x @ w.t(), atol=1e-5)


@pytest.mark.parametrize("n,E,own", [(40, 256, True), (4000, 256, False), (4000, 40, True)])
def test_wide_routers_of_long_steps_are_the_librarys(n, E, own):
    from nanovllm import mixops as mx, ops
    g = torch.Generator(device="cuda").manual_seed(E)
    x, w = torch.randn(n, 512, device="cuda", generator=g).bfloat16(), torch.randn(E, 512, device="cuda", generator=g)
    before = ops.LAUNCHES[0]
    got = mx.moe_logits(x, w)
    assert ops.LAUNCHES[0] - before == int(own)
    want = x.double() @ w.double().t()
    assert (got - want).norm() <= 2e-6 * want.norm()


def test_other_strides_go_to_the_library():
    """Rows, weights and biases that are views: what the library's product takes."""
    from nanovllm import mixops as mx
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, b = r(64, 30), r(64, 16), r(32)
    want = x.double().t() @ w.double() + b.double()[::2]
    for rows, weights, bias in ((x.t(), w.t().contiguous(), b[::2].contiguous()), (x.t().contiguous(), w.t(), b[::2].contiguous()), (x.t().contiguous(), w.t().contiguous(), b[::2])):
        assert (mx.moe_logits(rows, weights, bias) - want).norm() <= 2e-6 * want.norm()
