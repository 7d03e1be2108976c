"""Linear layers of at most 16 rows (csrc/linear_rows.cu) give bit for bit what the launches they replace give: the library's products and b200_linear's
partials, the norm kernels and SiluAndMul.  One and two 8-row tiles, full and not, one chain of sums and up to eight along k, one, two and four tiles of weights, rows that the
norm holds in registers and reads twice, strided inputs."""
import pytest
import torch
import torch.nn.functional as F

from test_gpu_kernels import bf

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from nanovllm import ops as o
    return o


@pytest.mark.parametrize("rows", [1, 5, 8, 9, 16])
@pytest.mark.parametrize("n,k,splits", [(1024, 2048, 8), (1024, 3072, 8), (128, 512, 8), (2048, 1536, 4), (1024, 1024, 2)])
def test_product_in_parts(ops, rows, n, k, splits):
    x, w = bf(rows, k + 8, seed=1).cuda()[:, :k], (bf(n, k, seed=2) * k ** -0.5).cuda()
    got, res = ops.linear_rows(x, w, splits=splits)
    parts = ops.linear(x.contiguous(), w, ops.EPI_PARTIAL, 64, splits)
    want = torch.zeros(rows, n, device="cuda")
    for p in parts.view(splits, rows, n):
        want = want + p
    assert res is x and torch.equal(got, want.bfloat16())


@pytest.mark.parametrize("rows", [1, 4, 8, 11, 16])
@pytest.mark.parametrize("n,k", [(64, 512), (4096, 1024), (3072, 1024), (1600, 2048), (128, 2560), (64, 3072)])
@pytest.mark.parametrize("add,silu", [(False, False), (True, False), (True, True)])
def test_normed_product(ops, rows, n, k, add, silu):
    x, a, nw = (bf(rows, k, seed=3) * 2).cuda(), bf(rows, k + 16, seed=4).cuda()[:, :k], (1 + 0.2 * bf(k, seed=5)).cuda()
    w = (bf(2 * n if silu else n, k, seed=6) * k ** -0.5).cuda()
    x0 = x.clone()
    got, res = ops.linear_rows(x, w, nw, 1e-6, a if add else None, silu=silu, pdl=True)
    assert torch.equal(x, x0)
    if add:
        residual = x.clone()
        z, _ = ops.add_rmsnorm_partials(a.float().contiguous()[None], residual, nw, 1e-6)
        assert torch.equal(res, residual)
    else:
        z = ops.rmsnorm(x, nw, 1e-6)
    y = ops.linear(z, w, ops.EPI_BF16, 64)
    assert torch.equal(got, ops.silu_mul(y) if silu else y)


@pytest.mark.parametrize("rows", [1, 4, 16])
@pytest.mark.parametrize("n,k", [(4096, 1024), (6144, 1024)])
def test_one_chain_is_the_library(ops, rows, n, k):
    """What the step took its wide projections from before: the library's kernels of these sizes add the same products in the same order."""
    x, w = bf(rows, k, seed=7).cuda(), (bf(n, k, seed=8) * k ** -0.5).cuda()
    got, _ = ops.linear_rows(x, w)
    assert torch.equal(got, F.linear(x, w))


def test_refused_sizes(ops):
    from nanovllm._native import B200Error
    for rows, n, k, splits in [(17, 16, 512, 1), (1, 24, 512, 1), (1, 16, 544, 1), (1, 16, 512, 3), (1, 16, 1152, 9), (9, 16, 8192, 1)]:
        with pytest.raises(B200Error):
            ops.linear_rows(bf(rows, k).cuda(), bf(n, k).cuda(), splits=splits)


def test_norm_weights_of_another_size_or_type_are_refused(ops):
    """On the host: the kernel reads as many as x has columns."""
    from nanovllm._native import B200Error
    x, w = bf(4, 512).cuda(), bf(16, 512).cuda()
    for norm_w in (bf(256).cuda(), bf(1024).cuda()[::2], bf(512).cuda().float(), bf(512)):
        with pytest.raises((AssertionError, B200Error)):
            ops.linear_rows(x, w, norm_w, 1e-6)
