"""Which router logits the own kernel forms and which the library (mixops.router_kernel): sizes that were measured in both, host arithmetic."""
import pytest

from nanovllm.mixops import router_kernel


@pytest.mark.parametrize("is32,own,sizes", [
    (False, True, [(1, 16, 1024), (1, 256, 2048), (64, 33, 2048), (64, 1000, 4096), (512, 256, 2048), (8192, 40, 2048), (8192, 80, 2048), (4, 1000, 1024), (0, 40, 2048)]),
    (False, False, [(1, 1000, 2048), (1, 256, 4096), (512, 1000, 1024), (2048, 256, 2048), (8192, 128, 2048), (8192, 256, 2048), (8192, 512, 4096)]),
    (True, True, [(1, 40, 2048), (1, 256, 1024), (64, 512, 2048), (256, 256, 2048), (8192, 40, 2048), (8, 1000, 1024)]),
    (True, False, [(1, 256, 2048), (1, 1000, 1024), (2, 1000, 1024), (256, 512, 2048), (2048, 64, 2048), (8192, 41, 2048), (8192, 128, 1024), (8192, 1000, 2048)])])
def test_the_faster_one(is32, own, sizes):
    for n, outputs, K in sizes:
        assert router_kernel(n, outputs, K, is32) == own, (n, outputs, K)
