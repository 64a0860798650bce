"""Which grouped-product kernel a routed layer's step gets (on the host)."""
import pytest
import torch

from ginfer_b200.ops import moe


@pytest.mark.parametrize("pairs, experts, streamed, kernel", [
    (1, 4, True, "few"), (192, 4, True, "few"), (193, 4, True, True), (384, 8, True, "few"), (386, 8, True, True),
    (768, 16, True, "few"), (768, 64, True, "few"), (770, 64, True, True), (768, None, True, "few"),
    (1023, 64, True, True), (1024, 4, True, "tcgen05"), (1, 4, False, "gemv"), (20, 32, False, "gemv"),
    (21, 32, False, True), (1024, 32, False, "tcgen05")])
def test_the_kernel_follows_the_pairs_and_the_experts(pairs, experts, streamed, kernel):
    x = torch.zeros(2, 256, dtype=torch.bfloat16)
    assert moe.kernel_for(x, pairs, (256, 64), (64, 256), streamed, experts) == kernel
    assert moe.kernel_for(x.float(), pairs, (256, 64), (64, 256), streamed, experts) is False


@pytest.mark.parametrize("K, kernel", [(4096, "few"), (4104, True)])
def test_rows_that_shared_memory_does_not_hold_go_elsewhere(K, kernel):
    x = torch.zeros(2, K, dtype=torch.bfloat16)
    assert moe.kernel_for(x, 8, (K, 64), (64, K)) == kernel
    assert moe.kernel_for(x, 8, (K, 64), (64, K), streamed=False) == (True if kernel is True else "gemv")
