"""Global norm of mixed gradients on the kernels (needs a B200)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_global_norm_is_summed_in_64_bits():
    from dmuon_b200.grad_clip import local_pow_sum

    torch.manual_seed(6)
    dev = torch.device("cuda", 0)
    grads = [torch.randn(n, device=dev).to(dt) for n, dt in (
        (1, torch.float32), (4099, torch.bfloat16), (5_000_000, torch.float32), (300_001, torch.float16))]
    want = sum(g.double().square().sum() for g in grads)
    # block totals are fp32 sums of some thousand products by 256 threads; what is left is their rounding and the
    # result's own (6e-8 each)
    assert abs(local_pow_sum(grads, 2.0, dev).double() - want) < 4e-7 * want


def test_small_blocks_are_not_lost_beside_a_large_one():
    """Totals below half an ulp of what is there already: 32-bit addition would drop every one of them."""
    from dmuon_b200.grad_clip import local_pow_sum

    dev = torch.device("cuda", 0)
    # 2^24 first (its ulp is 2), then 2000 tensors of one block each with a total of 0.9, in later launches
    grads = [torch.full((1,), 4096.0, device=dev)]
    grads += list(torch.full((2000, 8), (0.9 / 8) ** 0.5, device=dev).unbind())
    want = sum(g.double().square().sum() for g in grads)
    assert want > 2**24 + 1700
    # rounding of the block totals (6e-8 of a ten-thousandth of the sum) and of the result
    assert abs(local_pow_sum(grads, 2.0, dev).double() - want) < 1.2e-7 * want
