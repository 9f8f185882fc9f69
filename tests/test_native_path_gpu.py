"""The native call path of ``attention()`` where it branches: with and without a backward pass to come."""
import pytest
import torch

import flash_tt_attn as fta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L1,L2,D,dtype", [(1, 8, 32, torch.float16), (5, 64, 32, torch.bfloat16), (3, 136, 64, torch.bfloat16)])
def test_forward_without_a_backward_pass_gives_the_same_output(L1, L2, D, dtype):
    """No statistics and no residual are written when nothing requires a gradient: same O, bit for bit,
    and tensors of one batch element keep working whatever stride that dimension carries."""
    g = torch.Generator(device="cuda").manual_seed(L2)
    q, k, v = (torch.randn(1, 2, L1, L2, D, device="cuda", dtype=dtype, generator=g) for _ in range(3))
    b = torch.randn(1, 2, L2, L2, device="cuda", dtype=dtype, generator=g)
    plain = fta.attention(q, k, v, b, 0.2)
    kept = fta.attention(q.clone().requires_grad_(), k, v, b, 0.2)
    with torch.no_grad():
        quiet = fta.attention(q.clone().requires_grad_(), k[:1].expand(1, -1, -1, -1, -1), v, b, 0.2)
    fta.check_device_status()
    assert plain.grad_fn is None and quiet.grad_fn is None and kept.grad_fn is not None
    assert torch.equal(plain, kept) and torch.equal(plain, quiet)
