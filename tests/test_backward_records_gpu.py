"""Backward pass where the statistics of a query do not go into its record (an operand of the tensor core): logits far
from zero, masked rows, rows without a key, gradients that are not finite."""
import numpy as np
import pytest
import torch

import flash_tt_attn as fta
from oracle import tt_attn_oracle as npo

pytestmark = pytest.mark.gpu


def _run(q, k, v, bias, do, scale):
    leaves = [x.cuda().requires_grad_(True) for x in (q, k, v, bias)]
    o = fta.attention(*leaves, scale)
    o.backward(do.cuda())
    fta.check_device_status()
    return {"o": o.detach(), "dq": leaves[0].grad, "dk": leaves[1].grad, "dv": leaves[2].grad, "dbias": fta.last_dbias_f32()}


@pytest.mark.parametrize("L1,L2,D,dtype,scale", [
    (5, 64, 32, torch.bfloat16, 32 ** -0.5), (4, 200, 32, torch.float16, -0.25), (7, 256, 64, torch.bfloat16, 0.125),
    (3, 130, 64, torch.float16, 0.125), (4, 128, 32, torch.float16, 0.0), (4, 136, 32, torch.bfloat16, 1.0e-30),
])
def test_queries_with_and_without_a_record(L1, L2, D, dtype, scale):
    g = torch.Generator().manual_seed(L2 * D)
    q, k, v, do = (torch.randn(1, 2, L1, L2, D, generator=g).to(dtype) for _ in range(4))
    bias = torch.randn(1, 2, L2, L2, generator=g).to(dtype)
    bias[:, :, 1] += 120.0           # |c| below the limit
    bias[:, :, 2] -= 190.0           # and above it
    bias[:, 0, 33] += 8000.0         # (the sum rounds to 16 bits: the oracle sees the same values)
    if dtype == torch.bfloat16:
        bias[:, 1, 40] = -1.0e9      # uniform
        bias[:, 0, 63] = torch.finfo(dtype).min
    got = _run(q, k, v, bias, do, scale)
    ref = npo.forward_backward(*(x.float().numpy() for x in (q, k, v, bias, do)), scale)
    for name, t in got.items():
        a = t.float().cpu().numpy()
        assert np.isfinite(a).all(), name
        # 16-bit P and results: see the tolerances of the other parity tests
        assert npo.max_abs(a, ref[name]) <= 2e-2, (name, npo.max_abs(a, ref[name]))
        if np.linalg.norm(ref[name]) > 1e-6:
            assert npo.rel_l2(a, ref[name]) <= 1e-2, (name, npo.rel_l2(a, ref[name]))


@pytest.mark.parametrize("L2,D", [(64, 32), (256, 64)])
def test_a_gradient_that_is_not_finite_stays_where_it_belongs(L2, D):
    """delta of one query is infinite: dQ of that query and its row of dBias are lost, and dV in the one column;
    everything else is what it is without."""
    g = torch.Generator().manual_seed(L2)
    q, k, v, do = (torch.randn(1, 1, 4, L2, D, generator=g).to(torch.bfloat16) for _ in range(4))
    bias = torch.randn(1, 1, L2, L2, generator=g).to(torch.bfloat16)
    bias[0, 0, 11] = float("-inf")  # a query without a key beside it
    want = _run(q, k, v, bias, do, D ** -0.5)
    do2 = do.clone()
    do2[0, 0, 2, 9, 5] = float("inf")
    got = _run(q, k, v, bias, do2, D ** -0.5)
    assert torch.isfinite(torch.stack([t.float().abs().sum() for t in want.values()])).all()
    assert (want["dq"][0, 0, :, 11] == 0).all() and (want["dbias"][0, 0, 11] == 0).all()
    assert not torch.isfinite(got["dq"][0, 0, 2, 9]).any() and not torch.isfinite(got["dbias"][0, 0, 9]).any()
    assert not torch.isfinite(got["dv"][0, 0, 2, :, 5]).any()
    keep = torch.ones(D, dtype=torch.bool)
    keep[5] = False
    assert torch.equal(got["dv"][0, 0, 2][:, keep], want["dv"][0, 0, 2][:, keep])
    rows = [0, 1, 3]
    for name in ("dq", "dk", "dv"):
        assert torch.equal(got[name][:, :, rows], want[name][:, :, rows]), name
