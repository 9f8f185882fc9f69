"""Forward pass at the sizes where its two kernels and their tiles meet: key blocks of 64 and 128, groups of two and
four rows, one wave of CTAs and more."""
import numpy as np
import pytest
import torch

import flash_tt_attn as fta
from oracle import tt_attn_oracle as npo

pytestmark = pytest.mark.gpu

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _inputs(B, H, L1, L2, D, dtype):
    g = torch.Generator().manual_seed(L1 * 4096 + L2 + D)
    q, k, v = (torch.randn(B, H, L1, L2, D, generator=g).to(DTYPES[dtype]) for _ in range(3))
    return q, k, v, torch.randn(B, H, L2, L2, generator=g).to(DTYPES[dtype])


def _check(o, q, k, v, bias, scale, dtype):
    fta.check_device_status()
    want = npo.forward(*(x.float().numpy() for x in (q, k, v, bias)), scale)
    got = o.float().cpu().numpy()
    assert np.isfinite(got).all()
    # P and O are rounded to 8 (bf16) or 11 (fp16) bits, half a unit each: 2^-9 and 2^-12 of the result, twice, and O is
    # an average of N(0, 1) values, below 5 in magnitude
    eps = 2.0 ** -9 if dtype == "bf16" else 2.0 ** -12
    assert npo.rel_l2(got, want) <= 2 * eps
    assert npo.max_abs(got, want) <= 2 * 5 * eps


@pytest.mark.parametrize("B,H,L1,L2,D,dtype", [
    # one and an odd number of 64-key blocks, their edges; L1 around groups of two and four, one wave and more
    (1, 1, 1, 64, 32, "bf16"), (1, 2, 5, 63, 32, "fp16"), (4, 8, 19, 64, 32, "bf16"), (2, 16, 21, 40, 64, "fp16"),
    (1, 2, 3, 129, 32, "bf16"), (2, 8, 22, 192, 32, "fp16"), (1, 1, 6, 191, 64, "bf16"), (2, 8, 21, 160, 64, "bf16"),
    (1, 4, 66, 320, 32, "bf16"), (1, 4, 66, 448, 64, "bf16"), (1, 2, 9, 576, 64, "fp16"),
    # an even number: four rows at D = 32, two where all CTAs fit in one wave and at D = 64
    (2, 8, 38, 128, 32, "bf16"), (1, 8, 8, 512, 32, "bf16"), (2, 8, 39, 256, 32, "fp16"), (1, 4, 67, 250, 64, "bf16"),
    (1, 4, 37, 65, 32, "bf16"), (1, 16, 41, 193, 32, "fp16"),
])
def test_edges_of_tiles_and_groups(B, H, L1, L2, D, dtype):
    q, k, v, bias = _inputs(B, H, L1, L2, D, dtype)
    o = fta.attention(q.cuda(), k.cuda(), v.cuda(), bias.cuda(), D ** -0.5)
    _check(o, q, k, v, bias, D ** -0.5, dtype)


@pytest.mark.parametrize("L2,D", [(64, 32), (192, 64), (256, 32), (320, 32)])
def test_masked_rows_and_blocks(L2, D):
    """Query rows whose bias is the type's lowest value or -1e9 throughout (uniform), key blocks masked from their
    first key (the running maximum starts at -inf), and a negative scale."""
    q, k, v, bias = _inputs(1, 2, 6, L2, D, "bf16")
    bias[:, 0, 3] = -1.0e9
    bias[:, 1, 5] = torch.finfo(torch.bfloat16).min
    bias[:, :, 7, :L2 // 2] = float("-inf")
    for scale in (D ** -0.5, -0.3):
        o = fta.attention(q.cuda(), k.cuda(), v.cuda(), bias.cuda(), scale)
        _check(o, q, k, v, bias, scale, "bf16")
    bias[:, :, 9] = float("-inf")  # no key at all: zeros
    o = fta.attention(q.cuda(), k.cuda(), v.cuda(), bias.cuda(), D ** -0.5)
    assert (o[:, :, :, 9] == 0).all() and torch.isfinite(o).all()
