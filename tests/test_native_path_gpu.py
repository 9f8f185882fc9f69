"""The native call path of ``attention()`` where it branches: with and without a backward pass to come, any L2,
small and unequal shares of rows."""
import numpy as np
import pytest
import torch

import flash_tt_attn as fta
from oracle import tt_attn_oracle as npo

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


@pytest.mark.parametrize("B,H,L1,L2,D,dtype,masked", [
    (1, 1, 1, 1, 32, "fp16", False), (2, 1, 3, 7, 32, "bf16", True), (1, 2, 4, 33, 64, "fp16", False),
    (1, 2, 7, 127, 32, "bf16", True), (2, 1, 5, 129, 32, "fp16", True), (1, 1, 9, 317, 64, "bf16", False),
    (1, 1, 67, 261, 32, "bf16", True), (1, 1, 150, 130, 64, "fp16", False), (1, 3, 70, 12, 32, "bf16", False),
])
def test_any_l2_with_and_without_a_mask(B, H, L1, L2, D, dtype, masked):
    """L2 of any size: rows of the bias and of dBias that start at any alignment, padded planes, last blocks of
    every length; up to 64 dBias planes, row groups that do not come out even."""
    dt = {"fp16": torch.float16, "bf16": torch.bfloat16}[dtype]
    g = torch.Generator().manual_seed(L1 * 1000 + L2)
    q, k, v, do = (torch.randn(B, H, L1, L2, D, generator=g).to(dt) for _ in range(4))
    bias = torch.randn(B, H, L2, L2, generator=g).to(dt)
    mask = None
    if masked:
        mask = torch.rand(B, L2, generator=g) > 0.2
        mask[:, 0] = True
    leaves = [a.cuda().requires_grad_(True) for a in (q, k, v, bias)]
    o = fta.attention(*leaves, D ** -0.5, key_mask=None if mask is None else mask.cuda())
    o.backward(do.cuda())
    fta.check_device_status()
    bm = bias.float()
    if mask is not None:
        bm = torch.where(mask[:, None, None, :], bm, torch.tensor(-1.0e9))
    ref = npo.forward_backward(q.float().numpy(), k.float().numpy(), v.float().numpy(), bm.numpy(), do.float().numpy(), D ** -0.5)
    got = {"o": o, "dq": leaves[0].grad, "dk": leaves[1].grad, "dv": leaves[2].grad, "dbias": fta.last_dbias_f32()}
    assert leaves[3].grad.shape == bias.shape and got["dbias"].shape == bias.shape
    for name, t in got.items():
        a = t.detach().float().cpu().numpy()
        assert np.isfinite(a).all(), name
        assert npo.max_abs(a, ref[name]) <= 2e-2, (name, npo.max_abs(a, ref[name]))
        if np.linalg.norm(ref[name]) > 1e-6:
            assert npo.rel_l2(a, ref[name]) <= 1e-2, (name, npo.rel_l2(a, ref[name]))
    want = got["dbias"].to(dt)
    assert torch.equal(leaves[3].grad, want)


@pytest.mark.parametrize("D,L1,L2", [(64, 6, 512), (64, 40, 256), (32, 7, 640)])
def test_backward_is_bit_reproducible_over_many_blocks(D, L1, L2):
    """Many flushes of the dBias boxes through few spare buffers: a box sent twice or too early shows as a
    difference between runs, or from the sum over two shares of the rows."""
    g = torch.Generator(device="cuda").manual_seed(D + L2)
    q, k, v, do = (torch.randn(1, 4, L1, L2, D, device="cuda", dtype=torch.bfloat16, generator=g) for _ in range(4))
    b = torch.randn(1, 4, L2, L2, device="cuda", dtype=torch.bfloat16, generator=g)

    def run(rows):
        t = [x[:, :, rows].contiguous().requires_grad_() for x in (q, k, v)]
        bb = b.clone().requires_grad_()
        o = fta.attention(*t, bb, 0.2)
        o.backward(do[:, :, rows].contiguous())
        return [o.detach(), t[1].grad, t[2].grad, fta.last_dbias_f32()]

    first = run(slice(0, L1))
    for _ in range(3):
        assert all(torch.equal(x, y) for x, y in zip(first, run(slice(0, L1))))
    parts = [run(slice(0, L1 // 2)), run(slice(L1 // 2, L1))]
    for i in range(3):
        assert torch.equal(torch.cat([p[i] for p in parts], dim=2), first[i])
    assert torch.allclose(parts[0][3] + parts[1][3], first[3], atol=1e-4, rtol=1e-5)
    fta.check_device_status()


@pytest.mark.parametrize("B,H,L1,L2,D", [(1, 1, 256, 256, 64), (1, 4, 300, 576, 32)])
def test_streamed_call_with_blocks_that_need_more_scratch_than_the_largest(B, H, L1, L2, D):
    """Default blocks, where a short block is split over more dBias planes than a full one: accepted, and equal to
    the call on device tensors (dQ and dBias: float32 sums whose order may differ)."""
    g = torch.Generator().manual_seed(L2)
    host = {n: torch.randn(B, H, L1, L2, D, generator=g).bfloat16().pin_memory() for n in ("q", "k", "v", "do")}
    host["bias"] = torch.randn(B, H, L2, L2, generator=g).bfloat16().pin_memory()
    out = {n: torch.full_like(host["q"], float("nan")).pin_memory() for n in ("o", "dq", "dk", "dv")}
    out["dbias"] = torch.empty_like(host["bias"]).pin_memory()
    fta.attention_fwd_bwd_streamed(host, 0.2, out)
    db32 = fta.last_dbias_f32().clone()
    leaves = [host[n].cuda().requires_grad_() for n in ("q", "k", "v", "bias")]
    o = fta.attention(*leaves, 0.2)
    o.backward(host["do"].cuda())
    fta.check_device_status()
    assert torch.equal(out["o"], o.detach().cpu())
    assert torch.equal(out["dk"], leaves[1].grad.cpu()) and torch.equal(out["dv"], leaves[2].grad.cpu())
    # one bf16 ulp of the largest value
    assert float((out["dq"].float() - leaves[0].grad.cpu().float()).abs().max()) <= float(out["dq"].float().abs().max()) * 2.0 ** -8
    ref = fta.last_dbias_f32()
    assert float((db32 - ref).abs().max()) <= 1e-4 * float(ref.abs().max()) + 1e-5


@pytest.mark.parametrize("L1,L2,D", [(3, 104, 32), (2, 128, 64), (4, 200, 32), (2, 264, 64)])
@pytest.mark.parametrize("layout", ["rows_exchanged", "padded"])
def test_outputs_of_any_strides_and_nothing_beside_them(L1, L2, D, layout):
    """Through the C ABI the caller lays out O and the gradients. With one key block dQ, and always dK and dV, leave
    through tensor maps made from those strides; the elements between and behind the rows keep what they held."""
    import _cabi
    from _cabi import FtaProblem, check, t4, t5
    B, H, dt = 2, 2, torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(L2)
    q, k, v, do = (torch.randn(B, H, L1, L2, D, device="cuda", dtype=dt, generator=g) for _ in range(4))
    b = torch.randn(B, H, L2, L2, device="cuda", dtype=dt, generator=g)
    leaves = [x.clone().requires_grad_() for x in (q, k, v, b)]
    want_o = fta.attention(*leaves, 0.2)
    want_o.backward(do)

    def out():
        if layout == "rows_exchanged":
            whole = torch.full((B, L2 + 1, H, L1 + 1, D + 8), 77.0, device="cuda", dtype=dt)
            return whole, whole[:, :L2, :, :L1, :D].permute(0, 2, 3, 1, 4)
        whole = torch.full((B, H, L1 + 1, L2 + 3, D + 8), 77.0, device="cuda", dtype=dt)
        return whole, whole[:, :, :L1, :L2, :D]

    outs = {n: out() for n in ("o", "dq", "dk", "dv")}
    view = {n: t5(x[1]) for n, x in outs.items()}
    L, prob, st = _cabi.lib(), FtaProblem(B, H, L1, L2, D, _cabi.FTA_BF16), torch.cuda.current_stream().cuda_stream
    pitch = (L2 + 127) // 128 * 128
    f32 = lambda *s: torch.empty(s, device="cuda")
    lse, delta, db32, status = f32(3, B, H, L1, pitch), f32(B, H, L1, pitch), f32(B, H, L2, L2), torch.zeros(1, dtype=torch.int32, device="cuda")
    bias = b
    if pitch != L2:
        bias = torch.empty(B, H, pitch, pitch, device="cuda", dtype=dt)
        check(L.fta_mask_bias(prob, t4(b), None, bias.data_ptr(), st), "fta_mask_bias")
    check(L.fta_forward(prob, t5(q), t5(k), t5(v), t4(bias), 0.2, view["o"], None, lse.data_ptr(), status.data_ptr(), st), "fta_forward")
    # without the rounding residual of O, which attention() adds to delta: dQ and dK agree within bf16
    check(L.fta_bwd_preprocess(prob, view["o"], None, t5(do), delta.data_ptr(), st), "fta_bwd_preprocess")
    ws = torch.empty(L.fta_bwd_workspace_bytes(prob), dtype=torch.uint8, device="cuda")
    check(L.fta_backward(prob, t5(q), t5(k), t5(v), t4(bias), t5(do), lse.data_ptr(), delta.data_ptr(), 0.2, view["dq"], view["dk"],
                         view["dv"], db32.data_ptr(), None, ws.data_ptr(), ws.numel(), status.data_ptr(), st), "fta_backward")
    torch.cuda.synchronize()
    assert int(status) == 0
    want = {"o": want_o.detach(), "dq": leaves[0].grad, "dk": leaves[1].grad, "dv": leaves[2].grad}
    for n, (whole, x) in outs.items():
        a, w = x.float().cpu().numpy(), want[n].float().cpu().numpy()
        assert npo.rel_l2(a, w) <= 1e-2, (n, npo.rel_l2(a, w))
        if n in ("o", "dv"):  # no delta in these
            assert np.array_equal(a, w), n
        untouched = torch.ones_like(whole, dtype=torch.bool)
        (untouched[:, :L2, :, :L1, :D] if layout == "rows_exchanged" else untouched[:, :, :L1, :L2, :D]).fill_(False)
        assert bool((whole[untouched] == 77.0).all()), n
