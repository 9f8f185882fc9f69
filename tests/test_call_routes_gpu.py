"""Ways of calling ``attention()`` in which the launches are not seen by the caller's machinery: what cannot be done
is refused, nothing is answered from memory that no kernel has written."""
import pytest
import torch

import flash_tt_attn as fta

pytestmark = pytest.mark.gpu


def _inputs(L2=128, dtype=torch.float16, L1=2, D=32):
    g = torch.Generator(device="cuda").manual_seed(L2)
    r = lambda *s: torch.randn(s, device="cuda", dtype=dtype, generator=g)
    return [r(1, 1, L1, L2, D) for _ in range(3)] + [r(1, 1, L2, L2)]


@pytest.mark.parametrize("grad", [False, True])
def test_jit_trace_is_refused(grad):
    q, k, v, b = _inputs()
    q.requires_grad_(grad)
    with pytest.raises(AssertionError, match="torch.jit.trace"):
        torch.jit.trace(lambda *a: fta.attention(*a, 0.2), (q, k, v, b), check_trace=False)
    assert torch.isfinite(fta.attention(q, k, v, b, 0.2)).all()  # the tracer is gone again
    fta.check_device_status()


@pytest.mark.parametrize("which", range(4))
@pytest.mark.parametrize("mode", ["no_leaf", "leaf", "no_grad"])
def test_forward_mode_tangents_are_refused_not_dropped(which, mode):
    import torch.autograd.forward_ad as fwad
    t = _inputs()
    if mode == "leaf":
        t[0].requires_grad_()
    with fwad.dual_level(), torch.set_grad_enabled(mode != "no_grad"):
        args = list(t)
        args[which] = fwad.make_dual(t[which], torch.ones_like(t[which]))
        with pytest.raises((RuntimeError, NotImplementedError), match="jvp"):
            fta.attention(*args, 0.2)
        assert torch.isfinite(fta.attention(*t, 0.2)).all()  # no tangent, no objection
    fta.check_device_status()


def test_device_cuda_names_the_word_the_kernels_write():
    q, k, v, b = _inputs()
    fta.attention(q, k, v, b, 0.2)
    fta.check_device_status("cuda")
    host = {n: torch.randn(1, 1, 5, 128, 32).bfloat16().pin_memory() for n in ("q", "k", "v", "do")}
    host["bias"] = torch.randn(1, 1, 128, 128).bfloat16().pin_memory()
    out = {n: torch.empty_like(host["q"]).pin_memory() for n in ("o", "dq", "dk", "dv")}
    out["dbias"] = torch.empty_like(host["bias"]).pin_memory()
    fta.attention_fwd_bwd_streamed(host, 0.2, out, device="cuda")
    fta._status_of(q.device).word.fill_(0x1042)
    with pytest.raises(RuntimeError, match="0x1042"):
        fta.check_device_status("cuda")
    fta.check_device_status("cuda")
