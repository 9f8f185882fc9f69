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



@pytest.mark.parametrize("route", ["attention", "forward_pass", "backward_pass"])
def test_other_threads_run_while_a_pass_waits_in_native_code(route):
    """Behind a kernel of half a second the launch queue fills up and a launch waits for room. Meanwhile a second
    thread must have the interpreter: its longest pause is a fraction of that wait."""
    import threading
    import time
    ext = fta._native()
    q, k, v, b = _inputs()
    fta.attention(q, k, v, b, 0.2)
    state = ext.forward_pass(q, k, v, b, 0.2, None)
    dout = torch.ones_like(q)
    call = {"attention": lambda: fta.attention(q, k, v, b, 0.2),
            "forward_pass": lambda: ext.forward_pass(q, k, v, b, 0.2, None),
            "backward_pass": lambda: ext.backward_pass(*state, dout, 0.2, True)}[route]
    call()
    torch.cuda.synchronize()
    pause, waiting, stop = [0.0], [], []

    def other():
        last = time.perf_counter()
        while not stop:
            time.sleep(0.001)
            now = time.perf_counter()
            if waiting:
                pause[0] = max(pause[0], now - last)
            last = now

    thread = threading.Thread(target=other)
    thread.start()
    try:
        time.sleep(0.05)
        waiting.append(1)
        torch.cuda._sleep(1_000_000_000)  # cycles: about half a second
        longest = 0.0
        for _ in range(2000):
            t = time.perf_counter()
            call()
            longest = max(longest, time.perf_counter() - t)
        time.sleep(0.01)
    finally:
        stop.append(1)
        thread.join()
    fta.check_device_status()
    if longest < 0.1:
        pytest.skip(f"no launch had to wait (longest call {longest * 1e3:.1f} ms)")
    assert pause[0] < 0.5 * longest, (pause[0], longest)


def _train():
    q, k, v, b = _inputs()
    q.requires_grad_()
    return fta.attention(q, k, v, b, 0.2)


def test_debug_mode_checks_the_backward_pass(monkeypatch):
    """With FTA_DEBUG=1 a failure shows in the pass it happens in (the word is set by hand, as a wait that runs out
    would)."""
    monkeypatch.setattr(fta, "_DEBUG", True)
    o = _train()
    fta._status_of(o.device).word.fill_(0x1046)
    with pytest.raises(RuntimeError, match="0x1046"):
        o.sum().backward()
    _train().sum().backward()
    fta.check_device_status()


def test_a_failure_in_a_backward_pass_raises_in_the_next_one_without_a_sync():
    """The last kernel of a backward pass mirrors the word; the next backward pass looks at the mirror on the autograd
    thread before it launches anything."""
    first, second, third = _train(), _train(), _train()
    fta._status_of(first.device).word.fill_(0x1047)
    first.sum().backward()  # its last kernel mirrors the word
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="0x1047"):
        second.sum().backward()
    third.sum().backward()  # cleared when it was reported
    fta.check_device_status()


def test_a_refused_call_does_not_fail_the_next_one():
    """The runtime refuses to wait for a stream that is being captured, on the host. That error belongs to that call
    alone: launches learn how they went from the runtime's last error."""
    import ctypes
    import _cabi
    L = _cabi.lib()
    rt = ctypes.CDLL("libcudart.so.12")  # torch's; a stream means the same to every runtime of the process
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    x = torch.ones(64, device="cuda")
    y = torch.zeros(64, device="cuda", dtype=torch.bfloat16)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    handle, code, graph = ctypes.c_void_p(side.cuda_stream), ctypes.c_int32(0), ctypes.c_void_p()
    relaxed = 2
    assert rt.cudaStreamBeginCapture(handle, relaxed) == 0
    try:
        assert L.fta_read_status(status.data_ptr(), ctypes.byref(code), side.cuda_stream) == -9  # FTA_ERR_CUDA
        refused = L.fta_last_cuda_error()
    finally:
        rt.cudaStreamEndCapture(handle, ctypes.byref(graph))  # says that the capture came to nothing
        rt.cudaGetLastError()
    assert refused != 0
    st = torch.cuda.current_stream().cuda_stream
    assert L.fta_dbias_cast(x.data_ptr(), y.data_ptr(), 64, _cabi.FTA_BF16, st) == 0
    assert float(y.sum()) == 64.0 and L.fta_last_cuda_error() == refused


def test_a_streamed_call_that_raises_leaves_no_copy_in_flight(monkeypatch):
    """The device buffers of the call die with it: copies on its own streams must not outlive them, and the caller's
    host tensors are the caller's again."""
    host = {n: torch.randn(1, 4, 288, 512, 64).bfloat16().pin_memory() for n in ("q", "k", "v", "do")}
    host["bias"] = torch.randn(1, 4, 512, 512).bfloat16().pin_memory()
    out = {n: torch.empty_like(host["q"]).pin_memory() for n in ("o", "dq", "dk", "dv")}
    out["dbias"] = torch.empty_like(host["bias"]).pin_memory()
    fta.attention_fwd_bwd_streamed(host, 0.2, out)
    want = out["o"].clone()
    with monkeypatch.context() as m:
        m.setattr(fta, "_blocks_workspace_bytes", lambda *a: 256)  # refused on the host by the first fta_backward
        with pytest.raises(fta._cabi.FtaError):
            fta.attention_fwd_bwd_streamed(host, 0.2, out)
        streams = fta._copy_streams["cuda", torch.cuda.current_device()]
        assert all(s.query() for s in (*streams, torch.cuda.current_stream()))
    fta.attention_fwd_bwd_streamed(host, 0.2, out)
    assert torch.equal(out["o"], want)
