"""Host-side logic that needs no GPU: the autograd boundary's argument checks, the workload
generator, and the L1 sharding scheme (with a 2-rank gloo group standing in for NCCL)."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import flash_tt_attn as fta
import workloads
from oracle import tt_attn_oracle as npo

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_attention_asserts_like_the_reference():
    q = torch.zeros(1, 1, 2, 128, 32, dtype=torch.float16)
    b = torch.zeros(1, 1, 128, 128, dtype=torch.float16)
    with pytest.raises(AssertionError):          # dtype mismatch (flash_tt_attn.py:561)
        fta.attention(q, q, q, b.float(), 1.0)
    with pytest.raises(AssertionError):          # head-dim mismatch (flash_tt_attn.py:559)
        fta.attention(q, q[..., :16], q, b, 1.0)
    with pytest.raises(AssertionError):          # no CPU path
        fta.attention(q, q, q, b, 1.0)
    with pytest.raises(AssertionError):
        fta.attention(q.float(), q.float(), q.float(), b.float(), 1.0)


def test_shard_rows_partition():
    for L1, world in [(768, 8), (384, 4), (10, 4), (3, 8), (1024, 2)]:
        seen = []
        for r in range(world):
            s = fta.shard_rows(L1, r, world)
            seen.extend(range(s.start, s.stop))
        assert seen == list(range(L1))


def test_workloads_are_seeded_and_masked():
    w = workloads.WORKLOADS["c3_crop_l384"].with_rows(4)
    a, b = workloads.make_inputs(w), workloads.make_inputs(w)
    for k in ("q", "k", "v", "do", "bias"):
        assert np.array_equal(a[k], b[k])
    masked = a["mask"][0, 0, 0]
    assert 10 < masked.sum() < 80 and not masked[0]
    assert np.all(a["bias"][0, :, :, masked] < -1e8)
    ns = workloads.WORKLOADS["ns_l768"]
    assert ns.flops_fwd() == 4.0 * 4 * 768 ** 3 * 32
    assert abs(ns.flops_fwd() + ns.flops_bwd() - 811.75e9) < 0.01e9


def test_reference_tt_attn_matches_oracle():
    w = workloads.Workload("t", 1, 2, 3, 128, 32, "fp32", 5)
    x = workloads.make_inputs(w)
    o = fta.reference_tt_attn(*(torch.from_numpy(x[k]) for k in ("q", "k", "v", "bias")), w.sm_scale)
    ref = npo.forward(x["q"], x["k"], x["v"], x["bias"], w.sm_scale)
    np.testing.assert_allclose(o.numpy(), ref, atol=2e-5, rtol=1e-4)


_WORKER = r"""
import os, sys
sys.path.insert(0, {root!r}); sys.path.insert(0, os.path.join({root!r}, "flash-triangle-attention_b200"))
import numpy as np, torch, torch.distributed as dist
import flash_tt_attn as fta, workloads
from oracle import tt_attn_oracle as npo
dist.init_process_group("gloo", init_method="tcp://127.0.0.1:{port}", rank=int(sys.argv[1]), world_size=2)
rank = dist.get_rank()
w = workloads.Workload("t", 1, 2, 6, 128, 32, "fp32", 9)
rows = fta.shard_rows(w.L1, rank, 2)
x = workloads.make_inputs(w, rows)          # this rank's shard of the L1 rows; bias replicated
part = npo.forward_backward(x["q"], x["k"], x["v"], x["bias"], x["do"], w.sm_scale)
db = torch.from_numpy(part["dbias"].copy())
dist.all_reduce(db)                          # the path's only collective: sum of partial dBias
full = workloads.make_inputs(w)
ref = npo.forward_backward(full["q"], full["k"], full["v"], full["bias"], full["do"], w.sm_scale)
assert np.allclose(db.numpy(), ref["dbias"], atol=1e-4), "dbias"
for k in ("o", "dq", "dk", "dv"):
    assert np.allclose(part[k], ref[k][:, :, rows], atol=1e-5), k
dist.destroy_process_group()
print("rank", rank, "ok")
"""


def test_sharded_rows_with_gloo_allreduce(tmp_path):
    """Two CPU ranks: rows sharded, bias replicated, float32 dBias all-reduced (the scheme the
    GPU path runs over NCCL), checked against the unsharded oracle."""
    script = tmp_path / "worker.py"
    script.write_text(_WORKER.format(root=ROOT, port=29000 + os.getpid() % 2000))
    procs = [subprocess.Popen([sys.executable, str(script), str(r)], stdout=subprocess.PIPE,
                              stderr=subprocess.STDOUT, text=True) for r in range(2)]
    outs = [p.communicate(timeout=120)[0] for p in procs]
    for p, out in zip(procs, outs):
        assert p.returncode == 0, out


def test_shard_plan_covers_every_head_and_row_once():
    """Heads first, rows second: every (head, row) belongs to exactly one rank; ranks that share a
    head are consecutive and form one all-reduce group; different heads never share a group."""
    import numpy as np
    for H, L1, world in [(4, 768, 1), (4, 768, 2), (4, 768, 4), (4, 768, 8), (8, 2048, 8), (3, 10, 4), (2, 5, 8)]:
        cover = np.zeros((H, L1), dtype=np.int32)
        groups = {}
        for rank in range(world):
            heads, rows, peers = fta.shard_plan(H, L1, rank, world)
            cover[heads, rows] += 1
            assert rank in peers and peers == list(range(peers[0], peers[0] + len(peers)))
            groups.setdefault((heads.start, heads.stop), set()).add(tuple(peers))
        assert (cover == 1).all(), (H, L1, world)
        assert all(len(g) == 1 for g in groups.values())


def test_streamed_workspace_serves_every_block():
    """One workspace for blocks of several heights: the need does not grow with the rows, since a short block may be
    split over more dBias planes than a long one."""
    import _cabi
    not_the_largest = 0
    for B, H, L1, L2, D in [(1, 1, 256, 256, 64), (1, 4, 576, 576, 32), (1, 4, 512, 512, 64), (1, 4, 640, 640, 32),
                            (2, 4, 320, 64, 32), (1, 4, 768, 768, 32), (1, 2, 97, 136, 64), (1, 1, 5, 8, 32)]:
        sizes = fta._block_sizes(L1, 96)
        assert sum(sizes) == L1
        have = fta._blocks_workspace_bytes(B, H, L2, D, _cabi.FTA_BF16, sizes)
        need = {n: _cabi.lib().fta_bwd_workspace_bytes(_cabi.FtaProblem(B, H, n, L2, D, _cabi.FTA_BF16)) for n in sizes}
        assert 0 < max(need.values()) <= have
        not_the_largest += need[max(sizes)] < have
    assert not_the_largest >= 2  # the case this is about is among them


class _FakeNative:
    def __init__(self):
        self.calls = []

    def set_status(self, index, word, mirror):
        assert isinstance(index, int)
        self.calls.append((index, word, mirror))


@pytest.fixture
def fake_device(monkeypatch):
    """The status bookkeeping with CPU tensors in the place of a device's."""
    class FakeStatus(fta._Status):
        def __init__(self, device):
            self.word, self.mirror = torch.zeros(1, dtype=torch.int32), torch.zeros(1, dtype=torch.int32)

    native = _FakeNative()
    monkeypatch.setattr(fta, "_native", lambda: native)
    monkeypatch.setattr(fta, "_Status", FakeStatus)
    monkeypatch.setattr(fta, "_status_words", {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    return native


def test_a_device_without_an_index_is_the_current_one(fake_device):
    """The word that attention() registers for cuda:3 is the one that "cuda" names while device 3 is current."""
    st = fta._status_of(torch.device("cuda", 3))
    assert fta._status_of(torch.device("cuda")) is st and fta._status_of("cuda") is st
    assert [c[0] for c in fake_device.calls] == [3]
    fta.check_device_status("cuda")
    st.word.fill_(0x1042)
    with pytest.raises(RuntimeError, match="0x1042"):
        fta.check_device_status("cuda")
    fta.check_device_status()


def test_a_status_word_is_kept_only_once_it_is_registered(fake_device, monkeypatch):
    def fails(*a):
        raise RuntimeError("not registered")
    monkeypatch.setattr(fake_device, "set_status", fails)
    with pytest.raises(RuntimeError, match="not registered"):
        fta._status_of("cuda")
    assert not fta._status_words


def test_threads_that_meet_a_device_together_share_one_status_word(fake_device, monkeypatch):
    """A second word for the device would replace the first, which kernels of the other thread still write to."""
    import threading
    import time
    slow = fta._Status

    class SlowStatus(slow):
        def __init__(self, device):
            time.sleep(0.05)  # as an allocation does, this lets the other threads in
            super().__init__(device)

    monkeypatch.setattr(fta, "_Status", SlowStatus)
    got, start = [], threading.Barrier(8)

    def meet():
        start.wait()
        got.append(fta._status_of("cuda"))

    threads = [threading.Thread(target=meet) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 8 and all(st is got[0] for st in got) and len(fake_device.calls) == 1


_LAST_DBIAS = r"""
import os, sys, threading, weakref
sys.path.insert(0, {root!r}); sys.path.insert(0, os.path.join({root!r}, "flash-triangle-attention_b200"))
import torch
import flash_tt_attn as fta
ext = fta._native()
seen = []

def hold():  # a tensor whose Python side is finalised when the library lets go of it
    t = torch.zeros(3)
    weakref.finalize(t, lambda: seen.append(fta.last_dbias_f32().numel()))
    ext.set_last_dbias_f32(t)

for n in range(3):
    hold()
assert len(seen) == 2, seen
stop = []

def look():
    while not stop:
        fta.last_dbias_f32()

threads = [threading.Thread(target=look) for _ in range(3)]
for t in threads:
    t.start()
for n in range(300):
    hold()
stop.append(1)
for t in threads:
    t.join()
print("through", flush=True)
"""


def test_last_dbias_lets_go_of_the_old_tensor_outside_its_lock(tmp_path):
    """Letting go of a tensor that Python has seen runs the interpreter (its lock, its finalisers). Under the lock
    of ``last_dbias_f32()`` that is a deadlock with whoever holds the interpreter and waits for that lock; here a
    finaliser asks for it. In a process of its own, which ends by itself unless it is stuck."""
    script = tmp_path / "last_dbias.py"
    script.write_text(_LAST_DBIAS.format(root=ROOT))
    r = subprocess.run([sys.executable, str(script)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                       timeout=120)
    assert r.returncode == 0 and "through" in r.stdout, r.stdout
