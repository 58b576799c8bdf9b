"""The wait for the stream that fills device buffers: one event per context records that stream, so the record, the
wait and the call it is for have to be one step with respect to other threads of the same context.  Checked on the
host with a library that only notes its calls (no GPU): every method makes the wait under the context's lock, and
another thread's wait cannot come between a thread's wait and its call."""
import ctypes
import threading
import types

import numpy as np
import pytest
import torch

import fmma_b200


class FakeLibrary:
    """Notes (function, first argument, whether the calling thread holds the lock); every call succeeds."""

    def __init__(self, lock):
        self.lock, self.calls, self.on_call = lock, [], None

    def __getattr__(self, name):
        if not name.startswith("fmma_"):
            raise AttributeError(name)

        def call(*args):
            if name in ("fmma_ctx_destroy", "fmma_plan_destroy"):
                return 0
            self.calls.append((name, args[0], self.lock._is_owned(), threading.current_thread().name))
            if self.on_call:
                self.on_call(name)
            return 0
        return call


@pytest.fixture
def fake(monkeypatch):
    """A context on the fake library; CPU tensors pass for device memory."""
    ctx = fmma_b200.Context.__new__(fmma_b200.Context)
    ctx.lock, ctx.device, ctx.kernel = threading.RLock(), 0, ("inv_r", 0.0)
    ctx._h = ctypes.c_void_p(11)
    ctx._L = FakeLibrary(ctx.lock)
    monkeypatch.setattr(fmma_b200, "_torch", types.SimpleNamespace(
        Tensor=torch.Tensor, float64=torch.float64, float32=torch.float32,
        cuda=types.SimpleNamespace(current_stream=lambda device: types.SimpleNamespace(cuda_stream=7))))
    monkeypatch.setattr(fmma_b200, "_mem_kind", lambda *a: fmma_b200._lib.MEM_DEVICE)
    yield ctx
    ctx._h = ctypes.c_void_p(0)


def _tensors(n=6, d=3):
    g = torch.Generator().manual_seed(1)
    return tuple(torch.rand(s, generator=g, dtype=torch.float64) for s in ((n, d), (n, d), (n,)))


T, S, W = _tensors()
OFF = np.array([0, 6])
CALLS = {
    "fmma_solve_d": lambda c: c.solve(T, S, W),
    "fmma_solve_grad_d": lambda c: c.solve_grad(T, S, W),
    "fmma_forest_depths_d": lambda c: c.forest_depths(T, OFF, S, OFF, 4),
    "fmma_forest_solve_d": lambda c: c.forest_solve(T, OFF, S, OFF, W, [3]),
    "fmma_exact_rows_d": lambda c: c.exact_rows([0, 1], T, S, W),
    "fmma_cheb_fit_d": lambda c: c.cheb_fit(torch.rand(16, dtype=torch.float64), 2, 3),
    "fmma_cheb_eval_d": lambda c: c.cheb_eval(torch.rand(16, dtype=torch.float64), T[:, :2].contiguous(), 3),
    "fmma_max_leaf_occupancy_d": lambda c: c.max_leaf_occupancy(T, S, 3),
    "fmma_plan_create_d": lambda c: c.plan(T, OFF, S, OFF, 1, [3]),
}


@pytest.mark.parametrize("entry", sorted(CALLS))
def test_wait_and_call_are_made_under_the_lock(fake, entry):
    CALLS[entry](fake)
    names = [c[0] for c in fake._L.calls]
    assert names.count("fmma_wait_stream") == 1 and names.index("fmma_wait_stream") == names.index(entry) - 1
    assert all(held for name, _, held, _ in fake._L.calls if name in ("fmma_wait_stream", entry))


def test_plan_waits_on_its_own_stream(fake, monkeypatch):
    # a replay copies the weights on the plan's stream: the wait has to be that stream's, under the plan's lock
    plan = fake.plan(T, OFF, S, OFF, 1, [3])
    plan._h = ctypes.c_void_p(22)

    class DeviceView(fmma_b200._Arr):
        def __init__(self, *a):
            super().__init__(*a)
            self.kind = fmma_b200._lib.MEM_DEVICE
    monkeypatch.setattr(fmma_b200, "_Arr", DeviceView)
    fake._L.calls.clear()
    held = []
    fake._L.on_call = lambda name: held.append(plan._lock._is_owned())
    plan.execute(W, torch.empty(6, dtype=torch.float64))
    assert [(name, h.value) for name, h, _, _ in fake._L.calls] == [("fmma_plan_wait_stream", 22),
                                                                   ("fmma_plan_execute_d", 22)]
    assert held == [True, True]
    plan._h = ctypes.c_void_p(0)


@pytest.mark.gpu
def test_device_buffers_written_late_are_waited_for():
    # points, then weights, appear on torch's stream only after a pause in front of their copies
    r = np.random.default_rng(1)
    t, s = (torch.from_numpy(r.random((4000, 3))) for _ in range(2))
    w1, w2 = (torch.from_numpy(r.standard_normal(4000)) for _ in range(2))
    ctx = fmma_b200.Context()
    ctx.set_kernel("inv_r_safe")
    off = [0, 4000]
    plan = ctx.plan(t.cuda(), off, s.cuda(), off, 1, [4])
    want = [plan.execute(w.cuda()).cpu() for w in (w1, w2)]
    plan.close()
    td, sd, wd = (x.pin_memory().cuda() * 0 for x in (t, s, w1))
    torch.cuda.synchronize()

    def late(dst, src):
        torch.cuda._sleep(40_000_000)  # about 20 ms of SM clocks
        dst.copy_(src.pin_memory(), non_blocking=True)
    with torch.cuda.stream(torch.cuda.Stream()):
        late(td, t)
        sd.copy_(s.pin_memory(), non_blocking=True)
        plan = ctx.plan(td, off, sd, off, 1, [4])
        for w, ref in ((w1, want[0]), (w2, want[1])):
            late(wd, w)
            assert torch.equal(plan.execute(wd).cpu(), ref)
        late(wd, w1)
        a = ctx.solve(td, sd, wd, poly_ord=4, depth=4)[0].cpu()
        late(wd, w2)
        b = ctx.solve(td, sd, wd, poly_ord=4, depth=4)[0].cpu()
    plan.close()
    assert torch.equal(a, want[0]) and torch.equal(b, want[1])


def test_other_threads_wait_stays_outside(fake):
    # the first thread stops inside its wait until the second one has had time to make its own
    inside, second = threading.Event(), threading.Event()

    def on_call(name):
        if name == "fmma_wait_stream" and threading.current_thread().name == "first":
            inside.set()
            second.wait(0.3)  # runs out when the second thread is held back
    fake._L.on_call = on_call

    def other():
        inside.wait(5)
        fake.solve(T, S, W)
        second.set()
    threads = [threading.Thread(target=lambda: fake.solve(T, S, W), name="first"),
               threading.Thread(target=other, name="second")]
    for t in threads:
        t.start()
    for t in threads:
        t.join(10)
    order = [(who, name) for name, _, _, who in fake._L.calls]
    assert order == [("first", "fmma_wait_stream"), ("first", "fmma_solve_d"),
                     ("second", "fmma_wait_stream"), ("second", "fmma_solve_d")]
