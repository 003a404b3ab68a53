"""Calls from several Python threads: nothing of a call that waits for the GPU keeps other threads from running, and calls of two
threads on one stream do not share their scratch while they use it."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ssd(gen, s, h=4, act=torch.float32):
    n = lambda *z: torch.randn(*z, generator=gen, device="cuda")
    return dict(x=n(2, s, h, 64).to(act), dt=0.05 + 0.01 * n(2, s, h), a=-1.0 - n(h).abs(), b=n(2, s, 1, 128).to(act), c=n(2, s, 1, 128).to(act))


def _beats_during(wait):
    """How often another thread got to run while `wait()` waited for the GPU."""
    beats, stop = [0], threading.Event()

    def beat():
        while not stop.is_set():
            beats[0] += 1
            time.sleep(0.002)

    t = threading.Thread(target=beat)
    t.start()
    time.sleep(0.02)
    before, t0 = beats[0], time.perf_counter()
    wait()
    took, n = time.perf_counter() - t0, beats[0] - before
    stop.set()
    t.join()
    return n, took


@pytest.mark.parametrize("what", ["last_workspace_status", "ssd2_fwd", "ssd2_bwd"])
def test_a_call_that_waits_for_the_gpu_lets_other_threads_run(bm, what):
    gen = torch.Generator(device="cuda").manual_seed(3)
    k = _ssd(gen, 256, act=torch.bfloat16)
    bm.ops.ssd2_fwd(**k)
    dy = torch.ones_like(k["x"])
    calls = dict(last_workspace_status=bm.ops.last_workspace_status, ssd2_fwd=lambda: bm.ops.ssd2_fwd(**k, check_status=True),
                 ssd2_bwd=lambda: bm.ops.ssd2_bwd(**k, d=None, h0=None, dy=dy, check_status=True))
    calls[what]()
    torch.cuda.synchronize()
    torch.cuda._sleep(700_000_000)   # 0.3 s and more at any clock of the part
    n, took = _beats_during(calls[what])
    assert took > 0.2 and n > 0.2 * took / 0.002, (n, took)


@pytest.mark.parametrize("entry", ["workspace", "noalloc"])
def test_two_threads_on_one_stream(bm, entry):
    """float32: three kernels per call that hand chunk states on through the stream's workspace, or the built-in array."""
    gens = [torch.Generator(device="cuda").manual_seed(s) for s in (1, 2)]
    ks = [_ssd(g, s) for g, s in zip(gens, (300, 500))]
    call = (lambda **k: bm.ops.ssd2_fwd(**k, path="exact")) if entry == "workspace" else bm.ops.ssd2_fwd_noalloc
    want = [call(**k) for k in ks]
    wrong, start = [], threading.Barrier(2)

    def work(i):
        start.wait()
        for _ in range(1500):
            y, h = call(**ks[i])
            if not (torch.equal(y, want[i][0]) and torch.equal(h, want[i][1])):
                wrong.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
