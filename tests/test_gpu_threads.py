"""The operators beside other Python threads."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_other_threads_run_while_a_launch_waits():
    """A call whose launch waits for room in the queue (here behind 1.5 s of work) does not hold the interpreter lock."""
    from xattn_b200 import check_device_status, ops
    q, k, v = (torch.randn(1, h, n, 128, device=DEV).bfloat16() for h, n in ((4, 1), (2, 300), (2, 300)))
    want = ops.decode_attention(q, k, v)
    torch.cuda.synchronize()
    ticks, done = [], threading.Event()

    def tick():
        while not done.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.002)

    other = threading.Thread(target=tick)
    other.start()
    try:
        torch.cuda._sleep(int(1.5 * 1.9e9))
        start = time.perf_counter()
        for _ in range(6000):
            out = ops.decode_attention(q, k, v)
        waited = time.perf_counter() - start
        torch.cuda.synchronize()
    finally:
        done.set()
        other.join()
    check_device_status()
    assert torch.equal(out, want)
    assert waited > 0.5, "no launch waited: the queue holds more than the test assumes"
    assert max(b - a for a, b in zip(ticks, ticks[1:])) < 0.5 * waited


def test_calls_from_several_threads():
    """Each thread on a stream of its own, all kinds of calls at once: the results of one thread alone."""
    from xattn_b200 import api, check_device_status, ops
    inputs = []
    for i, n in enumerate((300, 1003, 2048, 4100)):
        g = torch.Generator(device=DEV).manual_seed(i)
        inputs.append([torch.randn(1, h, n, 128, device=DEV, generator=g).bfloat16() for h in (4, 2, 2)])

    def calls(q, k, v):
        return (api.Xattention_prefill(q, k, v, 16), api.xattn_estimate(q, k, 128, 16)[1], ops.decode_attention(q[:, :, -1:], k, v),
                api.Xattention_prefill(q.float(), k.float(), v.float(), 8))

    want = [calls(*x) for x in inputs]
    torch.cuda.synchronize()
    got, errors = [None] * len(inputs), []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    got[i] = calls(*inputs[i])
                torch.cuda.current_stream().synchronize()
        except Exception as e:                       # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(inputs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    check_device_status()
    assert not errors, errors
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            assert torch.equal(x, y)
