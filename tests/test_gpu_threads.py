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


def test_calls_under_stream_capture():
    """Every kind of call in one CUDA graph, behind a fill, a copy and a join with another stream: replays give the results of
    the calls made directly, on new inputs in the same memory."""
    from xattn_b200 import api, check_device_status, ops
    g = torch.Generator(device=DEV).manual_seed(3)
    q, k, v = (torch.randn(1, h, 2500, 128, device=DEV, generator=g).bfloat16() for h in (4, 2, 2))
    new = [torch.randn(x.shape, device=DEV, generator=g).bfloat16() for x in (q, k, v)]
    f = [x.float() for x in (q, k, v)]

    def calls():
        idx, cnt = ops.mask_to_lists(torch.ones(1, 4, 20, 20, dtype=torch.bool, device=DEV), 2500, 2500, True)
        return (api.Xattention_prefill(q, k, v, 16), *api.xattn_estimate(q, k, 128, 8), ops.decode_attention(q[:, :, -1:], k, v),
                api.Xattention_prefill(*f, 8), ops.block_sparse_attention(q, k, v, idx, cnt, True, use_workspace=True),
                ops.block_sparse_attention(q, k, v, idx, cnt, False, use_workspace=True), ops.block_sparse_attention(q, k, v, None, None))

    calls()                                          # (everything that is asked once per kernel and device)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph):
        zero = torch.zeros(1000, device=DEV)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            aside = ops.decode_attention(q[:, :, :1], k, v)
        for x, y in zip(f, (q, k, v)):
            x.copy_(y)
        torch.cuda.current_stream().wait_stream(side)
        got = calls()
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip((aside, *got), (ops.decode_attention(q[:, :, :1], k, v), *calls())):
            assert torch.equal(a, b)
        for x, y in zip((q, k, v), new):
            x.copy_(y)
    assert not zero.any()
    check_device_status()
