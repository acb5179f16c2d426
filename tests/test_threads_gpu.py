"""Host threads that call the same entry point with different sizes at the same time."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

REPS = 300


def _nvfp4(lib, dev, k):
    rows = 16
    g = torch.Generator(device=dev).manual_seed(k)

    def codes(*shape):
        return torch.randint(0, 256, shape, dtype=torch.uint8, device=dev, generator=g)

    act, w, y = codes(1, k // 2), codes(rows, k // 2), torch.zeros((rows,), device=dev)
    acts, ws = (torch.randint(0x30, 0x40, (n, k // 16), dtype=torch.uint8, device=dev, generator=g) for n in (1, rows))
    return (lambda s: lib.raw("gemb_nvfp4_gemv", act, acts, w, ws, y, rows, k, 100.0, 100.0, s)), y


def _fp8(lib, dev, k):
    rows = 16
    g = torch.Generator(device=dev).manual_seed(k)
    act, w = (torch.randint(0, 0x70, (n, k), dtype=torch.uint8, device=dev, generator=g) for n in (1, rows))
    scale, ws = torch.ones((1,), device=dev), torch.full((rows,), 0x3F80, dtype=torch.int16, device=dev)
    y = torch.zeros((rows,), device=dev)
    return (lambda s: lib.raw("gemb_fp8_gemv", act, scale, w, ws, y, rows, k, s)), y


def _head(lib, dev, hidden):
    rows, vocab = 4, 4096
    g = torch.Generator(device=dev).manual_seed(hidden)
    w = torch.randn((vocab, hidden), device=dev, generator=g).to(torch.bfloat16).view(torch.int16)
    h, y = torch.randn((rows, hidden), device=dev, generator=g), torch.zeros((rows, vocab), device=dev)
    return (lambda s: lib.raw("gemb_output_head_candidates", w, h, rows, None, 0, None, None, y, vocab, hidden, s)), y


def _router_input(lib, dev, hidden):
    tokens = 9
    g = torch.Generator(device=dev).manual_seed(hidden)
    x = torch.randn((tokens, hidden), device=dev, generator=g).to(torch.bfloat16).view(torch.int16)
    scale = torch.full((hidden,), 0x3F80, dtype=torch.int16, device=dev)
    y = torch.zeros((tokens, hidden), dtype=torch.int16, device=dev)
    return (lambda s: lib.raw("gemb_moe_router_input", x, scale, y, tokens, hidden, 1e-6, s)), y


# Both sizes of a pair need more than the 48 KB of shared memory that a kernel has by itself.
@pytest.mark.parametrize("make,small,large", [(_nvfp4, 20480, 98304), (_fp8, 32768, 112640), (_head, 1536, 4096), (_router_input, 4096, 12288)],
                         ids=["nvfp4_gemv", "fp8_gemv", "output_head", "router_input"])
def test_threads_with_different_sizes(lib, dev, make, small, large):
    """The kernel's shared-memory limit suits both: no launch of one thread fails for the size of the other."""
    calls = [make(lib, dev, n) for n in (small, large)]
    want = []
    for call, y in calls:
        assert call(None) == 0, lib.last_error()
        torch.cuda.synchronize()
        want.append(y.clone())
        y.zero_()
    streams = [torch.cuda.Stream(device=dev) for _ in calls]
    torch.cuda.synchronize()
    failures, gate = [], threading.Barrier(len(calls))

    def work(i):
        gate.wait()
        for _ in range(REPS):
            rc = calls[i][0](streams[i])
            if rc != 0:
                failures.append((i, rc, lib.last_error()))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failures, failures[:3]
    for (_, y), w in zip(calls, want):
        assert torch.equal(y.view(torch.int32 if y.dtype == torch.float32 else y.dtype), w.view(torch.int32 if w.dtype == torch.float32 else w.dtype))
