"""Smoothed fields and surrogate features from several threads and streams at once: the bits of serial calls."""
import threading

import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own_stream", [False, True])
@pytest.mark.parametrize("n", [32, 128])
def test_concurrent_calls_match_serial_ones(n, own_stream):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sg, radii, workers, rounds = module("surrogate"), (2.0, 5.0), 4, 8
    g = torch.Generator(device="cuda").manual_seed(n)
    boxes = [torch.randn((n, n, n), device="cuda", generator=g) for _ in range(workers)]
    ref = [sg.smoothed_fields(b, radii) for b in boxes]
    torch.cuda.synchronize()
    start, bad = threading.Barrier(workers), []

    def work(i):
        s = torch.cuda.Stream() if own_stream else torch.cuda.current_stream()
        start.wait()
        with torch.cuda.stream(s):
            got = [sg.smoothed_fields(boxes[i], radii) for _ in range(rounds)]
            s.synchronize()
            bad.extend(1 for x in got if not torch.equal(x, ref[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(workers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_a_captured_call_replays():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sg, n = module("surrogate"), 32
    x = torch.randn((n, n, n), device="cuda")
    y = torch.randn((n, n, n), device="cuda")
    want = sg.smoothed_fields(y, (3.0,)).clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = sg.smoothed_fields(x, (3.0,))
    x.copy_(y)
    graph.replay()
    assert torch.equal(out, want)
