"""Scratch of the stage calls (allocated in stream order, kept between calls):
calls of several sizes from several threads and streams at once, and a call
that is captured in a graph."""
import threading

import numpy as np
import pytest

from cases import bits, make_case

pytestmark = pytest.mark.gpu


def test_stage_calls_from_threads_and_streams(cuda):
    import torch
    from cageo_gb300 import api
    sizes = [(120, 90), (300, 200), (64, 500), (31, 33)]

    def work(W, H):
        dem, streams = make_case(W, H, seed=W)
        v, s = torch.from_numpy(dem).to(cuda), torch.from_numpy(streams).to(cuda)
        api.stream_burn(v, s)
        f = api.pitfill(v)
        d = api.route_d8(f)
        return f, d, api.trace(d, s)

    want = [[t.cpu().numpy() for t in work(W, H)] for W, H in sizes]
    errors = []

    def run(k):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for i in range(12):
                    j = (k + i) % len(sizes)
                    got = [t.cpu().numpy() for t in work(*sizes[j])]
                    for a, b in zip(got, want[j]):
                        assert np.array_equal(bits(a), bits(b))
        except Exception as e:  # shown by the main thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_burning_in_a_graph(cuda):
    """A captured call's scratch belongs to the graph."""
    import torch
    from cageo_gb300 import api
    dem, streams = make_case(200, 150, seed=4)
    src, s = torch.from_numpy(dem).to(cuda), torch.from_numpy(streams).to(cuda)
    want = api.stream_burn(src.clone(), s).clone()
    v = torch.empty_like(src)
    g = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        v.copy_(src)
        stream.synchronize()
        with torch.cuda.graph(g, stream=stream):
            api.stream_burn(v, s)
        for _ in range(3):
            v.copy_(src)
            g.replay()
            stream.synchronize()
            assert torch.equal(v, want)
