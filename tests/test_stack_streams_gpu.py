"""A Stack's time reversal on several streams and inside a captured graph."""
import pytest
import torch

import haste_b200

pytestmark = pytest.mark.gpu


def _stack(T):
    torch.manual_seed(0)
    net = haste_b200.Stack(haste_b200.GRU, 16, 32, num_layers=2, bidirectional=True).cuda().eval()
    return net, torch.randn(T, 5, 16, device="cuda")


def test_first_call_of_a_length_inside_a_graph():
    net, x = _stack(48)
    long = torch.randn(64, 5, 16, device="cuda")
    stream = torch.cuda.Stream()
    with torch.no_grad():
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            net(long)  # scratch of this stream grows outside the graph
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            captured = net(x)
        with torch.cuda.stream(stream):
            eager = net(x)  # before the graph has run
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        torch.testing.assert_close(captured, eager, rtol=0, atol=0)
        del graph
        torch.cuda.empty_cache()
        with torch.cuda.stream(stream):
            again = net(x)  # after the graph's memory is gone
        torch.cuda.synchronize()
        torch.testing.assert_close(again, eager, rtol=0, atol=0)


def test_streams_that_know_nothing_of_one_another():
    net, x = _stack(57)
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    got = []
    with torch.no_grad():
        for s in streams:
            with torch.cuda.stream(s):
                got.append(net(x))
        torch.cuda.synchronize()
        want = net(x)
    for y in got:
        torch.testing.assert_close(y, want, rtol=0, atol=0)
