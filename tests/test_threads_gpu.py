"""Several threads at once, on one stream and on streams of their own."""
import threading

import pytest
import torch

import haste_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own_streams", [False, True])
def test_threads_get_what_one_thread_gets(own_streams):
    # layers whose scratch differs in size and in use: cluster, grid and step-wise recurrences
    shapes = [("LSTM", 9, 7, 40), ("GRU", 5, 70, 512), ("LSTM", 3, 5, 1040), ("LayerNormLSTM", 6, 9, 96),
              ("LayerNormGRU", 4, 20, 400), ("IndRNN", 20, 30, 64)]
    work = []
    for cell, T, N, H in shapes:
        torch.manual_seed(H)
        layer = getattr(haste_b200, cell)(32, H).cuda()
        work.append((layer, torch.randn(T, N, 32, device="cuda"), torch.randn(T, N, H, device="cuda")))

    def one_pass(layer, x, dy):
        y = layer(x)[0]
        return [y.detach()] + list(torch.autograd.grad(y, list(layer.parameters()), dy))

    want = [one_pass(*w) for w in work]
    torch.cuda.synchronize()
    got, errors = [[] for _ in work], []

    def run(i):
        try:
            stream = torch.cuda.Stream() if own_streams else torch.cuda.default_stream()
            with torch.cuda.stream(stream):
                for _ in range(8):
                    got[i].append(one_pass(*work[i]))
            stream.synchronize()
        except Exception as e:  # handed to the main thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for w, passes in zip(want, got):
        assert len(passes) == 8
        for tensors in passes:
            for a, b in zip(tensors, w):
                torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)
