"""Steps that a caller captures into a CUDA graph of its own on the context's stream: any count, replayed as
often as the caller likes, in between direct steps.  The reference is a context stepped directly.  A graph of
an odd count n ends in the other buffer while its first one holds the state after n - 1 steps, where the next
replay starts: r replays make n + (r - 1)(n - 1) steps; with an even count they make r n."""
import numpy as np
import pytest
import torch

import microsim_b200 as mb
from microsim_b200 import configs

pytestmark = pytest.mark.gpu


def _same(a, b, what):
    for x, y in zip(a.download(), b.download()):
        assert np.array_equal(x, y), what


@pytest.mark.parametrize("precision", [mb.GP_FP64, mb.GP_FP32])
@pytest.mark.parametrize("n", [1, 3, 8, 64, 71])
def test_captured_steps_equal_direct_ones(n, precision):
    m, phi, mu = mb.load_case(configs.binary_case(70, 90, gap=1.0, supersat=0.5, eps=4.0, delta=0.03, dt=0.05,
                                                  tau=1.7776, seed=(0, 0, 20.0)))
    with mb.Context(m, precision) as a, mb.Context(m, precision) as b:
        for c in (a, b):
            c.upload(phi, mu)
            for _ in range(5):  # both buffers and every kernel in use before the capture
                c.step(1)
            c.sync()
        stream = torch.cuda.ExternalStream(a.stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="relaxed")
            try:
                a.step(n)
            finally:
                graph.capture_end()
            for _ in range(4):
                graph.replay()
        a.sync()
        for _ in range(n + 3 * (n - n % 2)):
            b.step(1)
        _same(a, b, "replays")
        for k in (1, 9, 66):
            a.step(k)
            b.step(k)
        _same(a, b, "direct steps after the replays")
        del graph


@pytest.mark.parametrize("precision", [mb.GP_FP64, mb.GP_FP32])
@pytest.mark.parametrize("first", [True, False])
def test_a_state_changed_between_replays_is_seen(first, precision):
    """The caller writes a patch of solid into the bulk between replays of its graph; `first`: the capture is
    the first step after an upload, whose state no step has looked at."""
    m, phi, mu = mb.load_case(configs.binary_case(70, 90, gap=1.0, supersat=0.5, eps=4.0, delta=0.03, dt=0.05,
                                                  tau=1.7776, seed=(0, 0, 20.0)))

    def write(c, k):
        p, _ = c.device_state()
        p[0, 40:50, 30 + 8 * k:36 + 8 * k], p[1, 40:50, 30 + 8 * k:36 + 8 * k] = 1.0, 0.0
        torch.cuda.synchronize()
        c.state_changed()

    with mb.Context(m, precision) as a, mb.Context(m, precision) as b:
        for c in (a, b):
            c.upload(phi, mu)
            c.step(4)
            if first:
                c.upload(*c.download())
            c.sync()
        stream = torch.cuda.ExternalStream(a.stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="relaxed")
            try:
                a.step(2)
            finally:
                graph.capture_end()
        for k in range(6):
            if k != 1:
                write(a, k)
                write(b, k)
            if k % 3 == 2:
                a.step(8)
                b.step(8)
            else:
                with torch.cuda.stream(stream):
                    graph.replay()
                a.sync()
                b.step(2)
            b.sync()
            _same(a, b, k)
        del graph
