"""Transforms of alternating lengths on one context (tables kept per
length), from aligned and odd-offset rows, and recorded into a caller's
CUDA graph: bit-identical to the first call of each."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# a power of two, Cooley-Tukey steps, Bluestein (even and odd half lengths)
LENGTHS = [4, 1 << 12, 3 << 13, 15 << 8, 2 * 4099, 2 * 17 * 64, 2 * 30011, 34]


def run(s, x, spec):
    s.rfft(x.data_ptr(), x.numel(), spec.data_ptr())


def test_alternating_lengths_and_offsets():
    from gpu_accelsearch_gb300.search import AccelSearch
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    with AccelSearch(zmax=0, numharm=1, fftlen=128) as s:
        want = {}
        for turn in range(3):
            for n in (LENGTHS if turn != 1 else LENGTHS[::-1]):
                if n not in want:
                    x = torch.randn(n, generator=g, device="cuda")
                    want[n] = (x, None)
                x, ref = want[n]
                row = torch.zeros(n + 1, device="cuda")
                row[1:] = x
                for src in (x, row[1:]):
                    spec = torch.full((n + 2,), np.nan, device="cuda")
                    run(s, src, spec)
                    s.synchronize()
                    if ref is None:
                        ref = spec
                        exact = torch.fft.rfft(x.double())
                        err = (torch.view_as_complex(spec.view(-1, 2)) - exact).abs()
                        assert err.max() <= 2e-5 * exact.abs().square().mean().sqrt()
                    assert torch.equal(spec, ref), (n, turn)
                want[n] = (x, ref)


@pytest.mark.parametrize("n", [1 << 12, 3 << 13, 2 * 4099])
def test_recorded_into_a_graph(n):
    from gpu_accelsearch_gb300 import native as N
    from gpu_accelsearch_gb300.search import AccelSearch
    with AccelSearch(zmax=0, numharm=1, fftlen=128) as s:
        st = torch.cuda.Stream()
        N.check(N.lib().accel_set_stream(s._h, st.cuda_stream))
        x = torch.randn(n, device="cuda")
        a, b = (torch.zeros(n + 2, device="cuda") for _ in range(2))
        run(s, x, a)
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st, capture_error_mode="thread_local"):
            run(s, x, b)
        for m in LENGTHS:  # other lengths come and go
            y, c = torch.randn(m, device="cuda"), torch.zeros(m + 2, device="cuda")
            torch.cuda.synchronize()
            run(s, y, c)
        s.synchronize()
        for _ in range(2):
            b.zero_()
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(a, b)
        del graph
        torch.cuda.synchronize()
        N.check(N.lib().accel_set_stream(s._h, None))
