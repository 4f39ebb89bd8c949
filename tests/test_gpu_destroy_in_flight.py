"""Destroying a context while its transform or whitening still runs: the
memory they use is given back only after them.  Bit-identical to the same
calls waited for, on the context's own stream and on a caller's, which the
destruction leaves usable."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# Bluestein, the Cooley-Tukey step from a row at an odd offset, a power of two
@pytest.mark.parametrize("n,odd", [(2 * 2097169, 0), (15 << 19, 1), (1 << 23, 0)])
@pytest.mark.parametrize("own_stream", [True, False])
def test_transform_and_whitening(n, odd, own_stream):
    from gpu_accelsearch_gb300 import native as N
    from gpu_accelsearch_gb300.search import AccelSearch
    x = torch.randn(n + odd, device="cuda")[odd:]
    st = torch.cuda.Stream()
    out = []
    for wait in (True, False, False):
        spec = torch.full((n + 2,), np.nan, device="cuda")
        torch.cuda.synchronize()
        s = AccelSearch(zmax=0, numharm=1, fftlen=128)
        if not own_stream:
            N.check(N.lib().accel_set_stream(s._h, st.cuda_stream))
        for _ in range(3):  # the last of several: the others keep the GPU behind the host
            s.rfft(x.data_ptr(), n, spec.data_ptr())
        s.whiten(spec.data_ptr(), n // 2)
        if wait:
            s.synchronize()
        s.close()
        other = torch.zeros(1 << 24, device="cuda")  # what was freed may be used again
        other.fill_(1.0)
        torch.cuda.synchronize()
        out.append(spec)
    assert torch.equal(out[0][: n // 2 * 2], out[1][: n // 2 * 2])
    assert torch.equal(out[0][: n // 2 * 2], out[2][: n // 2 * 2])
