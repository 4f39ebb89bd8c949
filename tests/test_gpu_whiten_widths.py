"""Whitening at the block widths where its kernels change form: 128, 256 and
1024 bins (registers per lane of the median, warp and CTA forms) and the
warp's own edges, on spectra with ties: bit-identical to the oracle."""
import numpy as np
import pytest

from gpu_accelsearch_gb300.synth import synth_red_spectrum
from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def same(a, b):
    a, b = a.view(np.float32), b.view(np.float32)
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("width", [2, 3, 31, 32, 33, 127, 128, 129, 255, 256, 257, 1023, 1024, 1025])
def test_widths_bit_exact(width):
    from gpu_accelsearch_gb300.search import AccelSearch
    with AccelSearch(zmax=0, numharm=1, fftlen=128, whiten_initbuf=width, whiten_maxbuf=width) as s:
        for numbins in (width + 2, 3 * width + 1, 70 * width + 11):
            red = synth_red_spectrum(numbins, seed=width)
            flat = np.ones(numbins, np.complex64)  # every power equal
            few = (np.random.default_rng(width).integers(0, 3, numbins) + 1j).astype(np.complex64)
            for spec in (red, flat, few, np.zeros(numbins, np.complex64)):
                d = torch.from_numpy(spec.view(np.float32).copy()).cuda()
                s.whiten(d.data_ptr(), numbins)
                s.synchronize()
                got = d.cpu().numpy().view(np.complex64)
                assert same(got, O.deredden(spec, width, width)), (numbins,)
