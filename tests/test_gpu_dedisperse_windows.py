"""The windowed dedispersion where its copies and tiles can go wrong: every
tile height (16, 8 and 4 trials, chosen by trial count and delay spread), one
past and one short of a tile and of a stage of channels, output lengths around
a time tile, filterbanks at odd float offsets and of odd row lengths (window
starts rounded down to 16 bytes, first and last windows leaving the array),
and the largest spread the windows take and the next.  Bit-exact."""
import numpy as np
import pytest

from gpu_accelsearch_gb300.dedisperse import dedisperse
from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def check(nchan, ndm, nout, delays, offset=0, slack=0):
    rng = np.random.default_rng(nchan * 131 + ndm * 17 + nout)
    nsamp = nout + int(delays.max()) + slack
    fb = rng.standard_normal((nchan, nsamp)).astype(np.float32)
    d_fb = torch.empty(nchan * nsamp + offset, dtype=torch.float32, device="cuda")
    d_fb[offset:] = torch.from_numpy(fb.reshape(-1)).cuda()
    d_out = torch.full((ndm, nout), np.nan, dtype=torch.float32, device="cuda")
    dedisperse(d_fb.data_ptr() + 4 * offset, nchan, nsamp, delays, d_out.data_ptr(), nout)
    torch.cuda.synchronize()
    want = O.dedisperse(fb, delays, nout)
    assert np.array_equal(d_out.cpu().numpy().view(np.uint32), want.view(np.uint32))


def slope(nchan, ndm, step):
    """Delays growing by up to `step` samples per trial over the band."""
    return np.floor(np.arange(ndm)[:, None] * step * np.arange(nchan)[None, :] / max(1, nchan - 1)).astype(np.int32)


@pytest.mark.parametrize("ndm", [1, 3, 4, 5, 8, 9, 15, 16, 17, 33])
@pytest.mark.parametrize("nchan,nout", [(1, 1), (3, 1023), (4, 1024), (5, 1025), (13, 4097)])
def test_tiles_and_stages(ndm, nchan, nout):
    check(nchan, ndm, nout, slope(nchan, ndm, 7.0))


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("slack", [0, 1, 2, 3])
def test_unaligned_rows(offset, slack):
    check(7, 6, 2050, slope(7, 6, 11.0), offset, slack)


# 16-trial tiles take 1250 samples of spread, 8- and 4-trial tiles the same;
# wider ones the one-load-per-addition kernel
@pytest.mark.parametrize("step", [60.0, 84.0, 170.0, 180.0, 400.0, 430.0, 900.0])
def test_spreads(step):
    check(9, 20, 3000, slope(9, 20, step))


def test_unordered_delays():
    rng = np.random.default_rng(5)
    check(11, 21, 1500, rng.integers(0, 900, (21, 11)).astype(np.int32))
