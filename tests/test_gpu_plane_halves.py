"""Rows of 8192 points, whose two transforms run in CTAs of their own: the same
bits as the sequential layout (the butterflies, twiddles and their order are the
same), nothing outside the rows' columns written, FP32 and FP16 templates."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# default and smaller windows (odd and even numbers of column pairs), one and
# several harmonics, one and several segments
@pytest.mark.parametrize("zmax,nh,uselen,nseg", [(0, 1, 0, 1), (60, 2, 0, 3), (40, 1, 12002, 2), (100, 4, 11000, 1)])
@pytest.mark.parametrize("fp16", [False, True])
def test_halves_equal_sequential(zmax, nh, uselen, nseg, fp16):
    from gpu_accelsearch_gb300.search import AccelSearch
    rng = np.random.default_rng(zmax + nseg)
    with AccelSearch(zmax=zmax, numharm=nh, fftlen=16384, uselen=uselen, template_fp16=fp16) as s:
        d = torch.from_numpy(rng.standard_normal((nseg, s.dhalf_stride, 2)).astype(np.float32)).cuda()
        got = []
        for split in (0, 1):
            s.set_tuning(plane_split=split)
            pl = torch.full((nseg, s.plane_stride), -1.0, device="cuda")
            s.power_planes(d.data_ptr(), nseg, pl.data_ptr())
            got.append(pl.cpu().numpy())
        assert np.array_equal(got[0], got[1])
        assert (got[0][:, 0] >= 0.0).all()
