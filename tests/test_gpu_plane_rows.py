"""Plane rows stored as one bulk copy each (half lengths 1024 and 2048) against
plain stores: planes that start on 8 bytes take the plain stores and must hold
the same bits; nothing outside the rows' columns is written."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# fundamentals of 1024 and 2048 points, odd and even numbers of column pairs
@pytest.mark.parametrize("zmax,nh,L,uselen", [(50, 4, 2048, 0), (50, 2, 2048, 1402), (120, 8, 4096, 0),
                                              (20, 1, 4096, 3302), (20, 1, 2048, 1702)])
@pytest.mark.parametrize("fp16", [0, 1])
def test_bulk_rows_equal_plain_stores(zmax, nh, L, uselen, fp16):
    from gpu_accelsearch_gb300.search import AccelSearch
    kw = {"uselen": uselen} if uselen else {}
    rng = np.random.default_rng(L + uselen)
    with AccelSearch(zmax=zmax, numharm=nh, fftlen=L, template_fp16=bool(fp16), **kw) as s:
        d = torch.from_numpy(rng.standard_normal((3, s.dhalf_stride, 2)).astype(np.float32)).cuda()
        n = 3 * s.plane_stride
        got = []
        for off in (0, 2):  # floats
            pl = torch.full((n + 8,), -1.0, device="cuda")
            s.power_planes(d.data_ptr(), 3, pl.data_ptr() + 4 * off)
            p = pl.cpu().numpy()
            assert np.all(p[:off] == -1.0) and np.all(p[off + n:] == -1.0)
            got.append(p[off:off + n].reshape(3, s.plane_stride))
        assert np.array_equal(got[0], got[1])
        for h, hi in enumerate(s.harmonics):
            rows = got[0][:, s.plane_off[h]: s.plane_off[h] + hi.numzs * s.plane_row[h]]
            assert (rows.reshape(3, hi.numzs, -1)[:, :, 0] >= 0.0).all(), h
