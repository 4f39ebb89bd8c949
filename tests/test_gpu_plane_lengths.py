"""Power planes at every transform length from 64 points, in every layout that
runs the shared-memory transform (default, sequential, fused sum): the planes
within the power tolerance of the FP64 oracle, |P - P64| / max(P64, 1) < 1e-4,
the layouts' candidates identical."""
import numpy as np
import pytest

from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# fundamentals of 64, 128, 256, 512, 1024, 2048 and 8192 points and their
# sub-harmonics
@pytest.mark.parametrize("zmax,nh,L", [(0, 1, 128), (2, 1, 256), (6, 2, 512), (14, 4, 1024), (50, 4, 2048),
                                       (120, 8, 4096), (60, 2, 16384)])
def test_planes_and_layouts(zmax, nh, L):
    from gpu_accelsearch_gb300.search import AccelSearch
    rng = np.random.default_rng(L)
    with AccelSearch(zmax=zmax, numharm=nh, fftlen=L, chunk_segments=3) as s:
        half = s.uselen // 2
        nb = 7 * half + 9
        spec = (rng.standard_normal(nb) + 1j * rng.standard_normal(nb)).astype(np.complex64)
        spec[3 * half + half // 2] += 12.0
        d = torch.from_numpy(spec.view(np.float32).copy()).cuda()
        starts = [5, 5 + 3 * half]
        dh = torch.zeros((2, s.dhalf_stride, 2), device="cuda")
        pl = torch.zeros((2, s.plane_stride), device="cuda")
        s.prepare_segments(d.data_ptr(), nb, starts, dh.data_ptr())
        s.power_planes(dh.data_ptr(), 2, pl.data_ptr())
        P = pl.cpu().numpy()
        o = O.Oracle(zmax, nh, s.uselen)
        for i, r in enumerate(starts):
            for h, hi in enumerate(s.harmonics):
                p64 = o.harmonic_plane(spec, float(r), h)
                g = P[i, s.plane_off[h]: s.plane_off[h] + hi.numzs * s.plane_row[h]]
                g = g.reshape(hi.numzs, s.plane_row[h])[:, : p64.shape[1]]
                assert (np.abs(g - p64) / np.maximum(p64, 1.0)).max() < 1e-4, (i, h)
        o.close()
        s.set_power_cuts([6.0 + 3.0 * k for k in range(s.nstages)])
        want = None
        for tuning in ({}, {"plane_split": 1}, {"fused_sum": 1}):
            s.set_tuning(plane_split=0, fused_sum=0)
            s.set_tuning(**tuning)
            s.search_spectra([d.data_ptr()], [nb], [5])
            got = s.candidates()
            assert len(got) > 0
            assert want is None or np.array_equal(got, want), tuning
            want = got
