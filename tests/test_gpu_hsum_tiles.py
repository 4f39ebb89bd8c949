"""Harmonic sums of caller-owned planes by box copies and by row copies, at
the tile heights the plan allows (16 harmonics: only the 8-row tiles fit),
with many candidates per tile (one reservation per warp) and a candidate
buffer that overflows: stage sums and candidates equal a NumPy restatement
on the same planes bit for bit (single-precision additions in harmonic
order)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def restated(s, planes, startr):
    """Stage sums [stage][z][i] of one segment's planes (float32 adds in bank order)."""
    U, hs = s.uselen, s.harmonics
    zz = np.arange(-hs[0].zmax, hs[0].zmax + 1, 2)
    i = np.arange(U)
    out, acc = [], None
    for h, hi in enumerate(hs):
        p, q = hi.harmnum, hi.maxharm
        P = planes[s.plane_off[h]: s.plane_off[h] + hi.numzs * s.plane_row[h]].reshape(hi.numzs, s.plane_row[h])
        if h == 0:
            acc = P[:, :U].copy()
        else:
            rlo = ((4 * startr * p + q) // (2 * q)) >> 1
            rind = ((2 * (2 * startr + i) * p + q) // (2 * q) - 2 * rlo) & 0xffff
            d = np.sign(zz) * (np.abs(zz) * p // q) - hi.zlo
            zind = np.sign(d) * (np.abs(d) // 2)
            acc = acc + P[zind][:, rind]
        if (h + 1) & h == 0:
            out.append(acc)
    return np.stack(out)


@pytest.mark.parametrize("zmax,nh,L", [(0, 1, 128), (20, 2, 1024), (50, 4, 2048), (200, 8, 4096), (100, 16, 8192)])
@pytest.mark.parametrize("tuning", [{}, {"hsum_row_copies": 1}, {"hsum_tile_rows": 8}, {"hsum_tile_rows": 32},
                                    {"hsum_rowwise": 1}], ids=str)
def test_sums_and_counts_on_callers_planes(zmax, nh, L, tuning):
    from gpu_accelsearch_gb300.search import AccelSearch
    with AccelSearch(zmax=zmax, numharm=nh, fftlen=L, chunk_segments=2) as s:
        s.set_tuning(**tuning)
        startr = [40, 41, 40 + s.uselen // 2 + 3]
        g = torch.Generator(device="cuda")
        g.manual_seed(L + nh)
        planes = -torch.log(torch.rand((len(startr), s.plane_stride), generator=g, device="cuda"))
        stage = torch.zeros((len(startr), s.nstages, s.harmonics[0].numzs, s.uselen), device="cuda")
        cuts = [3.0 + 2.0 * k for k in range(s.nstages)]
        s.set_power_cuts(cuts)
        n = s.sum_harmonics(planes.data_ptr(), startr, stage.data_ptr())
        n2 = s.sum_harmonics(planes.data_ptr(), startr)  # without stage planes
        P, got = planes.cpu().numpy(), stage.cpu().numpy()
        count = 0
        for k, r in enumerate(startr):
            want = restated(s, P[k], r)
            assert np.array_equal(got[k], want), (k, np.abs(got[k] - want).max())
            count += sum(int((want[st] > np.float32(c)).sum()) for st, c in enumerate(cuts))
        assert n == n2 == count and count > 0


def test_overflowing_candidate_buffer():
    from gpu_accelsearch_gb300.native import AccelError
    from gpu_accelsearch_gb300.search import AccelSearch
    g = torch.Generator(device="cuda")
    g.manual_seed(8)
    spec = torch.randn((1 << 15, 2), generator=g, device="cuda")
    with AccelSearch(zmax=50, numharm=4, fftlen=2048, chunk_segments=8, cand_capacity=1000) as s, \
            AccelSearch(zmax=50, numharm=4, fftlen=2048, chunk_segments=8) as full:
        for t in (s, full):
            t.set_power_cuts([9.0, 12.0, 16.0])
        n = full.search_spectra([spec.data_ptr()], [1 << 15], [16])
        whole = full.candidates()
        assert n == len(whole) > 1000
        with pytest.raises(AccelError):
            s.search_spectra([spec.data_ptr()], [1 << 15], [16])
        some = s.candidates()
        assert len(some) == 1000
        keys = lambda c: {tuple(x) for x in c[["step", "numharm", "z", "r", "power"]].tolist()}  # noqa: E731
        assert keys(some) <= keys(whole) and len(keys(some)) == 1000
