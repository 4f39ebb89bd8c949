"""Segment preparation's exact median and normalisation where its search can
go wrong: every half length from 64 to 8192 (one warp, part of a warp, up to
16 warps), ties, all-equal and all-zero segments, powers that differ in the
last bit or only in the sign of a wide exponent range, windows past both ends
of the spectrum.  The un-normalised tail and the median-scaled part are
compared through the transform: DFT of the oracle's segment in double
precision.

Tolerance: the segment values are bit-exact (the reference's operations), the
forward transform of M points in single precision is within 4e-7 sqrt(log2 M)
of the segment's norm; 2e-6 covers it."""
import numpy as np
import pytest

from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def spectra(nb, seed):
    rng = np.random.default_rng(seed)
    g = (rng.standard_normal(nb) + 1j * rng.standard_normal(nb)).astype(np.complex64)
    ties = (rng.integers(1, 4, nb) + 0j).astype(np.complex64)
    last = (np.float32(1.0) + rng.integers(0, 2, nb) * np.float32(2.0 ** -23)).astype(np.complex64)
    wide = (g * (2.0 ** rng.integers(-30, 30, nb))).astype(np.complex64)
    return [g, ties, last, wide, np.ones(nb, np.complex64), np.zeros(nb, np.complex64)]


# fundamentals of half length 64 .. 8192; with their sub-harmonics every
# smaller length runs in the same launch
@pytest.mark.parametrize("zmax,nh,L", [(0, 1, 128), (0, 2, 256), (4, 1, 512), (10, 2, 1024), (50, 4, 2048),
                                       (100, 8, 4096), (200, 8, 8192), (100, 16, 16384)])
def test_segments(zmax, nh, L):
    from gpu_accelsearch_gb300.search import AccelSearch
    with AccelSearch(zmax=zmax, numharm=nh, fftlen=L, chunk_segments=2) as s:
        half = s.uselen // 2
        nb = 6 * half + 5
        starts = [0, 3, half + 1, nb - half // 2]  # the first and last reach past the spectrum
        for spec in spectra(nb, L + nh):
            d = torch.from_numpy(spec.view(np.float32).copy()).cuda()
            out = torch.zeros((len(starts), s.dhalf_stride, 2), device="cuda")
            s.prepare_segments(d.data_ptr(), nb, starts, out.data_ptr())
            got = out.cpu().numpy().view(np.complex64)[..., 0]
            for i, r in enumerate(starts):
                for h, hi in enumerate(s.harmonics):
                    rlo, rhi, _, _ = O.step_ffdot(hi.harmnum, hi.maxharm, zmax, s.uselen, float(r), r + half - 0.5)
                    M = hi.fftlen // 2
                    seg = O.segment_data(spec, rlo, rhi, hi.halfwidth, hi.fftlen)
                    want = np.fft.fft(seg[0::2].astype(np.complex128)) if seg.size == 2 * M else None
                    g = got[i, s.dhalf_off[h]: s.dhalf_off[h] + M]
                    scale = np.linalg.norm(want)
                    if not np.isfinite(scale):
                        continue
                    assert np.linalg.norm(g - want) <= 2e-6 * scale + 1e-30, (zmax, L, i, h)
