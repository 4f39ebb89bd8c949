"""The phases of the real-to-complex transform's unpacking, to the last bit.

A series that is 1 at sample 1 and 0 elsewhere has Z[k] = i in every bin of
the half-length transform (a power of two, or an odd factor up to 15 whose
other subsequences are zero: no rounding), so that X[k] is the conjugate of
the unpacking's phase exp(2 pi i k / N) as the kernel rounds it.

Bound: the phase is a double-precision product rounded once to float.  The
table entries and the product are each within a few 2^-53, so a component is
within half a unit in the last place plus 2^-51 of the exact value.  11 * 2^17
has one component (of its 1.4 million) where a product of two-float numbers
rounds the other way."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

LD = np.longdouble


def exact_phase(K):
    """cos and sin of pi k / K, k = 0 .. K, in extended precision, every
    argument reduced to [0, pi/4]."""
    pi = LD("3.14159265358979323846264338327950288")
    k = np.arange(K + 1, dtype=np.int64)
    m = np.where(2 * k > K, K - k, k)
    swap = 4 * m > K
    x = np.where(swap, K - 2 * m, 2 * m).astype(LD) * pi / LD(2 * K)
    c, s = np.cos(x), np.sin(x)
    c, s = np.where(swap, s, c), np.where(swap, c, s)
    return np.where(2 * k > K, -c, c), s


def test_reference_phase():
    c, s = exact_phase(12)
    assert np.allclose(c.astype(float), np.cos(np.pi * np.arange(13) / 12), atol=1e-15)
    assert np.allclose(s.astype(float), np.sin(np.pi * np.arange(13) / 12), atol=1e-15)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [11 << 17, 1 << 21, 15 << 15, 1 << 13, 12, 4])
def test_phases_are_rounded_once(n):
    if np.finfo(LD).nmant < 63:
        pytest.skip("needs an extended long double")
    from gpu_accelsearch_gb300.search import AccelSearch
    x = torch.zeros(n, device="cuda")
    x[1] = 1.0
    spec = torch.full((n + 2,), np.nan, device="cuda")
    with AccelSearch(zmax=0, numharm=1, fftlen=128) as s:
        torch.cuda.synchronize()
        s.rfft(x.data_ptr(), n, spec.data_ptr())
        s.synchronize()
    got = spec.cpu().numpy().reshape(-1, 2)
    c, si = exact_phase(n // 2)
    for have, want in ((got[:, 0], c), (-got[:, 1], si)):
        ulp = np.spacing(np.abs(have)).astype(LD)
        err = np.abs(have.astype(LD) - want)
        assert np.all(err <= 0.5 * ulp + LD(2.0) ** -51), (err / ulp).max()
