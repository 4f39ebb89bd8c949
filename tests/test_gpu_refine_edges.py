"""Refinement's node-rule evaluation (refine.cu) where it can go wrong:
windows running off either end of the spectrum, f-dots at and around the
steps of the halfwidth, zero and sign changes within a grid, 1 to 16
harmonics, r on and off bin boundaries, and a window wide enough for the
direct form.  Against the same correlation with the response integrated
numerically in double precision.

Tolerance: both sides work in double precision on the same float spectrum
(rule and quadrature errors about 1e-12) and the result is rounded once to
float: 6e-8 relative, tested at 3e-7."""
import numpy as np
import pytest

from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, RLO, TOBS = 1 << 17, 16, 10.0


def response(x, z):
    """Integral over u in [0, 1] of exp(i pi (2 x u + z u^2))."""
    m = int(200 + 4 * (np.abs(x).max() + abs(z)))
    u, w = np.polynomial.legendre.leggauss(min(m, 1500))
    u, w = 0.5 * (u + 1), 0.5 * w
    return (w * np.exp(1j * np.pi * (2 * np.outer(x, u) + z * u * u))).sum(1)


def power(spec, r, z):
    hw = O.z_halfwidth(z)
    j = np.arange(int(np.ceil(r)) - hw, int(np.ceil(r)) + hw)
    ok = (j >= 0) & (j < spec.size)
    x = np.where(ok, spec[np.clip(j, 0, spec.size - 1)], 0).astype(np.complex128)
    return abs(np.sum(x * np.conj(response(r - j - z / 2, z)))) ** 2


@pytest.fixture(scope="module", params=[(50, 4, 2048), (100, 16, 8192)], ids=["z50_h4", "z100_h16"])
def bank(request):
    from gpu_accelsearch_gb300.search import AccelSearch
    zmax, nh, L = request.param
    rng = np.random.default_rng(L)
    spec = (rng.standard_normal(N // 2) + 1j * rng.standard_normal(N // 2)).astype(np.complex64)
    with AccelSearch(zmax=zmax, numharm=nh, fftlen=L, chunk_segments=4) as s:
        d = torch.from_numpy(spec.view(np.float32).copy()).cuda()
        yield s, spec, d, zmax, nh


def cands(rows):
    from gpu_accelsearch_gb300.search import CAND_DTYPE
    c = np.zeros(len(rows), CAND_DTYPE)
    for i, (step, r, z, nh) in enumerate(rows):
        c[i] = (0, step, r, z, nh, 30.0, 6.0)
    return c


@pytest.mark.parametrize("refine", [False, True])
def test_powers_at_the_refined_position(bank, refine):
    s, spec, d, zmax, nh = bank
    top = N // 2
    rows = []
    for i, (r, z) in enumerate([(0.0, 0.0), (3.25, -40.0), (17.5, 2.0), (1000.0, 0.0), (1000.5, 0.3), (2047.75, -1.0),
                                (5000.25, 39.4), (7000.0, -100.5), (9000.5, 101.0), (12000.125, 99.9),
                                (20000.0, 258.4), (top - 1.0, 20.0), (top - 0.5, -77.0), (top + 3.0, 4.0)]):
        rows.append((i % 5, r, z, min(nh, 1 << (i % 5))))
    rows += [(2, 30000.25, -33.3, nh), (0, 40000.0, 12.0, 1)]
    c = cands(rows)
    o = s.optimize(c, RLO, TOBS, spectra=[(d.data_ptr(), spec.size)], refine=refine)
    for row, g in zip(rows, o):
        step, r, z, H = row
        if not refine:
            assert g["r"] == r and g["z"] == z
        assert abs(g["r"] - r) <= 0.65626 and abs(g["z"] - z) <= 2.6251
        n2 = O.step_norms(spec, zmax, nh, s.uselen, RLO, step, H)
        want = [n2[k - 1] * power(spec, g["r"] * k / H, g["z"] * k / H) for k in range(1, H + 1)]
        assert np.allclose(g["harm_power"][:H], want, rtol=3e-7, atol=1e-9), (row, g["r"], g["z"])
        assert np.isclose(g["power"], sum(want), rtol=3e-7, atol=1e-9)


def test_refinement_does_not_lose_power(bank):
    s, spec, d, zmax, nh = bank
    c = cands([(1, 3000.25, 21.0, 1), (2, 9000.0, -44.0, min(nh, 2))])
    o = s.optimize(c, RLO, TOBS, spectra=[(d.data_ptr(), spec.size)])
    for g in o:
        H = int(g["numharm"])
        n2 = O.step_norms(spec, zmax, nh, s.uselen, RLO, int(g["step"]), H)
        at = lambda r, z: sum(n2[k - 1] * power(spec, r * k / H, z * k / H) for k in range(1, H + 1))  # noqa: E731
        best = at(g["r"], g["z"])
        assert best >= at(g["r_grid"], g["z_grid"]) * (1 - 1e-9)


def test_wide_windows_direct_form(bank):
    # f-dots far outside the bank: the second is too wide for the node rule
    # and sends the whole call to the direct form; the results agree with the
    # first call's where both ran
    s, spec, d, _, _ = bank
    sp = [(d.data_ptr(), spec.size)]
    near = cands([(0, 20000.25, 700.0, 1), (1, 30000.5, -44.0, 2)])
    both = cands([(0, 20000.25, 700.0, 1), (1, 30000.5, -44.0, 2), (0, 25000.0, 12000.0, 1)])
    a = s.optimize(near, RLO, TOBS, spectra=sp, refine=False)
    b = s.optimize(both, RLO, TOBS, spectra=sp, refine=False)
    assert np.allclose(a["power"], b["power"][:2], rtol=3e-7)
    assert np.isfinite(b["power"][2]) and b["power"][2] > 0
