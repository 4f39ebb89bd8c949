"""Lists of candidates for refinement: a candidate's result does not depend on
what else is in the list (windows too wide for the node rule take the direct
form each for itself; long lists go in several launches), and the direct form
itself, grids included, against the closed form.

Closed form of the response: completing the square,
    F(x; z) = exp(-i pi x^2 / z) / sqrt(2 z) [Fr(s (1 + x / z)) - Fr(s x / z)],
s = sqrt(2 z), Fr the Fresnel integral C + i S, for z > 0, and F(x; -z) =
conj(F(-x; z)).  Its phases reach 4e3 radians and more (error 1e-12); the
device rounds the power once to float: 6e-8 relative, tested at 3e-7."""
import numpy as np
import pytest

from oracle import oracle as O

torch = pytest.importorskip("torch")
special = pytest.importorskip("scipy.special")
pytestmark = pytest.mark.gpu

N, RLO, TOBS, ZMAX, NH = 1 << 17, 16, 10.0, 50, 4


def response(x, z):
    if z < 0:
        return np.conj(response(-x, -z))
    s = np.sqrt(2 * z)
    (s1, c1), (s0, c0) = special.fresnel(s * (1 + x / z)), special.fresnel(s * x / z)
    return np.exp(-1j * np.pi * x * x / z) / s * ((c1 - c0) + 1j * (s1 - s0))


def power(spec, r, z):
    hw = O.z_halfwidth(z)
    j = np.arange(int(np.ceil(r)) - hw, int(np.ceil(r)) + hw)
    j = j[(j >= 0) & (j < spec.size)]
    return abs(np.sum(spec[j].astype(np.complex128) * np.conj(response(r - j - z / 2, z)))) ** 2


@pytest.fixture(scope="module")
def bank():
    from gpu_accelsearch_gb300.search import AccelSearch
    rng = np.random.default_rng(12)
    spec = (rng.standard_normal(N // 2) + 1j * rng.standard_normal(N // 2)).astype(np.complex64)
    with AccelSearch(zmax=ZMAX, numharm=NH, fftlen=2048, chunk_segments=4) as s:
        d = torch.from_numpy(spec.view(np.float32).copy()).cuda()
        torch.cuda.synchronize()
        yield s, spec, [(d.data_ptr(), spec.size)]


def cands(rows):
    from gpu_accelsearch_gb300.search import CAND_DTYPE
    c = np.zeros(len(rows), CAND_DTYPE)
    for i, (step, r, z, nh) in enumerate(rows):
        c[i] = (0, step, r, z, nh, 30.0, 6.0)
    return c


# (the direct form takes |z| < 1e-4 for 0, the node rule does not: which of
# the two ran shows in the first two candidates' powers)
NEAR = [(0, 20000.4, 9.9e-5, 1), (2, 30000.3, -9.9e-5, 4), (1, 30000.5, -44.0, 2), (3, 41000.25, 700.0, 1),
        (0, 17.5, 3.0, 4), (4, N // 2 - 0.5, 21.3, 1)]
WIDE = [(0, 25000.0, 12000.0, 1), (1, 33000.75, -9100.5, 1), (2, N // 2 - 900.0, 19000.0, 2)]


@pytest.mark.parametrize("refine", [False, True])
def test_results_do_not_depend_on_the_list(bank, refine):
    s, _, sp = bank
    alone = np.concatenate([s.optimize(cands([row]), RLO, TOBS, spectra=sp, refine=refine) for row in NEAR + WIDE])
    order = [6, 0, 3, 7, 1, 2, 8, 4, 5]
    mixed = s.optimize(cands([(NEAR + WIDE)[i] for i in order]), RLO, TOBS, spectra=sp, refine=refine)
    assert mixed.tobytes() == alone[order].tobytes()


@pytest.mark.parametrize("refine", [False, True])
def test_long_lists(bank, refine):
    # 33000 one-panel candidates and more: three launches' worth of nodes
    s, _, sp = bank
    rng = np.random.default_rng(3)
    rows = [(int(rng.integers(5)), float(rng.uniform(100, N // 2 - 100)), float(rng.uniform(-60, 60)),
             int(rng.choice([1, 2, 4]))) for _ in range(97)]
    one = s.optimize(cands(rows), RLO, TOBS, spectra=sp, refine=refine)
    many = s.optimize(np.tile(cands(rows), 400), RLO, TOBS, spectra=sp, refine=refine)
    assert many.tobytes() == np.tile(one, 400).tobytes()


def test_direct_form(bank):
    s, spec, sp = bank
    norms = {}

    def summed(row, r, z):
        step, _, _, H = row
        n2 = norms.setdefault((step, H), O.step_norms(spec, ZMAX, NH, s.uselen, RLO, step, H))
        return [n2[k - 1] * power(spec, r * k / H, z * k / H) for k in range(1, H + 1)]

    flat = s.optimize(cands(WIDE), RLO, TOBS, spectra=sp, refine=False)
    best = s.optimize(cands(WIDE), RLO, TOBS, spectra=sp, refine=True)
    for row, a, b in zip(WIDE, flat, best):
        _, r, z, H = row
        want = summed(row, r, z)
        assert (a["r"], a["z"]) == (r, z)
        assert np.allclose(a["harm_power"][:H], want, rtol=3e-7) and np.isclose(a["power"], sum(want), rtol=3e-7)
        # the three nested 5 x 5 grids around the best point so far
        for lv in range(3):
            dr = 0.25 / 4 ** lv
            grid = [(r + (g // 5 - 2) * dr, z + (g % 5 - 2) * 4 * dr) for g in range(25)]
            p = [sum(summed(row, *at)) for at in grid]
            g = int(np.argmax(p))
            assert sorted(p)[-1] > sorted(p)[-2] * (1 + 1e-9)  # no tie that rounding could decide
            r, z = grid[g]
        assert (b["r"], b["z"]) == (r, z)
        want = summed(row, r, z)
        assert np.allclose(b["harm_power"][:H], want, rtol=3e-7) and np.isclose(b["power"], sum(want), rtol=3e-7)


# widths on either side of the two forms' limits (z about 152 for one point,
# 2070 with the grids) and of the window that is staged in shared memory
@pytest.mark.parametrize("refine", [False, True])
@pytest.mark.parametrize("z", [140.0, 150.0, 153.0, 156.0, 160.0, 1900.0, 2040.0, 2065.0, 2075.0, 2100.0, 2700.0])
def test_either_side_of_the_limits(bank, z, refine):
    s, spec, sp = bank
    rows = [(1, 30000.3, z, 1), (2, 41000.5, -z, 2)]
    for (step, r, zz, H), o in zip(rows, s.optimize(cands(rows), RLO, TOBS, spectra=sp, refine=refine)):
        assert abs(o["r"] - r) <= 0.65626 * refine and abs(o["z"] - zz) <= 2.6251 * refine
        n2 = O.step_norms(spec, ZMAX, NH, s.uselen, RLO, step, H)
        want = [n2[k - 1] * power(spec, o["r"] * k / H, o["z"] * k / H) for k in range(1, H + 1)]
        assert np.allclose(o["harm_power"][:H], want, rtol=3e-7) and np.isclose(o["power"], sum(want), rtol=3e-7)
