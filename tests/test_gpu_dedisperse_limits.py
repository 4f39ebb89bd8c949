"""The windowed dedispersion at its limits, bit-exact against the oracle: the
widest delay spread each tile height takes (1309, 1313 and 1317 samples for
16, 8 and 4 trials) and the next, with rows of every alignment (remainders of
0 to 3 samples), and the outcome when a window's copies do not land within
their bounded wait: the tile is summed from global memory.

The waits are made to run out by expecting 16 bytes that never arrive; every
wait ends by its own limit."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O

torch = pytest.importorskip("torch")

TILE, LIMIT = 1024, 110 * 1024  # output samples of a tile, shared memory of a CTA


def chosen(delays):
    """The tile height the host chooses, 0 for the one-load-per-addition
    kernel (restated: three stages of four channels, the height of least
    padding and copying among those that fit)."""
    best = (0, 0.0)
    for d in (16, 8, 4):
        spread = max(int((t.max(0) - t.min(0)).max()) for t in
                     (delays[i:i + d] for i in range(0, len(delays), d)))
        wlen = (TILE + spread + 6) & ~3
        if 4 * (spread + 3) > 65535 or 48 * wlen + 24 * d > LIMIT:
            continue
        cost = -(-len(delays) // d) * d * (1 + wlen / (TILE * d))
        if not best[0] or cost < best[1]:
            best = (d, cost)
    return best[0]


def alternating(nchan, ndm, spread):
    """Delays 0 and `spread` in turn: the same spread at every tile height."""
    return np.where(np.arange(ndm)[:, None] % 2 == 1, spread, 0).astype(np.int32) * np.ones((1, nchan), np.int32)


def run(delays, nout, seed, call="accel_dedisperse", offset=0):
    from gpu_accelsearch_gb300 import native as N
    ndm, nchan = delays.shape
    nsamp = nout + int(delays.max())
    nsamp += (1 - nsamp) % 4  # rows start at every remainder modulo 4
    fb = np.random.default_rng(seed).standard_normal((nchan, nsamp)).astype(np.float32)
    d_fb = torch.empty(nchan * nsamp + offset, dtype=torch.float32, device="cuda")
    d_fb[offset:] = torch.from_numpy(fb.reshape(-1)).cuda()
    d_out = torch.full((ndm, nout), np.nan, dtype=torch.float32, device="cuda")
    dl = np.ascontiguousarray(delays, np.int32)
    torch.cuda.synchronize()
    N.check(getattr(N.lib(), call)(d_fb.data_ptr() + 4 * offset, nchan, nsamp, dl.ctypes.data_as(C.POINTER(C.c_int)),
                                   ndm, d_out.data_ptr(), nout, None))
    torch.cuda.synchronize()
    want = O.dedisperse(fb, delays, nout)
    assert np.array_equal(d_out.cpu().numpy().view(np.uint32), want.view(np.uint32))


# (trials, spread, tile height: 0 is the one-load-per-addition kernel)
SPREADS = [(16, 1309, 16), (16, 1310, 8), (8, 1309, 8), (8, 1313, 8), (8, 1314, 4), (4, 1313, 4), (4, 1317, 4),
           (4, 1318, 0), (16, 1318, 0), (33, 1309, 8), (47, 1309, 16)]


@pytest.mark.parametrize("ndm,spread,height", SPREADS)
def test_height_chosen(ndm, spread, height):
    assert chosen(alternating(5, ndm, spread)) == height


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 3])
@pytest.mark.parametrize("ndm,spread,height", SPREADS)
def test_widest_windows(ndm, spread, height, offset):
    run(alternating(9, ndm, spread), 2051, ndm + spread, offset=offset)


# one to five stages of channels, a whole and a ragged time tile
@pytest.mark.gpu
@pytest.mark.parametrize("nchan", [1, 5, 18])
@pytest.mark.parametrize("ndm", [16, 7, 3])
def test_copies_that_do_not_land(ndm, nchan):
    delays = np.random.default_rng(ndm).integers(0, 300, (ndm, nchan)).astype(np.int32)
    for call in ("accel_dedisperse_wait_test", "accel_dedisperse"):
        run(delays, 1500, nchan, call)
