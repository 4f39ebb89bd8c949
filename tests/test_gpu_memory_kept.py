"""Device memory that a context keeps between calls: lengths of the transform
leave when the kept tables exceed their bound, a length too large to keep
leaves after its call, everything kept goes back when an allocation finds no
memory, and in the server it counts against the HBM budget.

What is kept comes from the device's stream-ordered memory pool, whose bytes in
use and bytes reserved the CUDA driver reports (destroying a context leaves the
former as they were: cudaFree of such memory is not counted there)."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MB = 1 << 20


USED, RESERVED = 7, 5  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT, CU_MEMPOOL_ATTR_RESERVED_MEM_CURRENT


def pool_used(what=USED):
    """Bytes in use (reserved) of the device's default memory pool."""
    cu = C.CDLL("libcuda.so.1")
    dev, pool, used = C.c_int(), C.c_void_p(), C.c_uint64()
    torch.cuda.synchronize()
    assert cu.cuDeviceGet(C.byref(dev), 0) == 0
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0
    assert cu.cuMemPoolGetAttribute(pool, what, C.byref(used)) == 0
    return used.value


def transform(s, x):
    spec = torch.full((x.numel() + 2,), np.nan, device="cuda")
    torch.cuda.synchronize()
    s.rfft(x.data_ptr(), x.numel(), spec.data_ptr())
    s.synchronize()
    return spec


def accurate(spec, x):
    # two single-precision transforms of at most 2^26 points, about 1e-6 of
    # the rms each: 2e-5 is far above the largest of 2^24 bins
    exact = torch.fft.rfft(x.double())
    err = (torch.view_as_complex(spec.view(-1, 2)) - exact).abs().max()
    return bool(err <= 2e-5 * exact.abs().square().mean().sqrt())


def test_lengths_leave_and_come_back():
    from gpu_accelsearch_gb300.search import AccelSearch
    torch.manual_seed(5)
    before, reserved = pool_used(), pool_used(RESERVED)
    # Bluestein lengths of about 100 MB of tables each: five are kept
    xs = [torch.randn(2 * k, device="cuda") for k in (4194301, 4194287, 4194277, 4194271, 4194247, 4194217, 4194199)]
    with AccelSearch(zmax=0, numharm=1, fftlen=128) as s:
        first = [transform(s, x) for x in xs]
        assert accurate(first[0], xs[0])
        assert 400 * MB < pool_used() - before <= (512 + 65) * MB  # tables, and 64 MB of working array
        for i in (6, 0, 1, 6, 3, 0):
            assert torch.equal(transform(s, xs[i]), first[i])
        assert pool_used() - before <= (512 + 65) * MB
        # 671 MB of tables and 512 MB of working array: not kept, and the
        # lengths that are kept stay
        kept = pool_used()
        big = torch.randn(2 * ((1 << 24) + 43), device="cuda")
        a = transform(s, big)
        assert pool_used() - before <= 2 * 512 * MB + 10 * MB
        assert pool_used() >= kept
        assert accurate(a, big)
        assert torch.equal(transform(s, big), a)
        assert torch.equal(transform(s, xs[3]), first[3])
    assert pool_used(RESERVED) <= reserved


def test_given_back_when_memory_runs_out():
    from gpu_accelsearch_gb300.search import AccelSearch
    torch.manual_seed(6)
    n = 1 << 24
    x = torch.randn(n, device="cuda")
    others = [torch.randn(2 * k, device="cuda") for k in (4194301, 4194287, 4194277, 4194271)]
    with AccelSearch(zmax=0, numharm=1, fftlen=8192, sigma=9.0, chunk_segments=64) as s:
        # everything loaded and planned (a power of two and the Bluestein
        # lengths share the plan of 2^23 points), little held yet
        s.search([x.data_ptr()], 1e-3, on_device=True, nsamples=[1 << 16])
        want = transform(s, x)
        for y in others:
            transform(s, y)
        held = pool_used()
        assert held > 400 * MB
        spec = torch.empty(n + 2, device="cuda")
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        fill = []
        try:
            # all but 48 MB: the search's buffers for 2^24 samples are 128 MB
            free = torch.cuda.mem_get_info()[0] - 48 * MB
            while free > 64 * MB:
                step = min(free, 32 << 30)
                fill.append(torch.empty(step // 4, device="cuda"))
                free -= step
            s.search([x.data_ptr()], 1e-3, on_device=True, nsamples=[n])
            assert pool_used() < held
            s.rfft(x.data_ptr(), n, spec.data_ptr())
            s.synchronize()
            assert torch.equal(spec, want)
        finally:
            fill.clear()
            torch.cuda.empty_cache()


def test_new_length_when_memory_runs_out():
    # the tables of a new length (100 MB) take the place of the others'
    from gpu_accelsearch_gb300.search import AccelSearch
    torch.manual_seed(7)
    xs = [torch.randn(2 * k, device="cuda") for k in (4194301, 4194287, 4194277, 4194271)]
    with AccelSearch(zmax=0, numharm=1, fftlen=128) as s:
        want = transform(s, xs[0])
        for x in xs[1:3]:
            transform(s, x)
    with AccelSearch(zmax=0, numharm=1, fftlen=128) as s:
        for x in xs[1:]:
            transform(s, x)
        held = pool_used()
        spec = torch.empty(xs[0].numel() + 2, device="cuda")
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        fill = []
        try:
            free = torch.cuda.mem_get_info()[0] - 48 * MB
            while free > 64 * MB:
                step = min(free, 32 << 30)
                fill.append(torch.empty(step // 4, device="cuda"))
                free -= step
            s.rfft(xs[0].data_ptr(), xs[0].numel(), spec.data_ptr())
            s.synchronize()
            assert torch.equal(spec, want)
            assert pool_used() <= held
        finally:
            fill.clear()
            torch.cuda.empty_cache()


def test_server_counts_it_against_its_budget():
    from gpu_accelsearch_gb300.serving import Server
    rng = np.random.default_rng(8)
    before = pool_used()
    # about 3 MB of tables and 2 MB of working array per length, eight lengths;
    # a request is 1.6 MB
    lengths = [2 * k for k in (100003, 100019, 100043, 100049, 100057, 100069, 100103, 100109)]
    budget = 8e6
    with Server(hbm_budget_bytes=budget, fftlen=2048, numharm=2, sigma=8.0, chunk_segments=8) as srv:
        ids = [srv.submit(rng.standard_normal(n).astype(np.float32), 1e-3, 20) for n in lengths]
        for i in ids:
            assert srv.wait(i, 60.0)
            srv.result(i)
        # (and 64 whitening plans at most, some 40 KB each)
        assert pool_used() - before <= budget + 1e6
