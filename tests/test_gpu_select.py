"""The exact selection that gives every segment its median
(block_select_reg), bit for bit against a sort: every CTA width in use,
1 to 16 keys a thread, the smallest, middle and largest rank; exponential
powers, ties, keys that differ in the last bit only, all equal, all zero, a
single zero, infinities and NaN, any 32 bits."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    from gpu_accelsearch_gb300 import build as B
    so = str(tmp_path_factory.mktemp("select") / "select.so")
    subprocess.run([B.nvcc(), *B._flags(), "-shared", "-o", so, os.path.join(HERE, "cu", "select_harness.cu")],
                   check=True)
    return C.CDLL(so)


def sets(n, rng):
    f = lambda a: np.asarray(a, np.float32).view(np.uint32)  # noqa: E731
    power = f(rng.exponential(1.0, n))
    one = np.uint32(0x3f800000)
    special = power.copy()
    special[rng.random(n) < 0.3] = 0x7f800000
    special[rng.random(n) < 0.1] = 0x7fffffff
    zero = power.copy()
    zero[rng.integers(n)] = 0
    zeros = np.zeros(n, np.uint32)
    few = zeros.copy()
    few[rng.integers(n)] = rng.integers(1, 1 << 20)
    return [power, f(rng.exponential(1.0, n) * 2.0 ** rng.integers(-120, 100, n)), f(rng.integers(1, 4, n)),
            one + rng.integers(0, 2, n).astype(np.uint32), one + rng.integers(0, 3, n).astype(np.uint32),
            np.full(n, one), zeros, few, zero, special,
            rng.integers(0, 0x7fffffff, n).astype(np.uint32), rng.integers(0, 0xfffffffe, n).astype(np.uint32)]


@pytest.mark.parametrize("nt", [32, 64, 256, 512])
def test_against_a_sort(harness, nt):
    rng = np.random.default_rng(nt)
    keys, ns, ks, want = [], [], [], []
    for n in sorted({1, 2, 3, 5, 31, 32, 33, nt - 1, nt, nt + 1, 5 * nt + 7, 16 * nt - 1, 16 * nt}):
        for own in sets(n, rng):
            for k in {0, (n - 1) // 2, n // 2, n - 1}:
                row = np.full(16 * nt, 0xffffffff, np.uint32)
                row[:n] = own
                keys.append(row)
                ns.append(n)
                ks.append(k)
                want.append(np.sort(own)[k])
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()  # noqa: E731
    d_keys, d_n, d_k = dev(np.stack(keys)), dev(np.array(ns, np.int32)), dev(np.array(ks, np.int32))
    out = torch.zeros((len(ns), nt), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert harness.select_run(nt, p(d_keys), p(d_n), p(d_k), p(out), len(ns)) == 0
    got = out.cpu().numpy().view(np.uint32)
    bad = np.nonzero((got != np.array(want, np.uint32)[:, None]).any(1))[0]
    assert bad.size == 0, [(ns[i], ks[i], hex(want[i]), hex(got[i, 0])) for i in bad[:5]]
