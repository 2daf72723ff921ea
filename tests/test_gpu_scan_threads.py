"""FFT scans of different transform sizes from several host threads, a handle
each: the short transforms' dynamic shared memory (48 bytes a point of a part,
1.5 to 192 KB) is an attribute of the kernel that all handles share, so that a
small scan must not take it from a large one between its setting and its
launch.  Every scan equals the one a thread makes alone, bit for bit."""
import threading

import numpy as np
import pytest

from clblm_gb300 import capi_types as T
from clblm_gb300 import synth

pytestmark = pytest.mark.gpu


def test_scans_of_different_sizes_in_threads(gpu_lib):
    rng = np.random.default_rng(5)
    # M = 131072 blocks (parts of 4096 points), and M = 8192 (parts of 256)
    cases = [(4300000, 2e-4, 0.26, 120)] + [(50001, 0.002, 0.6, 1500)] * 3
    work = []
    for n, dv, hw, count in cases:
        x = 1.0 + rng.uniform(-0.5, 0.5, n)
        sc = T.scan_struct(5, hw, 1000.0 + 0.4 * dv * n, 1000.0 + 0.6 * dv * n)
        h = gpu_lib.Handle(synth.line_list(1000, 600.0, 700.0, seed=0))
        work.append((h, sc, x, dv, count, h.fftscn(sc, x, 1000.0, dv)[0]))
    failed, done = [], threading.Event()
    start = threading.Barrier(len(work))

    def scan(i):
        h, sc, x, dv, count, want = work[i]
        start.wait()
        try:
            for _ in range(count):
                got, _, _ = h.fftscn(sc, x, 1000.0, dv)
                if not np.array_equal(got, want):
                    failed.append("thread %d: another result" % i)
                    break
                if done.is_set():
                    break
        except Exception as e:  # noqa: BLE001 (reported below)
            failed.append("thread %d: %s" % (i, e))
        done.set() if i == 0 or failed else None

    threads = [threading.Thread(target=scan, args=(i,)) for i in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w in work:
        w[0].close()
    assert not failed, failed
