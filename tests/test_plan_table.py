"""CPU: FFT plans are searched once per process and length, by whichever thread comes first.  Eight threads that ask
for the workspaces of all sides at once get what a single thread gets."""

import sys
from concurrent.futures import ThreadPoolExecutor

from cryojax_b200 import _native as nat

SIDES = [*range(2, 200), 360, 509, 512, 720, 997, 1000, 1021, 1023, 1024]


def _sizes(_):
    return [nat.workspace_size(nat.make_desc(n, max(2, n // 2), max(2, n // 3), 0, 0j, 1), 3) for n in SIDES]


def test_threads_agree():
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        with ThreadPoolExecutor(8) as pool:
            results = list(pool.map(_sizes, range(16)))
    finally:
        sys.setswitchinterval(interval)
    assert all(r == _sizes(None) for r in results)
