"""GPU: the top-m selection of the FP16 scores (cjx_ncc_topk) at the sizes where a warp's list can go wrong.

The scores are exact in single precision (den = 1), so the oracle is a stable sort: descending score, lower index
first on ties.  No tolerance: the outputs are indices.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,m", [(T, m) for T in (3, 31, 32, 33, 127, 128, 1023, 1025, 5000) for m in (1, 3, 8, 16)
                                 if m <= T])
@pytest.mark.parametrize("kind", ["random", "ties", "descending", "ascending", "zero den"])
def test_topk_matches_stable_sort(cuda_device, T, m, kind):
    import torch

    from cryojax_b200 import _native as nat

    rng = np.random.default_rng(T * 17 + m)
    n = 3
    if kind == "ties":
        num = rng.integers(0, 4, (n, T)).astype(np.float32)
    elif kind == "descending":
        num = np.tile(np.arange(T, 0, -1, dtype=np.float32), (n, 1))
    elif kind == "ascending":
        num = np.tile(np.arange(T, dtype=np.float32), (n, 1))
    else:
        num = rng.standard_normal((n, T)).astype(np.float32)
    den = np.ones((n, T), np.float32)
    if kind == "zero den":  # a zero denominator scores 0
        den[:, ::3] = 0.0
    score = np.where(den > 0, num, 0.0)
    t = lambda a: torch.as_tensor(a, device=cuda_device)
    one = torch.ones(n, dtype=torch.float32, device=cuda_device)
    idx = torch.empty((n, m), dtype=torch.int32, device=cuda_device)
    nat.ncc_topk(t(num), t(den), n, T, one, one, one, m, idx)
    got = idx.cpu().numpy()
    for b in range(n):
        np.testing.assert_array_equal(got[b], np.lexsort((np.arange(T), -score[b]))[:m])
