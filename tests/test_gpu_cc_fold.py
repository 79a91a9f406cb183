"""Cross-correlation kernels at the edges of their folds, tiles and shifts,
against the FP64 oracle (oracle/cc_oracle.py)."""
import numpy as np
import pytest

import cc_oracle as C
from test_cc_emul import TOL

pytestmark = pytest.mark.gpu

# nsta, npts, fftlen, steplen, nf, fstride, onebit, whiten
CASES = {
    "fold2_two_points": (3, 40, 8, 4, 2, 2, 0, 0),
    "fold3": (17, 4000, 1440, 360, 241, 3, 0, 1),
    "fold4_odd_start": (16, 3001, 960, 241, 121, 4, 1, 0),
    "fold5_fp64_sum": (5, 6000, 2400, 600, 33, 5, 0, 1),
    "fold_of_a_common_divisor": (4, 5000, 1440, 720, 32, 14, 0, 0),
    "fold_to_two_points": (4, 5000, 1440, 720, 2, 360, 0, 0),
    "last_bin_by_itself": (4, 5000, 1440, 720, 2, 720, 0, 0),
    "stride_without_divisor": (4, 5000, 1440, 720, 90, 7, 0, 0),
    "128_threads_full": (2, 8192, 4096, 1, 65, 1, 0, 0),
    "256_threads_first": (2, 8400, 4320, 4000, 2161, 1, 0, 0),
    "256_threads_full": (2, 16384, 8192, 4096, 1, 1, 0, 0),
    "512_threads_full": (3, 40001, 16384, 8191, 64, 2, 0, 1),
    "direct_padding": (3, 1000, 77, 50, 39, 1, 0, 0),
    "one_shift": (33, 128, 128, 1, 65, 1, 0, 1),
    "odd_shifts": (18, 700, 128, 64, 31, 1, 0, 1),
}


@pytest.mark.parametrize("gaps", [False, True], ids=["all", "gaps"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_cc_edges_match_oracle(name, gaps):
    import ccfj
    nsta, npts, fftlen, step, nf, fstride, onebit, white = CASES[name]
    rng = np.random.default_rng(len(name) + gaps)
    data = rng.standard_normal(nsta * npts).astype(np.float32)
    se = np.tile([0, npts + fftlen], nsta).astype(np.int32)
    pairs = np.array([(a, b) for a in range(nsta) for b in range(nsta) if (a * 7 + b) % 3 or a == b])
    if gaps:  # windows left out at both ends, a station without any, pairs twice
        se = np.stack([rng.integers(0, npts // 3, nsta), npts - rng.integers(0, npts // 3, nsta)], 1)
        se[nsta // 2] = (npts, npts)
        se = se.ravel().astype(np.int32)
        pairs = np.concatenate([pairs, pairs[::2]])
    pairs = pairs.ravel().astype(np.int32)
    overlap = 1 - (step + 0.5) / fftlen  # int(fftlen * (1 - overlap)) = step
    kw = dict(overlaprate=overlap, fstride=fstride, ifonebit=onebit, ifspecwhittenning=white)
    args = (npts, nsta, nf, fftlen, pairs, se)
    got = ccfj.CC(*args, data.copy(), **kw)
    ref = C.CC(*args, data.copy(), **kw)
    scale = np.abs(ref).max(axis=1, keepdims=True)
    none = scale[:, 0] == 0
    assert np.all(got[none] == 0)
    assert gaps or not none.any()
    if not none.all():
        assert (np.abs(got - ref)[~none] / scale[~none]).max() <= TOL
