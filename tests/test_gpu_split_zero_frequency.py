"""A column at f = 0 in a split launch of the direct kernels: the sum of the
trapezoid form (J0(0) = 1), as the unsplit launch and the FP64 form give it, and
NaN for the integral form."""
import numpy as np
import pytest

from test_gpu_expand import MODES, _case, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("itype", [0, 1])
@pytest.mark.parametrize("normalize", [False, True])
def test_zero_frequency_of_a_split_launch(lib, mode, itype, normalize):
    ins, r, c, f = _case(200, 70, 60, seed=3)
    f = f.copy()
    f[0] = 0.0
    kw = dict(mode=MODES[mode], itype=itype, normalize=normalize)
    out = []
    for split in (1, 3):
        try:
            assert lib.ccfj_set_fj_split(split) == 0
            out.append(_run((ins, r, c, f), **kw))
        finally:
            lib.ccfj_set_fj_split(0)
    z = _run((ins, r, c, f), precision=1, **kw)
    for y in out:
        assert np.array_equal(np.isnan(y), np.isnan(z)) and np.array_equal(np.isinf(y), np.isinf(z))
        if itype == 0 and mode in ("J", "|J|"):
            # FP32 sums of 200 terms of one sign or another: 200 roundings of 6e-8
            # of the sum of the terms' values, at most ten times the column here
            assert np.isfinite(y[:, 0]).all()
            assert np.abs(y[:, 0] - z[:, 0]).max() <= 200 * 6e-8 * 10 * np.abs(z[:, 0]).max()
