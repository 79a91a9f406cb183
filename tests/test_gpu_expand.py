"""The wave-cell expansion of the FP32 transform (csrc/fj_expand.cu) where its
tiles, chunks and cells end, against the FP64 station form of the same call.

Tolerance, per column, of its largest value: the 16-term series of a cell is
1e-8 off, the quadrature of an interval 2e-8; coefficients, moments and sums
are FP32, each rounding 6e-8 of its value, and a column adds up to 1e4
roundings of terms that are not larger than its largest value, 6e-6 if they
add like a random walk. TOL doubles their sum.

Calls that the expansion must leave alone (distances out of order, velocities
or frequencies below zero, a forced variant) give the direct kernels' bits.
"""
import ctypes
import warnings

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu
TOL = 1.2e-5
MODES = {"J": 0, "Y": 1, "J-Y": 2, "|J|": 3, "|H|": 4}


def _case(nr, nf, nc, seed=0, rmin=500.0, rmax=1e5, fmin=0.02, fmax=1.5, cmin=800.0):
    rng = np.random.default_rng(seed)
    r = np.sort(rng.uniform(rmin, rmax, nr))
    f = np.linspace(fmin, fmax, nf)
    c = np.linspace(cmin, 4500.0, nc)
    u = cases.noise_spectra(rng, r, np.maximum(f, 1e-3), sigma=0.3, overtone=True)
    return [np.ascontiguousarray(u.real), np.ascontiguousarray(u.imag)], r, c, f


def _run(case, mode=0, itype=1, precision=0, **kw):
    import ccfj
    ins, r, c, f = case
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return ccfj._transform(ins[:1 if mode < 2 else 2], r, c, f, 1, itype, mode,
                               precision=precision, **kw)


def _direct(lib, case, **kw):
    """The direct kernels with the tile choice of an untuned call of these sizes."""
    try:
        assert lib.ccfj_set_fj_variant(2 if kw.get("itype", 1) else 4) == 0
        return _run(case, **kw)
    finally:
        lib.ccfj_set_fj_variant(0)


def _check(y, z):
    assert np.array_equal(np.isnan(y), np.isnan(z))
    top = np.nanmax(np.abs(z), axis=0)
    err = np.nanmax(np.abs(y.astype(np.float64) - z), axis=0) / np.where(top > 0, top, 1)
    assert np.nanmax(err) <= TOL, (int(np.nanargmax(err)), float(np.nanmax(err)))


# pairs around chunk ends, frequencies around tiles of 64 (and 16 and 32),
# velocities around tiles of 128
@pytest.mark.parametrize("nr,nf,nc", [(2, 8191, 513), (3, 4000, 600), (33, 1025, 257),
                                      (64, 513, 255), (65, 511, 385), (129, 641, 128),
                                      (512, 193, 129), (513, 65, 256), (2049, 64, 127),
                                      (4097, 63, 130), (8193, 33, 129), (12000, 17, 131),
                                      (300, 700, 1100)])
@pytest.mark.parametrize("mode,itype", [("J", 1), ("J", 0), ("J-Y", 1), ("|H|", 1), ("|J|", 0)])
def test_sizes_at_tile_ends(lib, nr, nf, nc, mode, itype):
    case = _case(nr, nf, nc, seed=nr)
    y = _run(case, MODES[mode], itype)
    # the columns that the expansion took (few pairs: the others go direct)
    took = np.any(y != _direct(lib, case, mode=MODES[mode], itype=itype), axis=0)
    assert took.any()
    _check(y[:, took], _run(case, MODES[mode], itype, precision=1)[:, took])


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("itype", [0, 1])
def test_intervals_from_ties_to_many_cells(mode, itype):
    """Exact ties, gaps below the 0.1 m floor, gaps of a cell and of hundreds;
    for the J basis a pair at zero distance and (itype 1) a column at f = 0."""
    rng = np.random.default_rng(5)
    r = np.concatenate([rng.uniform(100, 300, 40), np.geomspace(400.0, 9e5, 60), [5e3] * 3,
                        5e3 + np.array([0.03, 0.07, 1.0])])
    if mode in ("J", "|J|"):
        r[0] = 0.0
    r = np.sort(r).astype(np.float32).astype(np.float64)
    f = np.linspace(0.0 if itype == 1 else 0.01, 1.2, 400)
    c = np.geomspace(700.0, 9000.0, 190)
    u = cases.noise_spectra(rng, r, np.maximum(f, 1e-3), sigma=0.3)
    case = ([np.ascontiguousarray(u.real), np.ascontiguousarray(u.imag)], r, c, f)
    _check(_run(case, MODES[mode], itype), _run(case, MODES[mode], itype, precision=1))


def test_distances_on_cell_ends():
    """Stations exactly on, just below and just above cell ends of every
    frequency's grid (all frequencies the same, so the grid is)."""
    rng = np.random.default_rng(6)
    c = np.linspace(1000.0, 4000.0, 300)
    hu = 10.0 / (2 * np.pi) * 1000.0
    ends = (hu * np.arange(1, 120)).astype(np.float32)
    r = np.sort(np.concatenate([ends, np.nextafter(ends, np.float32(0)),
                                np.nextafter(ends, np.float32(1e9))])).astype(np.float64)
    f = np.ones(300)
    u = cases.noise_spectra(rng, r, f, sigma=0.3)
    for itype in (0, 1):
        case = ([np.ascontiguousarray(u.real)], r, c, f)
        _check(_run(case, 0, itype), _run(case, 0, itype, precision=1))


@pytest.mark.parametrize("what", ["unsorted", "velocity", "frequency", "velocity nan"])
def test_left_to_the_direct_kernels(lib, what):
    ins, r, c, f = _case(400, 200, 300, seed=9)
    if what == "unsorted":
        r = r[np.random.default_rng(0).permutation(len(r))]
    elif what == "velocity":
        c = c.copy()
        c[7] = -900.0
    elif what == "velocity nan":
        c = c.copy()
        c[7] = np.nan
    else:
        f = f.copy()
        f[3] = -0.4
    case = (ins, r, c, f)
    y, d = _run(case), _direct(lib, case)
    if what == "frequency":  # one column only
        assert np.array_equal(y[:, 3], d[:, 3], equal_nan=True)
        assert not np.array_equal(y, d, equal_nan=True)
    else:
        assert np.array_equal(y, d, equal_nan=True)


def test_columns_with_too_many_cells_go_direct(lib):
    """12 pairs over 3000 km: the high frequencies cost less directly."""
    case = _case(12, 3000, 400, seed=11, rmax=3e6, fmax=4.0)
    y, d = _run(case), _direct(lib, case)
    same = np.all(y == d, axis=0)
    assert same[-1] and not same[0]
    _check(y[:, ~same], _run(case, precision=1)[:, ~same])


def test_windows_and_nan_columns():
    """A window of the frequencies gives the full call's bits, and a NaN or an
    infinity in one column's spectra stays in that column."""
    case = _case(700, 300, 260, seed=13)
    full = _run(case, normalize=True)
    for a, b in ((0, 65), (65, 130), (130, 300), (40, 41)):
        assert np.array_equal(_run(case, normalize=True, cols=(a, b)), full[:, a:b])
    ins = [case[0][0].copy()]
    ins[0][350, 77] = np.nan
    ins[0][10, 190] = np.inf
    y = _run((ins,) + case[1:], normalize=True)
    assert np.isnan(y[:, 77]).all() and not np.isfinite(y[:, 190]).any()
    keep = np.setdiff1d(np.arange(300), [77, 190])
    assert np.array_equal(y[:, keep], full[:, keep])


def test_without_memory_for_the_expansion(lib):
    """An allocator that refuses the expansion's block: the direct kernels
    compute every column, as in a call that forces their variant."""
    import torch
    case = _case(400, 200, 300, seed=17)
    direct = _direct(lib, case)
    live = {}
    ALLOC = ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_void_p)
    FREE = ctypes.CFUNCTYPE(None, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p)

    def alloc(n, stream, user):
        if n > 400 * 200 * 16:  # the direct kernels' largest block
            return None
        t = torch.empty(max(n, 1), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        live[t.data_ptr()] = t
        return t.data_ptr()

    def free(p, stream, user):
        torch.cuda.synchronize()
        live.pop(p, None)

    a, f = ALLOC(alloc), FREE(free)
    try:
        assert lib.ccfj_set_allocator(ctypes.cast(a, ctypes.c_void_p),
                                      ctypes.cast(f, ctypes.c_void_p), None) == 0
        y = _run(case)
    finally:
        lib.ccfj_set_allocator(None, None, None)
    assert np.array_equal(y, direct) and not live


@pytest.mark.parametrize("func,itype", [(0, 1), (1, 1), (0, 0)])
def test_batch_of_uneven_sets(lib, func, itype):
    """Sets of 1 to 2000 pairs: the large ones within TOL of the FP64 form alone,
    the small ones the direct kernel's bits; a batch with a forced variant keeps
    to the direct kernel."""
    import ccfj
    rng = np.random.default_rng(19)
    f = np.linspace(0.02, 1.2, 130)
    c = np.linspace(900.0, 4500.0, 140)
    rs = [np.sort(rng.uniform(300.0, 8e4, n)) for n in (1, 2, 64, 65, 66, 2000, 129, 700)]
    us = [cases.noise_spectra(rng, r, f, sigma=0.3) for r in rs]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        ys = ccfj.fj_noise_batch(us, rs, c, f, itype=itype, func=func)
        direct = ccfj.fj_noise_batch(us, rs, c, f, itype=itype, func=func, variant=2)
        for u, r, y, d in zip(us, rs, ys, direct):
            assert np.array_equal(np.isnan(y), np.isnan(d))
            if len(r) < 48:
                assert np.array_equal(y, d, equal_nan=True)
                continue
            z = ccfj._transform([u], r, c, f, 1, itype, 2 * func, hilbert=bool(func),
                                perm=np.arange(len(r)), precision=1)
            top = np.abs(z).max(axis=0)
            assert np.abs(y - z / top).max() <= TOL
    assert not all(np.array_equal(y, d, equal_nan=True) for y, d in zip(ys, direct))


def test_many_frequencies():
    """More frequencies than W has room for all cells of: those with many cells
    go direct, in a window of the frequencies as in the whole call."""
    case = _case(400, 9001, 257, seed=17, rmax=1.2e5, fmax=14.0)
    full = _run(case)
    _check(full, _run(case, precision=1))
    for a, b in ((0, 64), (8000, 9001)):
        assert np.array_equal(_run(case, cols=(a, b)), full[:, a:b])
