"""The expansion (csrc/fj_expand.cu) with stations at cell ends where chunks of
stations begin and end, against the FP64 station form of the same call.

The stations at the chunk ends are picked so that at one of the call's
frequencies the float product that names the cell lies one spacing below a
whole number that the exact product has reached (cell_carries of
cell_rule_check.cpp). A chunk that counts such a station to another cell than
its neighbour does loses a cell: 2e-3 and more of that column's largest value.
TOL is derived in test_gpu_expand.py.
"""
import numpy as np
import pytest

import cases
from test_cell_rule import load_rule
from test_gpu_expand import MODES, TOL, _run

pytestmark = pytest.mark.gpu
CMIN, RMAX = 500.0, 3e5


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    return load_rule(tmp_path_factory.mktemp("cell"))


def _carries(rule, f, r0, r1):
    out = np.zeros(1000, dtype=np.float32)
    return out[:rule.cell_carries(f, CMIN, r0, r1, len(out), out.ctypes.data)].copy()


def _check(case, mode, itype):
    y, z = _run(case, MODES[mode], itype), _run(case, MODES[mode], itype, precision=1)
    top = np.abs(z).max(axis=0)
    err = np.abs(y.astype(np.float64) - z).max(axis=0) / top
    assert err.max() <= TOL, (int(err.argmax()), float(err.max()))


def _case(rng, r, f):
    r = r.astype(np.float64)
    u = cases.noise_spectra(rng, r, f.astype(np.float64), sigma=0.3)
    return ([np.ascontiguousarray(u.real), np.ascontiguousarray(u.imag)], r,
            np.linspace(CMIN, 4500.0, 97), f.astype(np.float64))


# numbers of pairs whose chunks have 4, 8, 16, 32, 64 and 128 stations
@pytest.mark.parametrize("nr,chunk", [(121, 4), (1017, 8), (2033, 16), (4065, 32), (8129, 64),
                                      (9217, 128)])
@pytest.mark.parametrize("mode,itype", [("J", 1), ("J", 0), ("|H|", 1), ("J-Y", 0)])
def test_chunks_that_end_on_cell_ends(rule, nr, chunk, mode, itype):
    rng = np.random.default_rng(nr)
    f = np.linspace(0.6, 1.3, 700).astype(np.float32)
    found = np.unique(np.concatenate([_carries(rule, fk, 2e4, RMAX) for fk in f]))
    found = found[np.concatenate([[True], np.diff(found) > 5.0])]
    nch = (nr - 1) // chunk
    assert len(found) > nch
    ends = np.sort(rng.choice(found, nch + 1, replace=False))  # the first station, then chunks' last
    r = [np.concatenate([np.sort(rng.uniform(a + 0.1, b - 0.1, chunk - 1)), [b]])
         for a, b in zip(ends[:-1], ends[1:])]
    r = np.concatenate([ends[:1]] + r).astype(np.float32)
    assert len(r) == nr and np.all(np.diff(r) >= 0) and np.array_equal(r[::chunk], ends)
    _check(_case(rng, r, f), mode, itype)


@pytest.mark.parametrize("mode,itype", [("J", 1), ("J", 0), ("J-Y", 1), ("|H|", 0)])
def test_last_station_on_the_plan_s_last_cell_end(rule, mode, itype):
    """The highest frequency of the first tile (128 columns) begins a group of
    cells with the last station alone: the tile's cells end one group further."""
    rng = np.random.default_rng(3)
    lead = 23 if MODES[mode] in (1, 2, 4) else 0  # halved cells before the first one
    for _ in range(4000):
        f = np.linspace(0.6, rng.uniform(0.9, 1.1), 256).astype(np.float32)
        r = next((float(x) for x in _carries(rule, f[127], 2e5, RMAX)
                  if (rule.cell_locate(x, f[127], CMIN, 0) + lead) % 4 == 0), None)
        if r:
            break
    assert r
    rs = np.concatenate([np.sort(rng.uniform(2e4, r - 50.0, 600)), [r]]).astype(np.float32)
    _check(_case(rng, rs, f), mode, itype)


@pytest.mark.parametrize("mode,itype", [("J", 1), ("J", 0), ("|J|", 1)])
def test_distances_on_cell_ends_of_many_frequencies(rule, mode, itype):
    """Stations on, just below and just above the cell ends of 40 frequencies of
    the call's 600, and each of those frequencies among its neighbours."""
    rng = np.random.default_rng(6)
    f = np.linspace(0.3, 1.4, 600).astype(np.float32)
    ends = np.concatenate([(rule.cell_hu(CMIN) * rng.choice(np.arange(1, 90), 12, replace=False)) / fk
                           for fk in f[::15].astype(np.float64)]).astype(np.float32)
    r = np.sort(np.concatenate([ends, np.nextafter(ends, np.float32(0)),
                                np.nextafter(ends, np.float32(1e9))]))
    _check(_case(rng, r, f), mode, itype)


# sizes near the line between the two ways, where a problem's upper frequencies
# go direct: few pairs and many cells, few velocities, both rules, both bases
@pytest.mark.parametrize("nr,nf,nc,mode,itype", [(62, 289, 53, "J", 1), (40, 658, 260, "J", 1),
                                                 (257, 700, 23, "J-Y", 0), (57, 900, 508, "J", 0),
                                                 (117, 745, 288, "|J|", 1), (83, 500, 77, "|H|", 1)])
def test_windows_decide_as_the_whole_problem(nr, nf, nc, mode, itype):
    rng = np.random.default_rng(nr)
    r = np.sort(rng.uniform(500.0, RMAX, nr))
    f = np.linspace(0.01, 1.8, nf)
    u = cases.noise_spectra(rng, r, f, sigma=0.3)
    case = ([np.ascontiguousarray(u.real), np.ascontiguousarray(u.imag)], r,
            np.linspace(700.0, 4500.0, nc), f)
    full = _run(case, MODES[mode], itype, normalize=True)
    for a, b in ((0, 1), (1, 130), (130, 131), (131, nf)):
        assert np.array_equal(_run(case, MODES[mode], itype, normalize=True, cols=(a, b)),
                              full[:, a:b])
