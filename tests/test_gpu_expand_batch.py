"""Which columns of a batch the expansion (csrc/fj_expand.cu) takes is decided
set by set: by the set and the sizes of the whole batch, not by what the other
sets or the other groups of a host batch ask for."""
import ctypes
import warnings

import numpy as np
import pytest

from test_gpu_expand import MODES, TOL

pytestmark = pytest.mark.gpu


class Batch:
    """A batch on the device, its spectra the real parts of complex rows."""

    def __init__(self, counts, nf, nc, rmax=3e5, seed=0, shuffle=()):
        import torch
        g = torch.Generator(device="cuda").manual_seed(seed)
        rng = np.random.default_rng(seed)
        self.rs = [np.sort(rng.uniform(5e2, rmax, n)).astype(np.float32) for n in counts]
        for b in shuffle:
            rng.shuffle(self.rs[b])
        self.off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
        self.f = np.linspace(0.01, 1.0, nf, dtype=np.float32)
        self.c = np.linspace(1000.0, 5000.0, nc, dtype=np.float32)
        self.u = torch.randn((int(self.off[-1]), nf), generator=g, device="cuda",
                             dtype=torch.complex64)

    def run(self, lib, sets=None, variant=0, itype=1, mode="J"):
        """[set][c][f] of the sets [sets[0], sets[1]) as a device-resident call."""
        import torch
        from ccfj import _batch, _lib
        b0, b1 = sets or (0, len(self.rs))
        o0, o1 = int(self.off[b0]), int(self.off[b1])
        T = [torch.from_numpy(x).cuda() for x in (self.off[b0:b1 + 1] - o0,
                                                  np.concatenate(self.rs[b0:b1]), self.f, self.c)]
        u = self.u[o0:o1]
        out = torch.empty((b1 - b0, len(self.c), len(self.f)), device="cuda")
        a = _batch.BatchArgs()
        a.struct_size = ctypes.sizeof(a)
        a.nsets, a.nf, a.nc, a.itype, a.mode = b1 - b0, len(self.f), len(self.c), itype, MODES[mode]
        a.normalize, a.device_ptrs, a.variant, a.total_pairs = 1, 1, variant, o1 - o0
        a.offsets, a.r, a.f, a.c = (t.data_ptr() for t in T)
        a.u[0], a.u[1] = u.data_ptr(), u.data_ptr() + 4
        a.u_ld, a.u_rows, a.u_es, a.u_ncols, a.fstride = 2 * len(self.f), o1 - o0, 2, len(self.f), 1
        a.out = out.data_ptr()
        _lib.check(lib.ccfj_fj_batch_v1(ctypes.byref(a), None))
        torch.cuda.synchronize()
        return out.cpu().numpy()


@pytest.mark.parametrize("mode,itype", [("J", 1), ("|J|", 0)])
def test_many_sparse_sets(lib, mode, itype):
    """Sets of 50 to 200 pairs, whose cells take three times their interval data
    and more: the expansion takes them all the same."""
    rng = np.random.default_rng(1)
    batch = Batch(rng.integers(50, 200, 128), 512, 200)
    y = batch.run(lib, itype=itype, mode=mode)
    direct = batch.run(lib, variant=2, itype=itype, mode=mode)
    took = np.any(y != direct, axis=(1, 2))
    assert took.all()
    # either way is within TOL of the FP64 form
    assert np.abs(y.astype(np.float64) - direct).max() <= 2 * TOL


def test_a_set_out_of_order_leaves_the_others(lib):
    counts = [120, 300, 64, 900, 75]
    sorted_, mixed = Batch(counts, 300, 150, seed=5), Batch(counts, 300, 150, seed=5, shuffle=[1])
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        y, z = sorted_.run(lib), mixed.run(lib)
        direct = mixed.run(lib, variant=2)
    assert np.array_equal(z[1], direct[1], equal_nan=True)
    for b in (0, 2, 3, 4):
        assert np.array_equal(y[b], z[b]) and not np.array_equal(z[b], direct[b])


def test_host_batch_in_groups_equals_the_device_batch(lib):
    """200 sets x 400 pairs x 512 frequencies (327 MB: a host batch runs in
    groups). All cells together are more than the interval data and 64 MiB, each
    group's are less."""
    import ccfj
    batch = Batch([400] * 200, 512, 64, seed=7)
    dev = batch.run(lib)
    assert not np.array_equal(dev[0], batch.run(lib, sets=(0, 2), variant=2)[0])
    u = batch.u.cpu().numpy()
    us = [u[a:b] for a, b in zip(batch.off[:-1], batch.off[1:])]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        host = ccfj.fj_noise_batch(us, [r.astype(np.float64) for r in batch.rs],
                                   batch.c.astype(np.float64), batch.f.astype(np.float64))
    assert all(np.array_equal(h, d) for h, d in zip(host, dev))
