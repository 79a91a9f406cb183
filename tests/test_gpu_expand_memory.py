"""Calls whose device memory holds the direct kernels' buffers but not the
expansion's workspace (csrc/fj_expand.cu) beside them: they compute every
column directly and return no error, whatever the order in which the memory
runs out."""
import ctypes
import warnings

import numpy as np
import pytest

import cases
from test_gpu_expand import _case, _run

pytestmark = pytest.mark.gpu
ALLOC = ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_void_p)
FREE = ctypes.CFUNCTYPE(None, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p)


class Budget:
    """The library's allocator, with at most `limit` bytes live."""

    def __init__(self, lib, limit=None):
        import torch
        self.lib, self.live, self.now, self.peak = lib, {}, 0, 0

        def alloc(n, stream, user):
            if limit is not None and self.now + n > limit:
                return None
            t = torch.empty(max(n, 1), dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            self.live[t.data_ptr()] = t
            self.now += n
            self.peak = max(self.peak, self.now)
            return t.data_ptr()

        def free(p, stream, user):
            torch.cuda.synchronize()
            self.now -= self.live.pop(p).numel()

        self.fns = ALLOC(alloc), FREE(free)

    def __enter__(self):
        a, f = (ctypes.cast(x, ctypes.c_void_p) for x in self.fns)
        assert self.lib.ccfj_set_allocator(a, f, None) == 0
        return self

    def __exit__(self, *exc):
        self.lib.ccfj_set_allocator(None, None, None)
        assert not self.live


def _calls(lib):
    """name -> (the call, the same call by the direct kernels)."""
    import ccfj
    case = _case(400, 200, 300, seed=17)
    rng = np.random.default_rng(2)
    rs = [np.sort(rng.uniform(300.0, 8e4, n)) for n in (60, 700, 129, 300)]
    f, c = np.linspace(0.02, 1.2, 130), np.linspace(900.0, 4500.0, 140)
    us = [cases.noise_spectra(rng, r, f, sigma=0.3) for r in rs]

    def forced(call):
        def run():
            try:
                assert lib.ccfj_set_fj_variant(2) == 0
                return call()
            finally:
                lib.ccfj_set_fj_variant(0)
        return run

    def batch(variant=0, func=0):
        return np.stack(ccfj.fj_noise_batch(us, rs, c, f, func=func, variant=variant))

    out = {}
    for name, kw in (("plain", {}), ("two bases", dict(mode=4))):
        call = lambda kw=kw: _run(case, **kw)  # noqa: E731
        out[name] = call, forced(call)
    out["batch"] = batch, lambda: batch(variant=2)
    out["batch hankel"] = lambda: batch(func=1), lambda: batch(variant=2, func=1)
    return out


@pytest.mark.parametrize("name", ["plain", "two bases", "batch", "batch hankel"])
def test_memory_that_ends_between_the_two_needs(lib, name):
    call, direct = _calls(lib)[name]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        with Budget(lib) as all_of_it:
            full = call()
        with Budget(lib) as least:
            plain = direct()
        assert least.peak < all_of_it.peak and not np.array_equal(full, plain)
        # (256 bytes short: the workspace had its place before the last of the
        # direct kernels' buffers)
        top = all_of_it.peak
        for limit in [*np.linspace(least.peak, top, 7).astype(int), top - 256, top - least.peak // 4]:
            with Budget(lib, int(limit)):
                y = call()
            assert np.array_equal(y, full if limit == top else plain), limit


def test_captured_call_near_the_device_s_limit(lib):
    """A caller's graph takes its memory at its launch: a call captured while
    the device has room for the direct kernels alone still runs."""
    import torch
    from ccfj import _lib
    nr, nf, nc = 400, 4000, 300
    rng = np.random.default_rng(23)
    r = np.sort(rng.uniform(500.0, 1e5, nr)).astype(np.float32)
    f, c = np.linspace(0.02, 1.5, nf, dtype=np.float32), np.linspace(800, 4500, nc, dtype=np.float32)
    u = rng.standard_normal((nr, nf)).astype(np.float32)
    T = [torch.from_numpy(x).cuda() for x in (r, f, c, u)]
    out = torch.empty((nc, nf), device="cuda")
    a = _lib.FjArgs()
    a.struct_size = ctypes.sizeof(a)
    a.nr, a.nf, a.nc, a.itype, a.mode, a.normalize, a.device_ptrs = nr, nf, nc, 1, 0, 1, 1
    a.r, a.f, a.c, a.out = T[0].data_ptr(), T[1].data_ptr(), T[2].data_ptr(), out.data_ptr()
    a.u[0], a.u_ld, a.u_rows, a.u_es, a.u_ncols, a.fstride = T[3].data_ptr(), nf, nr, 1, nf, 1

    def captured():
        s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            _lib.check(lib.ccfj_fj_v1(ctypes.byref(a), ctypes.c_void_p(s.cuda_stream)))
        out.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        return out.cpu().numpy()

    def eager():
        out.fill_(float("nan"))
        _lib.check(lib.ccfj_fj_v1(ctypes.byref(a), None))
        torch.cuda.synchronize()
        return out.cpu().numpy()

    full = eager()
    try:
        assert lib.ccfj_set_fj_variant(2) == 0
        direct = eager()
    finally:
        lib.ccfj_set_fj_variant(0)
    # the direct kernels take 26 MB of interval data, the workspace 895 MB
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    rest = torch.empty(free - (450 << 20), dtype=torch.uint8, device="cuda")
    try:
        y = captured()
    finally:
        del rest
        torch.cuda.empty_cache()
    assert np.array_equal(y, direct)
    assert np.array_equal(captured(), full)
