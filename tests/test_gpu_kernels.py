"""Kernels at the sizes where their splits can go wrong.

Tolerances: the Poisson solve keeps test_gpu_parity's 1e-12, or the growth of
a rounding through the stiffest y system (condition about ny^2) where that is
larger; steps keep 1e-10; the FP32 form keeps test_gpu_fp32's bounds.  Copies
are exact.
"""
import numpy as np
import pytest

from oracle import oracle_lib as ol
from paratc_b200 import cases
from paratc_b200.abi import FT_CH, FT_HC
from paratc_b200.lib import ChannelSystem, ParatcError

from .helpers import fields_of, rel_err, scalar_opts, yp_of

pytestmark = pytest.mark.gpu

TOL_STEP1 = 1e-10
FP32_VEL = 1e-5
FP32_PR = 1e-3


def tol_poisson(ny):
    return max(1e-12, 2.0 ** -52 * ny * ny)


def _half(nx, ny, nz):
    return cases.small_channel(nx, ny, nz, flow_type=FT_HC, xnu=1e-3, yly=1.0, is_ux_const=0,
                               scalar=scalar_opts((-3, -2), 0.02, 1.0, (0.087, -0.996, 0.0)))


def _any(nx, ny, nz, **kw):
    """A closed channel, or where ny is odd, which it refuses, a half channel."""
    return cases.small_channel(nx, ny, nz, flow_type=FT_HC if ny % 2 else FT_CH, **kw)


def _source(case):
    return cases.gaussian_source(cases.Case("src", case.params, case.mesh, "gauss_src", 5, 1.0))


def _stepped(case, prec="fp64", schedule=None):
    """Fields after one step from a projected state."""
    yp = yp_of(case)
    f = fields_of(case, yp)
    with ChannelSystem(case.params, yp) as g:
        if schedule is not None:
            g.schedule = schedule
        g.set_fields(f["ux"], f["uy"], f["uz"], f["p"], f["c"])
        g.project()
        g.precision = prec
        g.iterate(1, raise_on_guard=False)
        return g.get_fields(("ux", "uy", "uz", "p", "c"))


def _close(a, b, vel, pr):
    for n in a:
        e = rel_err(a[n], b[n])
        assert e <= (pr if n == "p" else vel), "%s rel err %.3e" % (n, e)


# ny: the smallest, odd, a multiple and one off a multiple of the eight rows a
# sweep reads ahead, tall; nx / 2 + 1: a multiple of the eight modes of an
# item and remainders 1 and 7; nz / 2 its own mirror plane or between two
@pytest.mark.parametrize("dims", [(16, 4, 8), (30, 9, 10), (12, 16, 12), (32, 17, 18), (16, 33, 4), (24, 256, 8)])
def test_two_ended_y_solve(dims):
    case = _any(*dims)
    yp = yp_of(case)
    src = _source(case)
    with ChannelSystem(case.params, yp) as g:
        assert rel_err(g.poisson(src), ol.Oracle(case.params, yp).poisson(src)) <= tol_poisson(dims[1])


FP32_DIMS = [(24, 7, 12), (32, 16, 8)]  # lengths that the FP32 form takes


# nx nz columns: a multiple of the 32 of an item, remainders, fewer than one;
# with and without the scalar of the same launch
@pytest.mark.parametrize("make", [_any, _half])
@pytest.mark.parametrize("dims", [(4, 5, 4), (20, 9, 6), (24, 7, 12), (32, 16, 8), (18, 33, 10)])
def test_two_ended_helmholtz(dims, make):
    case = make(*dims)
    yp = yp_of(case)
    f = fields_of(case, yp)
    o = ol.Oracle(case.params, yp)
    g = ChannelSystem(case.params, yp)
    for s in (o, g):
        s.set_fields(f["ux"], f["uy"], f["uz"], f["p"], f["c"])
    o.step()
    g.iterate(1, raise_on_guard=False)
    fo, fg = o.get_fields(), g.get_fields()
    g.close()
    for n in ("ux", "uy", "uz", "p", "c"):
        if n in fg:
            assert rel_err(fg[n], fo[n]) <= TOL_STEP1, n
    if dims in FP32_DIMS:
        _close(_stepped(case, "fp32"), _stepped(case), FP32_VEL, FP32_PR)


# the x transforms fed by producers that march through z, against the kernels
# that read the field for themselves: rows and planes that fill no batch, every
# compiled length, and grids on both sides of the early-start and copy rules
@pytest.mark.parametrize("nx", [16, 24, 32, 48, 64, 80, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 2304, 3072])
def test_marching_divergence(nx):
    for ny, nz in ((7, 12), (10, 24)) + (((65, 48),) if nx >= 1024 else ()):
        case = _any(nx, ny, nz, xlx=0.1 * nx)
        ref = _stepped(case, schedule=2)
        _close(_stepped(case, schedule=8), ref, TOL_STEP1, TOL_STEP1)
        _close(_stepped(case, "fp32", schedule=8), ref, FP32_VEL, FP32_PR)


# both sides of each line of the default schedule (the plane kernels' shared
# memory, the z transform's plane stride, lengths without marching producers)
# against the transforms of any length
@pytest.mark.parametrize("dims", [(64, 24, 64), (96, 20, 96), (128, 24, 128), (768, 160, 128), (768, 180, 128),
                                  (256, 16, 512), (2304, 9, 12), (100, 18, 90)])
def test_default_schedule(dims):
    case = _any(*dims, xlx=0.1 * dims[0])
    src = _source(case)
    with ChannelSystem(case.params, yp_of(case)) as g:
        a = g.poisson(src)
        g.schedule = 4
        assert rel_err(a, g.poisson(src)) <= tol_poisson(dims[1])
    if dims[1] <= 24:
        ref = _stepped(case, schedule=4)
        _close(_stepped(case), ref, TOL_STEP1, TOL_STEP1)
        if dims[2] != 90:
            _close(_stepped(case, "fp32"), ref, FP32_VEL, FP32_PR)


# the line of the z transform's kind lies at a distance of the spectrum's planes
# in bytes of the storage form: 3/4 MiB in FP64, 1/2 MiB in the FP32 form
# (ny (nx / 2 + 1) values of 16 and 8 bytes)
@pytest.mark.parametrize("dims,fp64,fp32", [((768, 126, 128), 10, 10), ((768, 128, 128), 8, 10), ((768, 170, 128), 8, 10),
                                            ((768, 172, 128), 8, 8), ((768, 172, 512), 10, 10)])
def test_default_schedule_line(dims, fp64, fp32):
    case = _any(*dims)
    with ChannelSystem(case.params, yp_of(case)) as g:
        assert g.schedule == fp64
        g.precision = "fp32"
        assert g.schedule == fp32
        g.precision = "fp64"
        assert g.schedule == fp64


# state in and out of device arrays: the same bytes as through host arrays, for
# arrays at any 8-byte address, all of them and half of them read back
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("dims", [(16, 5, 8), (24, 9, 12), (64, 24, 32)])
def test_device_state(dims, prec, offset):
    import ctypes

    import torch

    case = _half(*dims)
    yp = yp_of(case)
    rng = np.random.default_rng(3)
    host = [rng.standard_normal((dims[2], dims[1], dims[0])) for _ in range(9)]
    n = host[0].size

    def dev(a=None):
        t = torch.zeros(n + offset, dtype=torch.float64, device="cuda")[offset:]
        return t if a is None else t.copy_(torch.from_numpy(a).reshape(-1))

    def ptr(t):
        return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double)) if t is not None else None

    with ChannelSystem(case.params, yp) as h, ChannelSystem(case.params, yp) as g:
        for s in (h, g):
            s.precision = prec
        h.set_fields(*host)
        d = [dev(a) for a in host]
        torch.cuda.synchronize()
        g._check(g._L.paratc_set_fields(g.handle, *[ptr(t) for t in d], 0), "set")
        fh, fg = h.get_fields(), g.get_fields()
        out = [dev() if i % 2 == 0 else None for i in range(9)]
        torch.cuda.synchronize()
        g._check(g._L.paratc_get_fields(g.handle, *[ptr(t) for t in out], 0), "get")
        for i, name in enumerate(g.FIELDS):
            assert np.array_equal(fh[name], fg[name]), name
            if out[i] is not None:
                assert np.array_equal(out[i].cpu().numpy().reshape(fh[name].shape), fh[name]), name


def _dev(a, offset=0):
    """A device copy of the array, `offset` values past an aligned address."""
    import torch

    t = torch.zeros(a.size + offset, dtype=torch.float64, device="cuda")[offset:]
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)).reshape(-1))
    torch.cuda.synchronize()
    return t


def _address(t):
    import ctypes

    if t is None:
        return None
    return ctypes.cast(t.ctypes.data if isinstance(t, np.ndarray) else t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _device_get(g):
    """All fields through device arrays."""
    n = 9 if g.params.scalar_on else 7
    names = ("ux", "uy", "uz", "p", "c", "hx", "hy", "hz", "hc") if n == 9 else ("ux", "uy", "uz", "p", None, "hx", "hy", "hz", None)
    t = [_dev(np.zeros(g.shape)) if name else None for name in names]
    g._check(g._L.paratc_get_fields(g.handle, *[_address(a) for a in t], 0), "get")
    return {name: a.cpu().numpy().reshape(g.shape) for name, a in zip(names, t) if name}


# a state field that a call leaves out keeps its values, whichever way the
# state before came and the other fields come
@pytest.mark.parametrize("missing", ["ux", "p", "c"])
@pytest.mark.parametrize("way", ["host", "device", "unaligned"])
@pytest.mark.parametrize("before", ["set", "step"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_field_left_out_is_kept(prec, before, way, missing):
    case = _half(24, 9, 12)
    yp = yp_of(case)
    f = fields_of(case, yp)
    rng = np.random.default_rng(4)
    a, b = ([rng.standard_normal((12, 9, 24)) for _ in range(5)] for _ in range(2))
    with ChannelSystem(case.params, yp) as g:
        g.set_fields(f["ux"], f["uy"], f["uz"], f["p"], f["c"])
        g.project()
        g.precision = prec
        if before == "set":
            d = [_dev(x) for x in a] + [None] * 4
            g._check(g._L.paratc_set_fields(g.handle, *[_address(t) for t in d], 0), "set")
        else:
            g.iterate(2, raise_on_guard=False)
        old = _device_get(g)
        names = ("ux", "uy", "uz", "p", "c")
        d = [None if n == missing else x if way == "host" else _dev(x, int(way == "unaligned")) for n, x in zip(names, b)]
        g._check(g._L.paratc_set_fields(g.handle, *[_address(t) for t in d + [None] * 4], 0), "set")
        new = g.get_fields()
        for n, x in zip(names, b):
            if n == missing:
                assert np.array_equal(new[n], old[n]), n
            elif n != "uy":  # (its wall row is the boundary condition's)
                assert np.array_equal(new[n], x.astype(np.float32) if prec == "fp32" and n != "p" else x), n
        for n in ("hx", "hy", "hz", "hc"):
            assert not new[n].any(), n


# a CUDA error that an earlier call left is reported by the next sync(),
# whichever way the arrays of the calls between take
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("call", ["set", "get"])
def test_pending_error_is_reported(call, offset):
    import ctypes

    case = _half(16, 5, 8)
    with ChannelSystem(case.params, yp_of(case)) as g:
        d = [_dev(np.ones(g.shape), offset) for _ in range(9)]
        host = np.zeros(8)  # no device memory: the runtime refuses a handle of it
        assert g._L.paratc_ipc_get_handle(ctypes.c_void_p(host.ctypes.data), ctypes.create_string_buffer(64))
        f = g._L.paratc_set_fields_async if call == "set" else g._L.paratc_get_fields_async
        g._check(f(g.handle, *[_address(t) for t in d], 0), call)
        with pytest.raises(ParatcError):
            g.sync()
        g.sync()  # once


# arrays of a get that overlap: the fields arrive in their order
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_overlapping_arrays_of_a_get(prec, shift):
    case = _half(32, 16, 64)
    rng = np.random.default_rng(5)
    with ChannelSystem(case.params, yp_of(case)) as g:
        g.precision = prec
        g.set_fields(*[rng.standard_normal(g.shape) for _ in range(9)])
        ref = g.get_fields()
        n = ref["ux"].size
        d = _dev(np.zeros(n + 8 * shift * n // 16))
        t = [d[i * shift * n // 16:] for i in range(9)]
        expect = np.zeros(d.numel())
        for i, name in enumerate(g.FIELDS):
            expect[i * shift * n // 16:][:n] = ref[name].reshape(-1)
        g._check(g._L.paratc_get_fields(g.handle, *[_address(a) for a in t], 0), "get")
        assert np.array_equal(d.cpu().numpy(), expect)


# 1-D spectra: one, two and more modes per thread, rows in one and two batches
@pytest.mark.parametrize("dims", [(16, 12, 128), (256, 10, 12), (384, 9, 24), (40, 11, 512), (1536, 5, 30)])
@pytest.mark.parametrize("make", [_any, _half])
def test_spectra_sizes(dims, make):
    case = make(*dims)
    yp = yp_of(case)
    f = fields_of(case, yp)
    o = ol.Oracle(case.params, yp)
    g = ChannelSystem(case.params, yp)
    for s in (o, g):
        s.set_fields(f["ux"], f["uy"], f["uz"], f["p"], f["c"])
    ref = o.spectra(2)
    g.spectra_accumulate(2)
    got = g.spectra_get()
    g.close()
    for a, b in zip(got, ref):
        for m in range(b.shape[0]):
            assert rel_err(a[m], b[m]) <= 1e-11, m
