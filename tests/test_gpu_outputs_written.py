"""A successful call writes every entry of every output that it was given: the
outputs start as a marker that no output takes (all are NaN or >= 0), and none
is left.  Host calls (both types, narrowed together), single outputs, T2part
alone, device pointers and served requests."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MARK = -7.0
PARTS = ("sfr", "sgm", "mfr", "mgm")
SAVE = dict(SaveResidualNorm=True, SaveDecayCurve=True, SaveRegParam=True, SaveNNLSBasis=True)
# masked voxels (a share of the image below the threshold, or all of it) with every optional output
CASES = {
    "mixed_lcurve_masked": dict(Reg="lcurve", precision="mixed", Threshold=200.0, **SAVE),
    "mixed_tc": dict(Reg="chi2", Chi2Factor=1.02, precision="mixed_tc", Threshold=200.0, **SAVE),
    "none": dict(Reg="none", **SAVE),
    "fixed_angle": dict(Reg="chi2", Chi2Factor=1.02, SetFlipAngle=165.0, Threshold=200.0, **SAVE),
    "legacy": dict(Reg="chi2", Chi2Factor=1.02, legacy=True, Threshold=200.0, **SAVE),
    "nothing_above": dict(Reg="gcv", Threshold=1e9, **SAVE),
    "plain_defaults": dict(Reg="lcurve", Threshold=200.0),
}
X, M, N, K = (7, 5, 3), 32, 40, 8


def _case(D, kw, dt):
    img = D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=M, BackgroundFraction=0.4), seed=11, dtype=dt)
    mo = D.T2mapOptions(MatrixSize=X, nTE=M, TE=10e-3, nT2=N, T2Range=(10e-3, 2.0), nRefAngles=K, **kw)
    po = D.T2partOptions.from_t2map(mo, SPWin=(10e-3, 25e-3), MPWin=(25e-3, 200e-3))
    return np.asfortranarray(img), mo, po


def _marked(mo, dt):
    from decaes_gb300 import _lib, api
    maps, dist, out = api._t2map_buffers(mo, dt)
    parts = {k: np.empty(X, dt, order="F") for k in PARTS}
    pout = _lib.T2partOutC(*[parts[k].ctypes.data_as(C.c_void_p) for k in PARTS])
    arrays = dict(maps, dist=dist, **parts)
    for a in arrays.values():
        a.fill(MARK)
    return arrays, out, pout


def _none_left(arrays):
    for k, a in arrays.items():
        assert not (np.asarray(a) == MARK).any(), k


def _vp(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("name", list(CASES))
def test_host_calls(D, ctx, name, dt):
    from decaes_gb300 import _lib
    img, mo, po = _case(D, CASES[name], dt)
    code = _lib.F32 if dt == np.float32 else _lib.F64
    arrays, out, pout = _marked(mo, dt)
    ctx.check(ctx.L.decaes_t2map_t2part(ctx.h, C.byref(mo.to_c()), C.byref(po.to_c()), _vp(img), code, None, C.byref(out),
                                        C.byref(pout)))
    _none_left(arrays)
    # each output requested alone: it is what it is among the others, and nothing else is touched
    for k in ("dist", "alpha") + (("decaycurve",) if mo.SaveDecayCurve else ()):
        alone, _, _ = _marked(mo, dt)
        ctx.check(ctx.L.decaes_t2map(ctx.h, C.byref(mo.to_c()), _vp(img), code, None, C.byref(_lib.T2mapOutC(**{k: _vp(alone[k])}))))
        np.testing.assert_array_equal(alone[k], arrays[k])
        assert all((a == MARK).all() for j, a in alone.items() if j != k)
    # T2part alone on the saved distribution
    parts = {k: np.full(X, MARK, dt, order="F") for k in PARTS}
    ctx.check(ctx.L.decaes_t2part(ctx.h, C.byref(po.to_c()), _vp(arrays["dist"]), code,
                                  C.byref(_lib.T2partOutC(**{k: _vp(a) for k, a in parts.items()}))))
    _none_left(parts)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("name", ["mixed_lcurve_masked", "none", "fixed_angle", "nothing_above"])
def test_device_calls(D, ctx, name, dt):
    import torch
    from decaes_gb300 import _lib
    img, mo, po = _case(D, CASES[name], dt)
    arrays, _, _ = _marked(mo, dt)
    names = [k for k in arrays if k not in ("echotimes", "t2times", "refangleset", "decaybasisset")]
    dev = {k: torch.from_numpy(arrays[k].reshape(-1, order="F").copy()).cuda() for k in names}
    d_img = torch.from_numpy(img.reshape(-1, order="F").copy()).cuda()
    mout = _lib.T2mapOutC(**{k: t.data_ptr() for k, t in dev.items() if k not in PARTS})
    pout = _lib.T2partOutC(**{k: dev[k].data_ptr() for k in PARTS})
    torch.cuda.synchronize()
    ctx.check(ctx.L.decaes_t2map_t2part_device(ctx.h, C.byref(mo.to_c()), C.byref(po.to_c()), C.c_void_p(d_img.data_ptr()),
                                               _lib.F32 if dt == np.float32 else _lib.F64, None, C.byref(mout),
                                               C.byref(pout), None))
    ctx.check(ctx.L.decaes_sync_stats(ctx.h, None))
    _none_left({k: t.cpu().numpy() for k, t in dev.items()})


def test_served_requests(D, ctx):
    from decaes_gb300 import _lib
    L = ctx.L
    srv = L.decaes_server_create(ctx.h, C.byref(_lib.ServerOptsC(64, 0)))  # several ticks a request
    assert srv
    try:
        reqs = []
        for name in ("mixed_lcurve_masked", "none", "fixed_angle", "nothing_above"):
            for dt in (np.float32, np.float64):
                img, mo, po = _case(D, CASES[name], dt)
                arrays, out, pout = _marked(mo, dt)
                rid = L.decaes_server_submit(srv, C.byref(mo.to_c()), C.byref(po.to_c()), _vp(img),
                                             _lib.F32 if dt == np.float32 else _lib.F64, C.byref(out), C.byref(pout))
                assert rid > 0
                reqs.append((rid, img, arrays, out, pout))
        for rid, _, arrays, _, _ in reqs:
            assert L.decaes_server_wait(srv, rid) == 0
            _none_left(arrays)
    finally:
        L.decaes_server_destroy(srv)
