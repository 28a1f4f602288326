"""A context that runs batches only: completing a batch's statistics leaves no
error behind for the next call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_sync_stats_without_a_single_volume_call(D, ctx):
    import torch
    from decaes_gb300 import _lib
    L = D.load()
    X, V, m, n = (3, 2, 2), 12, 32, 40
    img = D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=m), seed=8)
    mo = D.T2mapOptions(MatrixSize=X, nTE=m, TE=10e-3, nT2=n, T2Range=(10e-3, 2.0), Reg="none", nRefAngles=8)
    _, want = D.T2mapSEcorr(img, mo, ctx=ctx)
    d_img = torch.from_numpy(img.reshape(-1, order="F").copy()).cuda()
    out = {k: torch.full((V * (n if k == "dist" else 1),), 7.0, dtype=torch.float64, device="cuda")
           for k in ("dist", "gdn", "ggm", "gva", "fnr", "snr", "alpha")}
    arr = (_lib.VolumeC * 1)(_lib.VolumeC(mopts=mo.to_c(), has_t2part=0, dtype=_lib.F64, d_image=d_img.data_ptr(),
                                          d_mout=_lib.T2mapOutC(**{k: t.data_ptr() for k, t in out.items()})))
    torch.cuda.synchronize()
    fresh = D.Context(0)
    fresh.check(L.decaes_t2map_t2part_batch(fresh.h, arr, 1, None))
    fresh.check(L.decaes_sync_stats(fresh.h, None))
    s = fresh.stats()
    assert s["voxels"] == V and s["ms_total"] == 0 and s["ms_solve"] == 0
    out["dist"].fill_(7.0)
    torch.cuda.synchronize()
    b = L.decaes_batch_create(fresh.h, arr, 1)
    assert b, L.decaes_last_error(fresh.h).decode()
    fresh.check(L.decaes_batch_run(b, None))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out["dist"].cpu().numpy(), want.reshape(-1, order="F"))
    L.decaes_batch_destroy(b)
    fresh.close()
