"""What decaes_autotune reports: the fastest of its own block sizes, and the
shape that later calls take, which may be the untuned one."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Tuning(C.Structure):  # the report at its offsets
    _fields_ = [("warps_per_block", C.c_int32), ("kept_warps_per_block", C.c_int32), ("us_per_voxel", C.c_double),
                ("blocks_per_sm", C.c_int32), ("kept_blocks_per_sm", C.c_int32)]


def _lib():
    from decaes_gb300 import _lib
    return _lib


# the mixed method's untuned shape is one block of up to 16 warps, which none of
# the tuned block sizes reaches; legacy calls' is one of them (a warp per block)
@pytest.mark.parametrize("kw", [dict(Reg="chi2", Chi2Factor=1.02, precision="mixed"), dict(Reg="none", precision="fp64"),
                                dict(Reg="chi2", Chi2Factor=1.02, legacy=True)])
def test_report_names_the_kept_shape(D, kw):
    L, fresh = D.load(), D.Context(0)
    X = (5, 4, 3)
    mo = D.T2mapOptions(MatrixSize=X, nTE=32, TE=10e-3, nT2=40, T2Range=(10e-3, 2.0), nRefAngles=8, **kw)
    img = D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=32), seed=9)
    _, before = D.T2mapSEcorr(img, mo, ctx=fresh)
    assert C.sizeof(Tuning) == C.sizeof(_lib().TuningC) == 24
    for _ in range(2):  # a second tuning starts from the first one's
        t = Tuning(-1, -1, -1.0, -1, -1)
        fresh.check(L.decaes_autotune(fresh.h, C.byref(mo.to_c()), C.cast(C.byref(t), C.POINTER(_lib().TuningC))))
        assert t.warps_per_block in (1, 2, 4) and t.blocks_per_sm >= 0 and t.us_per_voxel > 0
        assert 1 <= t.kept_warps_per_block <= 16 and t.kept_blocks_per_sm >= 1
        if t.kept_warps_per_block in (1, 2, 4):
            # one of the tuned sizes, or an untuned launch of the same size
            assert t.kept_blocks_per_sm * t.kept_warps_per_block <= 32
        else:  # the untuned shape: more warps than any block size of 1, 2 or 4 leaves resident
            assert t.kept_warps_per_block * t.kept_blocks_per_sm >= t.warps_per_block * max(t.blocks_per_sm, 1)
        if kw.get("legacy"):
            assert t.kept_warps_per_block in (1, 2, 4)
        _, dist = D.T2mapSEcorr(img, mo, ctx=fresh)
        np.testing.assert_array_equal(dist, before)
    print(kw, "fastest tuned", t.warps_per_block, "x", t.blocks_per_sm, "kept", t.kept_warps_per_block, "x", t.kept_blocks_per_sm)
    fresh.close()
