"""The kernels' workspace rules at the sizes where they can go wrong, on the
GPU against the oracle: plain-method shapes whose last padding rows leave shared
memory (one more warp per SM), and mixed-method shapes around the factorization
tile's limits, the two-curve basis recursion's odd column and the staged basis's
overlap with the Gram matrix."""
import numpy as np
import pytest

from parity import DIST_RTOL, dist_rel_err

pytestmark = pytest.mark.gpu


def _image(D, X, m, seed):
    return D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=m, TE=8e-3), seed=seed)


# (nTE, nT2): one more warp by spilled rows at every shape but the last (which
# already holds eight); L-curve solves at large mu reach every padding row
@pytest.mark.parametrize("m,n", [(48, 40), (56, 60), (64, 60), (48, 48), (64, 40), (32, 40)])
def test_plain_spilled_rows(D, orc, ctx, m, n):
    X = (5, 3, 1)
    img = _image(D, X, m, 3)
    kw = dict(MatrixSize=X, nTE=m, TE=8e-3, nT2=n, T2Range=(10e-3, 2.0), Reg="lcurve", nRefAngles=8)
    maps, dist = D.T2mapSEcorr(img, D.T2mapOptions(**kw), ctx=ctx)
    om, od = orc.t2map(img, orc.T2mapOptions(**kw))
    err, ok = dist_rel_err(dist, od)
    assert ok.all() and err.max() <= DIST_RTOL
    np.testing.assert_allclose(maps["alpha"], om["alpha"], rtol=1e-12)


# nT2 around the 31-32 row limits of the tile and the substitutions, odd and
# even; few echoes (factor region smaller than the tile) and many
# (the discrepancy principle at a noise level above the image's reaches large mu,
# where nearly every column is passive)
@pytest.mark.parametrize("reg,rkw", [("chi2", dict(Chi2Factor=1.02)), ("mdp", dict(NoiseLevel=60.0))])
@pytest.mark.parametrize("m,n", [(8, 31), (8, 32), (9, 33), (128, 33), (47, 41), (24, 63), (128, 64)])
def test_mixed_workspace_edges(D, orc, ctx, m, n, reg, rkw):
    X = (4, 3, 1)
    img = _image(D, X, m, 5)
    kw = dict(MatrixSize=X, nTE=m, TE=8e-3, nT2=n, T2Range=(10e-3, 2.0), Reg=reg, nRefAngles=8, **rkw)
    mo = D.T2mapOptions(precision="mixed", **kw)
    po = D.T2partOptions.from_t2map(mo, SPWin=(10e-3, 40e-3), MPWin=(40e-3, 200e-3))
    maps, dist, parts = D.T2mapSEcorr_T2partSEcorr(img, mo, po, ctx=ctx)
    om, od = orc.t2map(img, orc.T2mapOptions(**kw))
    op = orc.t2part(od, orc.T2partOptions(MatrixSize=X, nT2=n, T2Range=(10e-3, 2.0), SPWin=(10e-3, 40e-3), MPWin=(40e-3, 200e-3)))
    assert np.isfinite(dist).all()
    assert np.abs(maps["alpha"] - om["alpha"]).max() <= 0.01      # the mixed method's stated gates
    assert np.abs(parts["sfr"] - op["sfr"]).max() <= 1e-3


# the mixed method's saved basis is the scalar FP32 recursion's, rounding for
# rounding (the coefficients may differ from numpy's by an FP64 ulp before they
# are rounded, so a coefficient next to a rounding boundary may differ: none do
# at these angles in more than 1 of 1000 curves' values)
@pytest.mark.parametrize("m,n", [(4, 2), (5, 3), (32, 40), (33, 41), (64, 60)])
def test_mixed_basis_is_the_scalar_recursion(D, ctx, m, n):
    f = np.float32
    TE, T1 = 10e-3, 1.0
    angles = [150.0, 171.2, 99.0]
    X = (len(angles), 1, 1)
    img = D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=m), seed=1)
    b1 = np.asfortranarray(np.array(angles).reshape(X))
    maps, _ = D.T2mapSEcorr(img, D.T2mapOptions(MatrixSize=X, nTE=m, TE=TE, nT2=n, T2Range=(0.01, 2.0), Reg="none",
                                                SaveNNLSBasis=True, precision="mixed"), b1map=b1, ctx=ctx)
    t2 = np.exp(np.linspace(np.log(0.01), np.log(2.0), n))
    fma = lambda a, b, c: (a.astype(np.float64) * b + c).astype(f)  # noqa: E731  (exact product, one rounding)
    for v, al in enumerate(angles):
        r = np.pi / 180
        E1, E2 = np.exp(-(TE / 2) / T1), np.exp(-(TE / 2) / t2)
        a = E2 * E2 / 2
        c = E1 * E2 * np.sin(al * r)
        q = [x.astype(f) for x in (a, a * np.cos(al * r), c, np.full(n, E1 * E1 * np.cos(al * r)), -c / 2,
                                   np.full(n, np.sin(al / 2 * r)))]
        A, B, Cc, Dd, Cp, m0 = q
        F, Fb, Z = (np.zeros((m + 3, n), f) for _ in range(3))
        out = np.zeros((m, n), f)
        out[0] = A - B
        F[1], Z[1], F[2] = A - B, Cp, A + B
        for i in range(2, m):
            kend = i if i <= m // 2 else m - i + 1
            nF, nFb, nZ = F.copy(), Fb.copy(), Z.copy()
            for k in range(1, kend + 1):
                s, d = A * (F[k] + Fb[k]), B * (F[k] - Fb[k])
                oF, oFb = fma(Cc, Z[k], s + d), fma(-Cc, Z[k], s - d)
                nF[k + 1], nZ[k] = oF, fma(Cp, F[k] - Fb[k], Dd * Z[k])
                if k == 1:
                    nF[1] = out[i - 1] = oFb
                else:
                    nFb[k - 1] = oFb
            F, Fb, Z = nF, nFb, nZ
            if i <= m // 2:
                Fb[i] = Fb[i + 1] = Z[i + 1] = 0
        out[m - 1] = fma(-Cc, Z[1], fma(A, F[1] + Fb[1], (-B) * (F[1] - Fb[1])))
        want, got = np.abs(m0 * out).astype(np.float64), maps["decaybasis"][v, 0, 0]
        assert (want != got).mean() <= 1e-3
        np.testing.assert_allclose(got, want, rtol=0, atol=4e-6)  # a changed coefficient: m steps of its half ulp


# T2part of float values that the integer widening does not cover, next to ones
# that it does
def test_t2part_float_special_values(D, orc, ctx):
    n = 12
    rng = np.random.default_rng(0)
    d = np.asfortranarray(rng.uniform(0, 100, (7, 3, 2, n)).astype(np.float32))
    d[0, 0, 0, 3] = np.float32(1e-42)      # subnormal
    d[1, 0, 0, 2] = np.inf
    d[2, 0, 0, 5] = np.nan
    d[3, 0, 0, :] = 0
    d[4, 0, 0, 1] = -0.0
    d[5, 0, 0, 4] = np.finfo(np.float32).max
    kw = dict(MatrixSize=d.shape[:3], nT2=n, T2Range=(10e-3, 2.0), SPWin=(10e-3, 40e-3), MPWin=(40e-3, 200e-3))
    for sig in (None, 20e-3):
        got = D.T2partSEcorr(d, D.T2partOptions(Sigmoid=sig, **kw), ctx=ctx)
        want = orc.t2part(d.astype(np.float64), orc.T2partOptions(Sigmoid=sig, **kw))
        for k in ("sfr", "sgm", "mfr", "mgm"):
            with np.errstate(over="ignore"):
                np.testing.assert_array_equal(got[k], want[k].astype(np.float32), err_msg=k)
