"""The mixed method at the edges of its workspace and of its basis recursion,
held to the method's gates on the outputs that would show a mistake there: the
distributions and the fitted curves (the fitted angle comes from the grid's
Gram matrices, before the voxel's basis exists), with every regularizer's
workspace (GCV's factor region differs), both control-angle recursions and
passive sets on both sides of the factorization tile's 32 rows."""
import numpy as np
import pytest

from parity import orc_opts
from test_gpu_mixed import ALPHA_ATOL, DIST_L1_P99, MPWIN, MWF_GATE, SPWIN, errors

pytestmark = pytest.mark.gpu


# 8 echoes: the factor region is smaller than the tile; 9 x 33, 47 x 41, 24 x 63:
# odd last column of the two-curve recursion; 128 x 64: the largest
@pytest.mark.parametrize("beta", [180.0, 150.0])
@pytest.mark.parametrize("reg,rkw", [("chi2", dict(Chi2Factor=1.02)), ("gcv", {}), ("mdp", dict(NoiseLevel=60.0))])
@pytest.mark.parametrize("m,n", [(8, 31), (8, 32), (9, 33), (47, 41), (24, 63), (128, 64)])
def test_edges_within_the_gates(D, orc, ctx, m, n, reg, rkw, beta):
    X, TE = (6, 5, 3), 8e-3
    img = D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=m, TE=TE), seed=5)
    kw = dict(MatrixSize=X, nTE=m, TE=TE, nT2=n, T2Range=(10e-3, 2.0), Reg=reg, nRefAngles=8, RefConAngle=beta,
              SaveDecayCurve=True, **rkw)
    mo = D.T2mapOptions(precision="mixed", **kw)
    po = D.T2partOptions.from_t2map(mo, SPWin=SPWIN, MPWin=MPWIN)
    maps, dist, parts = D.T2mapSEcorr_T2partSEcorr(img, mo, po, ctx=ctx)
    om, od = orc.t2map(img, orc_opts(orc, D.T2mapOptions(**kw)), nthreads=8)
    op = orc.t2part(od, orc.T2partOptions(MatrixSize=X, nT2=n, T2Range=(10e-3, 2.0), SPWin=SPWIN, MPWin=MPWIN))
    for a, b in ((dist, od), (parts["sfr"], op["sfr"]), (maps["decaycurve"], om["decaycurve"])):
        np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
    e = errors(dict(n=n), maps, dist, parts, om, od, op)
    assert e["mwf_max"] <= MWF_GATE and e["l1_p99"] <= DIST_L1_P99 and e["alpha_max"] <= ALPHA_ATOL, e
    # |A dx| <= |dx|_1 for curves <= 1, and gdn = |x|_1: the gate on the
    # distributions bounds the sums and the fitted curves (relative to gdn) as well
    dg = np.abs(maps["gdn"] - om["gdn"]) / om["gdn"]
    df = np.abs(maps["decaycurve"] - om["decaycurve"]).max(-1) / om["gdn"]
    assert np.quantile(dg, 0.99) <= DIST_L1_P99 and np.quantile(df, 0.99) <= DIST_L1_P99
    if reg == "mdp":
        # a noise level above the image's: nearly every column is passive, as in the
        # oracle (the first three: all of them, 31, 32 and 33 rows of the factor)
        k, ko = (dist.reshape(-1, n) > 0).sum(1), (od.reshape(-1, n) > 0).sum(1)
        assert k.max() == ko.max() and k.max() >= {31: 31, 32: 32, 33: 33}.get(n, 33)


# The saved basis with a general control angle is the scalar FP32 recursion's,
# rounding for rounding: every product and sum rounded by itself.  (The
# coefficients may differ from numpy's by an FP64 ulp before they are rounded:
# next to a rounding boundary, not in more than 1 of 1000 values, a changed
# coefficient moves a value by at most m steps of its half ulp.)
@pytest.mark.parametrize("beta", [150.0, 99.5])
@pytest.mark.parametrize("m,n", [(4, 2), (5, 3), (32, 40), (33, 41), (64, 63)])
def test_general_angle_basis_is_the_scalar_recursion(D, ctx, m, n, beta):
    f = np.float32
    TE, T1 = 10e-3, 1.0
    angles = [150.0, 171.2, 99.0]
    X = (len(angles), 1, 1)
    img = D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=m), seed=1)
    b1 = np.asfortranarray(np.array(angles).reshape(X))
    maps, _ = D.T2mapSEcorr(img, D.T2mapOptions(MatrixSize=X, nTE=m, TE=TE, nT2=n, T2Range=(0.01, 2.0), Reg="none",
                                                RefConAngle=beta, SaveNNLSBasis=True, precision="mixed"), b1map=b1, ctx=ctx)
    t2 = np.exp(np.linspace(np.log(0.01), np.log(2.0), n))
    dot = lambda a, v: (a[0] * v[0] + a[1] * v[1]) + a[2] * v[2]  # noqa: E731  (float32 throughout)
    for v, al in enumerate(angles):
        A, r = al / 180, np.pi / 180
        a1, ai = A * 180 * r, A * beta * r
        E1, E2 = np.exp(-(TE / 2) / T1), np.exp(-(TE / 2) / t2)
        sh, ch = np.sin(a1 / 2), np.cos(a1 / 2)
        c2, s2 = (1 + np.cos(ai)) / 2, 1 - (1 + np.cos(ai)) / 2
        pa, pb, pc, pd = E2 * E2 * c2, E2 * E2 * s2, E1 * E2 * np.sin(ai), np.full(n, E1 * E1 * np.cos(ai))
        F, Fb, Z = ([x.astype(f) for x in q] for q in ((pa, pb, pc), (pb, pa, -pc), (-pc / 2, pc / 2, pd)))
        a1c, b1c, c1c = ((E2 * E2 * ch * ch).astype(f), (E2 * E2 * sh * sh).astype(f), (E1 * E2 * 2 * sh * ch).astype(f))
        m0 = np.full(n, sh).astype(f)
        S = np.zeros((m + 4, 3, n), f)  # state j at S[j]; those not reached yet are zero
        S[1, 0], S[1, 2], S[2, 0] = b1c * m0, ((-c1c) * m0) / f(2), a1c * m0
        out = np.zeros((m, n), f)
        out[0] = np.abs(S[1, 0])
        for i in range(2, m):
            T = np.zeros_like(S)
            for j in range(1, m + 2):
                T[j, 0] = dot(Fb, S[1]) if j == 1 else dot(F, S[j - 1])
                T[j, 1], T[j, 2] = dot(Fb, S[j + 1]), dot(Z, S[j])
            S = T
            out[i - 1] = np.abs(S[1, 0])
        out[m - 1] = np.abs(dot(Fb, S[1]))
        want, got = out.astype(np.float64), maps["decaybasis"][v, 0, 0]
        assert (want != got).mean() <= 1e-3
        np.testing.assert_allclose(got, want, rtol=0, atol=4e-6)
