"""Device memory under a budget, or on a device that refuses: what the
narrowing buffer of host float calls and the warps' scratch hold is given up
before anything is refused for lack of it, and a launch whose scratch does not
fit runs with fewer warps, to the same outputs."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

POOL = r"""
#include <algorithm>
#include <cassert>
#include <cstdlib>
#include "devpool.h"
struct Ctx { size_t budget, used = 0; std::map<std::string, dh::DevBuf> bufs; };
int main() {
    size_t held = 0, room = 0;                      // a device of `room` bytes
    std::map<void *, size_t> sizes;
    auto alloc = [&](void **p, size_t n) {
        if (held + n > room) { *p = nullptr; return false; }
        *p = std::malloc(1); sizes[*p] = n; held += n;
        return true;
    };
    auto free_ = [&](void *p) { held -= sizes.at(p); sizes.erase(p); std::free(p); };
    void *p = nullptr;
    {   // the device refuses below the budget: the large request fails, a smaller one and the accounts do not
        room = 100; held = 0;
        Ctx c{1000};
        assert(dh::pool_get(c, "outputs", 60, alloc, free_, &p) == dh::kPoolOk);
        assert(dh::pool_get(c, dh::kNarrowBuf, 50, alloc, free_, &p) == dh::kPoolRefused);
        assert(c.used == 60 && c.bufs[dh::kNarrowBuf].p == nullptr);
        assert(dh::pool_get(c, dh::kNarrowBuf, 40, alloc, free_, &p) == dh::kPoolOk && c.used == 100);
        // ... and gives way to another buffer
        assert(dh::pool_get(c, "image", 30, alloc, free_, &p) == dh::kPoolOk);
        assert(c.used == 90 && held == 90 && c.bufs[dh::kNarrowBuf].p == nullptr);
        assert(dh::pool_get(c, "image", 30, alloc, free_, &p) == dh::kPoolOk && c.used == 90);
        assert(!dh::pool_alloc(c, &p, 11, alloc, free_) && dh::pool_alloc(c, &p, 10, alloc, free_));
    }
    {   // the budget refuses
        room = 1000; held = 0;
        Ctx c{100};
        assert(dh::pool_get(c, dh::kNarrowBuf, 40, alloc, free_, &p) == dh::kPoolOk);
        assert(dh::pool_fits(c, 60, free_) && c.used == 40);
        assert(dh::pool_get(c, "image", 70, alloc, free_, &p) == dh::kPoolOk);
        assert(c.used == 70 && c.bufs[dh::kNarrowBuf].p == nullptr);
        assert(dh::pool_get(c, dh::kNarrowBuf, 31, alloc, free_, &p) == dh::kPoolOverBudget && c.used == 70);
        assert(dh::pool_get(c, "image", 101, alloc, free_, &p) == dh::kPoolOverBudget && c.used == 0 && held == 0);
    }
    {   // the scratch: room for it beside a reserve, dropped for other buffers, never for the narrowing one
        room = 1000; held = 0;
        Ctx c{100};
        assert(dh::pool_get(c, "outputs", 30, alloc, free_, &p) == dh::kPoolOk);
        assert(dh::pool_scratch_room(c, 60, 10, free_) == 60);
        assert(dh::pool_get(c, dh::kScratchBuf, 60, alloc, free_, &p) == dh::kPoolOk);
        assert(dh::pool_get(c, dh::kNarrowBuf, 10, alloc, free_, &p) == dh::kPoolOk && c.used == 100);
        assert(dh::pool_scratch_room(c, 60, 10, free_) == 60 && c.used == 100);      // fits: nothing freed
        assert(dh::pool_scratch_room(c, 61, 10, free_) == 60 && c.used == 90);       // without the narrowing buffer
        assert(dh::pool_scratch_room(c, 61, 20, free_) == 50 && c.used == 30);       // and the scratch is too large
        assert(dh::pool_get(c, dh::kScratchBuf, 50, alloc, free_, &p) == dh::kPoolOk);
        assert(dh::pool_get(c, dh::kNarrowBuf, 21, alloc, free_, &p) == dh::kPoolOverBudget && c.used == 80);
        assert(dh::pool_get(c, "image", 21, alloc, free_, &p) == dh::kPoolOk && c.used == 51);
        assert(dh::pool_scratch_room(c, 60, 200, free_) == 0);
    }
    for (int g0 = 1; g0 < 40; ++g0)                  // a cut launch fits, keeps half of the warps, or is refused
        for (int w0 = 1; w0 <= 16; ++w0)
            for (long fit = 0; fit <= 2L * g0 * w0; ++fit) {
                int g = g0, w = w0;
                const bool ok = dh::shrink_launch(fit, &g, &w);
                assert(ok == (2 * fit >= (long)g0 * w0));
                if (!ok) { assert(g == g0 && w == w0); continue; }
                assert(g >= 1 && w >= 1 && g <= g0 && w <= w0 && ((long)g * w <= fit || fit >= (long)g0 * w0));
                assert(fit < (long)g0 * w0 || (g == g0 && w == w0));
                assert(3L * g * w >= std::min(fit, (long)g0 * w0));
            }
    return 0;
}
"""


def test_pool_rules(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "pool.cpp").write_text(POOL)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-UNDEBUG", "-I", os.path.join(ROOT, "decaes.jl_gb300", "csrc"),
                    str(tmp_path / "pool.cpp"), "-o", str(tmp_path / "pool")], check=True, timeout=120)
    subprocess.run([str(tmp_path / "pool")], check=True, timeout=60)


def _call(D, ctx, img, X, m, n, **kw):
    mo = D.T2mapOptions(MatrixSize=X, nTE=m, TE=10e-3, nT2=n, T2Range=(10e-3, 2.0), Reg="none", nRefAngles=8, **kw)
    po = D.T2partOptions.from_t2map(mo, SPWin=(10e-3, 25e-3), MPWin=(25e-3, 200e-3))
    maps, dist, parts = D.T2mapSEcorr_T2partSEcorr(img, mo, po, ctx=ctx)
    return dict(maps, dist=dist, **parts)


def _accepts(D, budget, f):
    c = D.Context(0, hbm_budget_bytes=budget)
    try:
        f(c)
        return True
    except RuntimeError as e:
        assert "ENOMEM" in str(e)
        return False
    finally:
        c.close()


def _least_budget(D, f, lo=1 << 20, hi=1 << 30):
    """The smallest budget (to 16 KB) of a new context that f's calls fit in."""
    assert _accepts(D, hi, f) and not _accepts(D, lo, f)
    while hi - lo > 1 << 14:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if _accepts(D, mid, f) else (mid, hi)
    return hi


def _same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


# A float call on a volume, then the same volume in double, in a context that
# holds the double call and the largest float output besides: the float call
# narrows its outputs together or one by one, as they fit, and leaves nothing
# behind that the double call is refused for.
@pytest.mark.gpu
def test_double_call_after_float_call_within_the_budget(D, ctx):
    X, m, n = (64, 64, 8), 32, 40
    img = D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=m), seed=2)
    f32 = np.asfortranarray(img, dtype=np.float32)
    want32, want64 = _call(D, ctx, f32, X, m, n), _call(D, ctx, img, X, m, n)
    least = _least_budget(D, lambda c: _call(D, c, img, X, m, n))
    tight = D.Context(0, hbm_budget_bytes=least + 4 * n * int(np.prod(X)) + (1 << 18))
    _same(_call(D, tight, f32, X, m, n), want32)
    _same(_call(D, tight, img, X, m, n), want64)
    _same(_call(D, tight, f32, X, m, n), want32)  # now without room for all of them together
    tight.close()


def _scratch_bytes(m, n, K):
    """Global scratch of one warp: basis, surrogate samples, caches, singular values, stored solutions, FP32 basis."""
    return 8 * (m * n + 3 * K + 19 * 128 + min(m, n) + 16 + 64 * (n + 1) + (m * n + 1) // 2)


# Budgets for the scratch of as many warps per SM as single-warp blocks with the
# whole workspace in shared memory hold (12 mixed, 3 plain), and 8 MB for
# the rest: fewer than the launches' own shapes (15, 4) take.
@pytest.mark.gpu
@pytest.mark.parametrize("m,n,precision,warps", [(48, 40, "mixed", 12), (56, 60, "fp64", 3)])
def test_fewer_warps_where_the_scratch_does_not_fit(D, ctx, m, n, precision, warps):
    import torch
    X, K = (5, 4, 3), 8
    img = D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=m), seed=4)
    mo = D.T2mapOptions(MatrixSize=X, nTE=m, TE=10e-3, nT2=n, T2Range=(10e-3, 2.0), Reg="lcurve", nRefAngles=K,
                        precision=precision)
    po = D.T2partOptions.from_t2map(mo, SPWin=(10e-3, 25e-3), MPWin=(25e-3, 200e-3))

    def host(c, dt):
        maps, dist, parts = D.T2mapSEcorr_T2partSEcorr(np.asfortranarray(img, dtype=dt), mo, po, ctx=c)
        return dict(maps, dist=dist, **parts)

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tight = D.Context(0, hbm_budget_bytes=warps * sms * _scratch_bytes(m, n, K) + (8 << 20))
    for dt in (np.float32, np.float64):
        _same(host(tight, dt), host(ctx, dt))
    tight.close()
    with pytest.raises(RuntimeError, match="ENOMEM"):  # a quarter of the warps is still refused
        host(D.Context(0, hbm_budget_bytes=warps * sms * _scratch_bytes(m, n, K) // 4), np.float64)


# the same for batches (one-shot, prepared), two classes
@pytest.mark.gpu
def test_batches_with_fewer_warps_where_the_scratch_does_not_fit(D, ctx):
    import torch
    from decaes_gb300 import _lib
    L = D.load()
    X, K, V = (4, 3, 2), 8, 24
    vols, outs = [], []
    for i, (m, n) in enumerate([(48, 40), (64, 60)]):
        img = D.mock_image(D.MockImageOptions(MatrixSize=X, nTE=m), seed=6 + i)
        mo = D.T2mapOptions(MatrixSize=X, nTE=m, TE=10e-3, nT2=n, T2Range=(10e-3, 2.0), Reg="chi2", Chi2Factor=1.02,
                            nRefAngles=K, precision="mixed")
        _, dist = D.T2mapSEcorr(img, mo, ctx=ctx)
        d_img = torch.from_numpy(img.reshape(-1, order="F").copy()).cuda()
        out = {k: torch.full((V * (n if k == "dist" else 1),), 7.0, dtype=torch.float64, device="cuda")
               for k in ("dist", "gdn", "ggm", "gva", "fnr", "snr", "alpha")}
        vols.append(_lib.VolumeC(mopts=mo.to_c(), has_t2part=0, dtype=_lib.F64, d_image=d_img.data_ptr(), d_b1map=None,
                                 d_mout=_lib.T2mapOutC(**{k: t.data_ptr() for k, t in out.items()})))
        outs.append((d_img, out, dist.reshape(-1, order="F")))
    arr = (_lib.VolumeC * len(vols))(*vols)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # 12 warps per SM of the smaller volume, 5 of the larger; 15 and 7 are launched
    need = sms * max(12 * _scratch_bytes(48, 40, K), 5 * _scratch_bytes(64, 60, K))
    tight = D.Context(0, hbm_budget_bytes=need + (16 << 20))

    def check():
        torch.cuda.synchronize()
        for _, out, want in outs:
            np.testing.assert_array_equal(out["dist"].cpu().numpy(), want)
            out["dist"].fill_(7.0)

    torch.cuda.synchronize()
    tight.check(L.decaes_t2map_t2part_batch(tight.h, arr, len(vols), None))
    check()
    b = L.decaes_batch_create(tight.h, arr, len(vols))
    assert b, L.decaes_last_error(tight.h).decode()
    assert L.decaes_batch_run(b, None) == 0
    check()
    L.decaes_batch_destroy(b)
    tight.close()
