"""Device memory under a budget, or on a device that refuses: what the
narrowing buffer of host float calls holds is given up before anything is
refused for lack of it."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

POOL = r"""
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
