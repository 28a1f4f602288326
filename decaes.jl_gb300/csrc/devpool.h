// devpool.h -- a context's named device buffers and their byte budget.  The
// allocator is passed in, so the rules can be exercised without a GPU.
#pragma once
#include <cstddef>
#include <map>
#include <string>

namespace dh {

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
};

enum PoolResult { kPoolOk, kPoolOverBudget, kPoolRefused };

// Buffers whose contents no call needs once it has returned: a host float call's
// narrowed outputs, and the warps' scratch, which a call asks for last but for
// the former (and can be made smaller).
constexpr const char *kNarrowBuf = "narrow", *kScratchBuf = "scratch";

// Frees a named buffer; false when it is empty.
template <class Pool, class Free>
bool pool_drop(Pool &c, const char *name, Free free_) {
    DevBuf &b = c.bufs[name];
    if (!b.p) return false;
    free_(b.p);
    c.used -= b.bytes;
    b = DevBuf{};
    return true;
}

// Whether `bytes` more fit the budget, with the narrowing buffer, then (if
// scratch) the scratch, freed for them if need be.
template <class Pool, class Free>
bool pool_fits(Pool &c, size_t bytes, Free free_, bool scratch = true) {
    const auto fit = [&] { return c.used + bytes <= c.budget; };
    return fit() || (pool_drop(c, kNarrowBuf, free_) && fit()) || (scratch && pool_drop(c, kScratchBuf, free_) && fit());
}

// alloc(&p, bytes), again without those buffers when the device refuses.
template <class Pool, class Alloc, class Free>
bool pool_alloc(Pool &c, void **p, size_t bytes, Alloc alloc, Free free_, bool scratch = true) {
    return alloc(p, bytes) || (pool_drop(c, kNarrowBuf, free_) && alloc(p, bytes)) ||
           (scratch && pool_drop(c, kScratchBuf, free_) && alloc(p, bytes));
}

// The named buffer grown to at least `bytes`.  When that fails it is left empty.
template <class Pool, class Alloc, class Free>
PoolResult pool_get(Pool &c, const std::string &name, size_t bytes, Alloc alloc, Free free_, void **out) {
    DevBuf &b = c.bufs[name];
    if (b.bytes < bytes) {
        const bool scratch = name != kNarrowBuf;
        pool_drop(c, name.c_str(), free_);
        if (!pool_fits(c, bytes, free_, scratch)) return kPoolOverBudget;
        void *p = nullptr;
        if (!pool_alloc(c, &p, bytes, alloc, free_, scratch)) return kPoolRefused;
        b = DevBuf{p, bytes};
        c.used += bytes;
    }
    *out = b.p;
    return kPoolOk;
}

// Bytes the scratch may take with `reserve` bytes left for the narrowing buffer;
// what the two hold above that is freed when `want` does not fit.
template <class Pool, class Free>
size_t pool_scratch_room(Pool &c, size_t want, size_t reserve, Free free_) {
    DevBuf &s = c.bufs[kScratchBuf], &nb = c.bufs[kNarrowBuf];
    const auto room = [&] {
        const size_t others = c.used - s.bytes + (reserve > nb.bytes ? reserve - nb.bytes : 0);
        return c.budget > others ? c.budget - others : 0;
    };
    if (room() < want) pool_drop(c, kNarrowBuf, free_);
    if (room() < s.bytes) pool_drop(c, kScratchBuf, free_);
    return room();
}

// A launch of *grid blocks of *wpb warps cut to `fit` warps, by smaller blocks
// first (every SM keeps one); false when that is less than half of them.
inline bool shrink_launch(long fit, int *grid, int *wpb) {
    const long all = (long)*grid * *wpb;
    if (fit >= all) return true;
    if (2 * fit < all) return false;
    const long least = (*wpb + 1) / 2, w = fit / *grid;
    *wpb = (int)(w > least ? w : least);
    if (fit / *wpb < *grid) *grid = (int)(fit / *wpb);
    return true;
}

}  // namespace dh
