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

// Host float calls narrow all their outputs into this buffer; no call needs its
// contents once it has returned.
constexpr const char *kNarrowBuf = "narrow";

// Frees the narrowing buffer; false when there is none.
template <class Pool, class Free>
bool pool_give_back(Pool &c, Free free_) {
    DevBuf &b = c.bufs[kNarrowBuf];
    if (!b.p) return false;
    free_(b.p);
    c.used -= b.bytes;
    b = DevBuf{};
    return true;
}

// Whether `bytes` more fit the budget, the narrowing buffer freed for them if need be.
template <class Pool, class Free>
bool pool_fits(Pool &c, size_t bytes, Free free_) {
    return c.used + bytes <= c.budget || (pool_give_back(c, free_) && c.used + bytes <= c.budget);
}

// alloc(&p, bytes), once more without the narrowing buffer when the device refuses.
template <class Pool, class Alloc, class Free>
bool pool_alloc(Pool &c, void **p, size_t bytes, Alloc alloc, Free free_) {
    return alloc(p, bytes) || (pool_give_back(c, free_) && alloc(p, bytes));
}

// The named buffer grown to at least `bytes`.  When that fails it is left empty.
template <class Pool, class Alloc, class Free>
PoolResult pool_get(Pool &c, const std::string &name, size_t bytes, Alloc alloc, Free free_, void **out) {
    DevBuf &b = c.bufs[name];
    if (b.bytes < bytes) {
        if (b.p) free_(b.p);
        c.used -= b.bytes;
        b = DevBuf{};
        if (!pool_fits(c, bytes, free_)) return kPoolOverBudget;
        void *p = nullptr;
        if (!pool_alloc(c, &p, bytes, alloc, free_)) return kPoolRefused;
        b = DevBuf{p, bytes};
        c.used += bytes;
    }
    *out = b.p;
    return kPoolOk;
}

}  // namespace dh
