// Device memory that is taken when it is first needed, in a way that leaves a
// state the next call can use where a call meets a full device.
#pragma once

#include <cstddef>
#include <initializer_list>

namespace mp {

struct Block {
    void **p;
    size_t bytes;
};

// Allocates the blocks in order; where one cannot be had, frees the ones before
// it, leaves every pointer null and returns false.  alloc(void **, size_t) is
// true on success.
template <typename Alloc, typename Release>
bool allocate_all(std::initializer_list<Block> blocks, Alloc alloc, Release release) {
    for (const Block &b : blocks) *b.p = nullptr;
    for (const Block &b : blocks) {
        if (alloc(b.p, b.bytes)) continue;
        *b.p = nullptr;
        for (const Block &q : blocks) {
            if (*q.p) release(*q.p);
            *q.p = nullptr;
        }
        return false;
    }
    return true;
}

// Makes p, of len elements, hold at least `need`: by a new array of `size`, the old
// contents lost.  Where that cannot be had: p null, len 0 and false.
template <typename T, typename Alloc, typename Release>
bool grow(T *&p, long long &len, long long need, long long size, Alloc alloc, Release release) {
    if (p && len >= need) return true;
    if (p) release(p);
    p = nullptr;
    len = 0;
    void *q = nullptr;
    if (!alloc(&q, sizeof(T) * (size_t)size)) return false;
    p = static_cast<T *>(q);
    len = size;
    return true;
}

}  // namespace mp
