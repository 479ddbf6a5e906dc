// Device memory that is taken when it is first needed: all of it or none, so
// that a call which meets a full device leaves a state that the next call can
// use.
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

}  // namespace mp
