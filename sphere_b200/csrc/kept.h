// kept.h -- the arrays that contexts keep between their differentiable sessions.
//
// A session's tape is large and costs more to allocate than a short session to
// run, so a context that ends one parks the tape here and takes it back when it
// begins the next.  While it is parked it belongs to whoever needs the memory: an
// allocation that fails gives every parked array of its device back and is tried
// once more (malloc_or_give_back), and the owner then finds nothing to take.  Host
// code only; any thread.
#pragma once

#include <cstddef>
#include <mutex>
#include <utility>
#include <vector>

namespace sphk {

class KeptArrays {
public:
    // Parks the owner's arrays, which leaves the caller's vector empty, unless the
    // device's parked bytes would pass `limit` (false: nothing is parked).
    bool park(const void *owner, int device, std::vector<void *> &arrays, size_t bytes, size_t limit)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        size_t total = bytes;
        for (const Set &s : sets_)
            if (s.device == device) total += s.bytes;
        if (total > limit || bytes == 0) return false;
        sets_.push_back(Set{owner, device, std::move(arrays), bytes});
        arrays.clear();
        return true;
    }

    // Gives the owner its arrays back (appended to `arrays`); their bytes, or 0
    // where none are parked.
    size_t take(const void *owner, std::vector<void *> &arrays)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        for (size_t k = 0; k < sets_.size(); ++k) {
            if (sets_[k].owner != owner) continue;
            const size_t bytes = sets_[k].bytes;
            arrays.insert(arrays.end(), sets_[k].arrays.begin(), sets_[k].arrays.end());
            sets_.erase(sets_.begin() + (std::ptrdiff_t)k);
            return bytes;
        }
        return 0;
    }

    // The bytes that the owner has parked.
    size_t parked(const void *owner)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        for (const Set &s : sets_)
            if (s.owner == owner) return s.bytes;
        return 0;
    }

    // Frees every parked array of a device; the bytes freed.
    template <class Free>
    size_t give_back(int device, Free free_array)
    {
        std::vector<Set> mine;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            for (size_t k = sets_.size(); k-- > 0;) {
                if (sets_[k].device != device) continue;
                mine.push_back(std::move(sets_[k]));
                sets_.erase(sets_.begin() + (std::ptrdiff_t)k);
            }
        }
        size_t bytes = 0;
        for (Set &s : mine) {
            for (void *p : s.arrays) free_array(p);
            bytes += s.bytes;
        }
        return bytes;
    }

private:
    struct Set {
        const void *owner;
        int device;
        std::vector<void *> arrays;
        size_t bytes;
    };
    std::mutex mutex_;
    std::vector<Set> sets_;
};

// allocate(), and where it says `none` (out of memory) and give_back() freed
// something, allocate() once more.
template <class Allocate, class Result, class GiveBack>
Result malloc_or_give_back(Allocate allocate, Result none, GiveBack give_back)
{
    const Result first = allocate();
    if (first != none || give_back() == 0) return first;
    return allocate();
}

}  // namespace sphk
