// idle_buffer.h -- device memory that is kept between calls, and when it goes back.
//
// A buffer of a few GiB is kept idle per device, because allocating and freeing it cost a call 5-20 ms
// on B200.  Other users of the device must not pay for that: the buffer goes back when an allocation of
// this library finds no memory, before a larger one takes its place, and with the last owner (a
// scene handle) on the device.  Plain C++, so that the rules are checked on the host as well.
#pragma once

#include <cstddef>
#include <mutex>
#include <utility>

namespace lum {

// alloc(), and once more after release() if it reports `out_of_memory`.
template <class Error, class Alloc, class Release>
Error alloc_or_release(Error out_of_memory, Alloc alloc, Release release) {
    Error e = alloc();
    if (e == out_of_memory) {
        release();
        e = alloc();
    }
    return e;
}

class IdleBuffer {
public:
    using Free = void (*)(void*);
    explicit IdleBuffer(Free free, size_t most) : free_(free), most_(most) {}

    // The idle buffer if it has *bytes (set to its size); one that is too small goes back, so that
    // it and the one allocated instead are not held together.  Null: the caller allocates.
    void* take(size_t* bytes) {
        std::lock_guard<std::mutex> lk(mu_);
        if (ptr_ && bytes_ < *bytes) drop();
        if (ptr_) *bytes = bytes_;
        bytes_ = 0;
        return std::exchange(ptr_, nullptr);
    }

    // A buffer that no work uses any more: kept if it is the largest and at most `most`, else freed.
    void put(void* ptr, size_t bytes) {
        std::lock_guard<std::mutex> lk(mu_);
        if (owners_ > 0 && bytes <= most_ && bytes > bytes_) {
            std::swap(ptr, ptr_);
            bytes_ = bytes;
        }
        if (ptr) free_(ptr);
    }

    void give_back() {
        std::lock_guard<std::mutex> lk(mu_);
        drop();
    }

    void add_owner() {
        std::lock_guard<std::mutex> lk(mu_);
        ++owners_;
    }
    void remove_owner() {
        std::lock_guard<std::mutex> lk(mu_);
        if (--owners_ == 0) drop();
    }

private:
    void drop() {
        if (ptr_) free_(ptr_);
        ptr_ = nullptr;
        bytes_ = 0;
    }
    std::mutex mu_;
    Free free_;
    size_t most_;
    void* ptr_ = nullptr;
    size_t bytes_ = 0;
    int owners_ = 0;
};

}  // namespace lum
