// Arrays in device and pinned host memory.
#pragma once

#include <utility>

#include "common.cuh"

namespace skmb {

// A typed array in memory that ALLOC / FREE hand out.
template <class T, MemoryBlock (*ALLOC)(size_t), void (*FREE)(const MemoryBlock&)>
class Buffer {
  public:
    Buffer() = default;
    Buffer(const Buffer&) = delete;
    Buffer& operator=(const Buffer&) = delete;
    ~Buffer() { release(); }
    void release() {
        FREE(m_);
        m_ = MemoryBlock{};
        cap_ = 0;
    }
    // Grows (never shrinks) to at least `count` elements; contents are not preserved on growth.
    T* ensure(size_t count) {
        if (count > cap_ || !m_.p) {
            release();
            m_ = ALLOC(sizeof(T) * (count ? count : 1));
            cap_ = count;
        }
        return get();
    }
    T* get() const { return static_cast<T*>(m_.p); }
    size_t capacity() const { return cap_; }
    void swap(Buffer& o) {
        std::swap(m_, o.m_);
        std::swap(cap_, o.cap_);
    }

  private:
    MemoryBlock m_;
    size_t cap_ = 0;
};
template <class T>
using DeviceBuffer = Buffer<T, device_alloc, device_free>;
template <class T>
using PinnedBuffer = Buffer<T, pinned_alloc, pinned_free>;

} // namespace skmb
