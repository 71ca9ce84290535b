// lbm_device_list.h -- a list in device memory that is replaced as a whole.  No CUDA in here: what allocates,
// fills and frees comes as a parameter, so that its errors can be tested on the host.
#pragma once

#include <stddef.h>

#include <vector>

namespace lbm {

// Mem: alloc(void**, bytes), upload(dst, src, bytes) and release(ptr); the first two return an error that is
// Mem::OK on success
template <class T, class Mem>
struct DeviceList {
    T* data = nullptr;
    int count = 0;
    DeviceList() = default;
    DeviceList(const DeviceList&) = delete;
    DeviceList& operator=(const DeviceList&) = delete;

    // After an error the former list is in place, data and count: kernels read `count` entries of it.
    decltype(Mem::OK) replace(const std::vector<T>& list) {
        T* fresh = nullptr;
        const size_t bytes = list.size() * sizeof(T);
        auto e = Mem::alloc((void**)&fresh, bytes);
        if (e != Mem::OK) return e;
        e = Mem::upload(fresh, list.data(), bytes);
        if (e != Mem::OK) {
            Mem::release(fresh);
            return e;
        }
        if (data) Mem::release(data);
        data = fresh;
        count = (int)list.size();
        return e;
    }
    void clear() {
        if (data) Mem::release(data);
        data = nullptr;
        count = 0;
    }
};

}  // namespace lbm
