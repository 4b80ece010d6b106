// context_slots.h -- a value per CUDA context, for state that dies with its
// context (device memory, mapped host memory).
#pragma once
#include <cstdint>

namespace goofy_gpu {

// Values of the N contexts that came last, found by the context's id.  Ids are
// never used again within a process, unlike context handles: after
// cudaDeviceReset a device's primary context has its old handle and a new id,
// so what belonged to the old one is not found.  The value of an id that is
// not there yet is T{} in the slot that was given out longest ago; nothing is
// released for the id it held.
template <typename T, int N>
class ContextSlots {
public:
    T& at(uint64_t id)
    {
        for (int i = 0; i < N; ++i)
            if (id_[i] == id) return value_[i];
        const int i = next_;
        next_ = (next_ + 1) % N;
        id_[i] = id;
        return value_[i] = T{};
    }

private:
    uint64_t id_[N] = {};  // 0: no context's
    T value_[N] = {};
    int next_ = 0;
};

}  // namespace goofy_gpu
