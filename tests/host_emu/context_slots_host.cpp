// context_slots_host.cpp -- TEST ONLY.  context_slots.h on the CPU.
#include "context_slots.h"

static goofy_gpu::ContextSlots<int, 4> slots;

// The value kept for context `id` before it is set to `value`.
extern "C" int swap_value(unsigned long long id, int value)
{
    int& v = slots.at(id);
    const int old = v;
    v = value;
    return old;
}
