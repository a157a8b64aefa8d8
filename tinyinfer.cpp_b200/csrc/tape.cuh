// Entry points that a tape of launches can call: `TI_TAPED(ti_x)` defines `ti_x_taped`, which takes the arguments of ti_x
// as an array of 64-bit slots (pointers and whole numbers as they are, a float in the low half) and hands each on with the
// type that ti_x declares.  kernels/tape.py records such calls, ti_tape_run (common.cu) repeats them.
#pragma once

#include <stdint.h>
#include <string.h>

#include <type_traits>
#include <utility>

template <typename T> T ti_slot_as(unsigned long long v) {
    if constexpr (std::is_pointer_v<T>) {
        return (T)(uintptr_t)v;
    } else if constexpr (std::is_same_v<T, float>) {
        const unsigned bits = (unsigned)v;
        float f;
        memcpy(&f, &bits, sizeof f);
        return f;
    } else {
        static_assert(std::is_integral_v<T>, "a slot holds a pointer, a float or a whole number");
        return (T)v;
    }
}
template <typename... A, size_t... I>
int ti_call_slots(int (*fn)(A...), const unsigned long long* slots, std::index_sequence<I...>) {
    return fn(ti_slot_as<A>(slots[I])...);
}
template <typename... A> int ti_call_slots(int (*fn)(A...), const unsigned long long* slots) {
    return ti_call_slots(fn, slots, std::index_sequence_for<A...>{});
}

#define TI_TAPED(name) \
    extern "C" int name##_taped(const unsigned long long* slots) { return ti_call_slots(&name, slots); }
