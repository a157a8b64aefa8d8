// Error message store of the C entry points.
#include "common.cuh"

#include <stdarg.h>
#include <stdio.h>

static thread_local char g_error[512] = "";

extern "C" const char* ti_last_error() { return g_error; }

int ti_fail(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
    return 1;
}

int ti_check_launch(const char* what) {
    cudaError_t err = cudaGetLastError();
    if (err == cudaSuccess) return 0;
    return ti_fail("%s: %s", what, cudaGetErrorString(err));
}

static int current_device_slot() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
    return dev;
}

bool TiPerDevice::first_use() {
    const int dev = current_device_slot();
    return dev < 0 || !done[dev];
}

void TiPerDevice::mark() {
    const int dev = current_device_slot();
    if (dev >= 0) done[dev] = true;
}

// Repeats a tape of launches for `layers` layers.  Call c is `calls[c]` (an entry point's `_taped` form) with the slots from
// first_slot[c] on; before a layer's calls, slot patch_slot[p] of every patch p gets that layer's value.  Returns 0, or one
// more than the number of the call that failed (its library keeps the message).
extern "C" int ti_tape_run(const void* const* calls, const int* first_slot, int num_calls, unsigned long long* slots,
                           const int* patch_slot, int num_patches, const unsigned long long* patch_values, int layers) {
    typedef int (*Taped)(const unsigned long long*);
    for (int layer = 0; layer < layers; ++layer) {
        const unsigned long long* values = patch_values + (size_t)layer * num_patches;
        for (int p = 0; p < num_patches; ++p) slots[patch_slot[p]] = values[p];
        for (int c = 0; c < num_calls; ++c)
            if (((Taped)calls[c])(slots + first_slot[c])) return c + 1;
    }
    return 0;
}
