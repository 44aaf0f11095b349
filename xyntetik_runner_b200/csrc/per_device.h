// What is asked of the driver once, such as more shared memory for a kernel, holds for the device that was current then: another
// device of the same process asks for itself.  (Host code without CUDA in it: common.cuh says which device is current.)
#pragma once

#define XR_DEVICES 64

// Whether `ask()` has succeeded on `device`: it is called until it does, then never again there.  Threads that meet here at the same
// time ask twice, which changes nothing.
template <typename Ask>
static inline bool xr_once_on_device(bool (&done)[XR_DEVICES], int device, Ask ask) {
    if (device < 0 || device >= XR_DEVICES) return ask();
    if (!done[device]) done[device] = ask();
    return done[device];
}
