// Which memory a kernel of a solver's device can take, and the device a launch has to be made under.
// Host code on the runtime API only: a host compiler builds it without CUDA's kernel syntax.
#pragma once

#include <cuda_runtime_api.h>
#include <stddef.h>
#include <stdint.h>

#include <initializer_list>

namespace crb200
{
    // Whether a kernel on `device` can take `count` floats at `p`: memory of that device, managed or
    // registered host memory from the first to the last of them, aligned to a float, whichever device is
    // current.  What it cannot take (another device's memory, odd addresses, arrays that end early) goes
    // through the copy engine, which refuses what cannot be copied.
    inline bool kernelReachable(const void *p, size_t count, int device)
    {
        const uintptr_t first = reinterpret_cast<uintptr_t>(p), last = first + (count ? count - 1 : 0) * sizeof(float);
        if (first & 3u)
            return false;
        for (const uintptr_t at : {first, last})
        {
            const void *q = reinterpret_cast<const void *>(at);
            cudaPointerAttributes a{};
            if (cudaPointerGetAttributes(&a, q) != cudaSuccess)
            {
                cudaGetLastError(); // an unknown pointer is not an error of this call
                return false;
            }
            if (!(a.type == cudaMemoryTypeManaged || (a.type == cudaMemoryTypeHost && a.devicePointer == q) ||
                  (a.type == cudaMemoryTypeDevice && a.device == device)))
                return false;
        }
        return true;
    }

    // Makes `device` the calling thread's current device for a scope.  A kernel is launched into a
    // stream only under the stream's device; a copy is enqueued under any.
    class DeviceScope
    {
    public:
        explicit DeviceScope(int device)
        {
            if (cudaGetDevice(&before) == cudaSuccess && before != device)
                changed = cudaSetDevice(device) == cudaSuccess;
        }
        ~DeviceScope()
        {
            if (changed)
                cudaSetDevice(before);
        }
        DeviceScope(const DeviceScope &) = delete;
        DeviceScope &operator=(const DeviceScope &) = delete;

    private:
        int before = 0;
        bool changed = false;
    };
} // namespace crb200
