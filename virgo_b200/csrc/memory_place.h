// Which memory a kernel may read where it is.  Host code without CUDA headers,
// so that it can be checked without several GPUs.
#pragma once
#include <cstdint>

enum MemoryKind { MEMORY_HOST, MEMORY_DEVICE, MEMORY_MANAGED };

// Whether a kernel on `device` may read 16-byte words at p, memory of the given
// kind (of `owner`, for device memory).  Another device's memory may not be
// mapped here: without peer access a kernel that touches it faults, while a
// copy by the driver goes through.
inline bool reads_in_place(const void *p, MemoryKind kind, int owner, int device)
{
    if ((uintptr_t)p & 15) return false;
    return kind == MEMORY_MANAGED || (kind == MEMORY_DEVICE && owner == device);
}
