// reads_in_place (virgo_b200/csrc/memory_place.h): this device's memory and
// managed memory on 16-byte boundaries, nothing else.  Built and run by
// tests/test_memory_place.py.
#include <cstdio>
#include "memory_place.h"

int main()
{
    int bad = 0;
    for (int device = 0; device < 3; ++device)
        for (int owner = 0; owner < 3; ++owner)
            for (uintptr_t off = 0; off < 32; ++off) {
                const void *p = (const void *)(0x7f0000000000ull + off);
                bad += reads_in_place(p, MEMORY_HOST, owner, device);
                bad += reads_in_place(p, MEMORY_DEVICE, owner, device) != (off % 16 == 0 && owner == device);
                bad += reads_in_place(p, MEMORY_MANAGED, owner, device) != (off % 16 == 0);
            }
    printf(bad ? "%d differ\n" : "places agree\n", bad);
    return bad != 0;
}
