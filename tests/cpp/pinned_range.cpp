// readable_in_place for lines of "host device start size bytes" (decimal): the address or 0, a line each.
#include <cstdio>

#include "pinned.h"

int main() {
    unsigned long long host, device, start, size, bytes;
    while (std::scanf("%llu %llu %llu %llu %llu", &host, &device, &start, &size, &bytes) == 5)
        std::printf("%llu\n", (unsigned long long)axr::readable_in_place(host, bytes, axr::PinnedRange{device, start, size}));
}
