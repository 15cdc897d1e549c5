// Test helper: reads "start size address bytes" lines and prints 1 where the range holds the array.
#include <cstdio>
#include "pe_host.h"

int main() {
    unsigned long long start, size, p, bytes;
    while (std::scanf("%llu %llu %llu %llu", &start, &size, &p, &bytes) == 4) std::printf("%d\n", pe::range_holds(start, size, p, bytes) ? 1 : 0);
    return 0;
}
