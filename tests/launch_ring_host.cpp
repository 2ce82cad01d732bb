// Reads launches "device stream thread tiles" and prints the split each would get on a chip of argv[1] SMs (csrc/launch_ring.h).
#include <cstdio>
#include <cstdlib>

#include "launch_ring.h"

int main(int, char **argv) {
    const int sms = std::atoi(argv[1]);
    wxk::LaunchRing ring;
    int device;
    unsigned long long stream, thread, tiles;
    while (std::scanf("%d %llu %llu %llu", &device, &stream, &thread, &tiles) == 4)
        std::printf("%u\n", wxk::pixel_split(tiles, ring.enter(device, stream, thread, tiles, (uint64_t)sms * wxk::kSplitWarps), sms));
}
