// round0_windows(): every rank lies in a window, and no dictionary is read more
// often than the measured line between windows and one pass allows.  Host only.
#include "gbwt_internal.cuh"
#include <stdio.h>

int main()
{
    const uint64_t W = gbwt::R0_WINDOW;
    int failures = 0;
    for (uint64_t N = 1; N < 0xFFFFFF00ull; N = N + N / 7 + 1)
        for (uint32_t texts : {1u, 2u, 4096u}) {
            const uint64_t w = gbwt::round0_windows((uint32_t)N, texts);
            const bool apart = N / texts <= W + W / 2, large = N > 20 * W;
            if (apart || large ? w != 0 : (w * W < N || (w - 1) * W >= N || w > 20)) {
                printf("N %llu texts %u: %llu windows\n", (unsigned long long)N, texts, (unsigned long long)w);
                failures++;
            }
        }
    return failures ? 1 : 0;
}
