// Host check (compiled with nvcc, run on the CPU) of the places that the halo walks take in the list of the next pass:
// from any place, those beyond the list and those of a counter that has run over included, the entries lie within the
// list; and walks that go on handing over to a full list leave its length where it is.
#include "halos.cuh"

#include <algorithm>
#include <climits>
#include <cstdio>

using namespace csg;

int main()
{
    const int stack      = 272; // most entries that a walk has left
    long long mismatches = 0;
    const int places[]   = {INT_MIN, INT_MIN + 1, -HALO_MORE, -stack, -1, 0, 1, HALO_MORE - stack - 1, HALO_MORE - stack,
                            HALO_MORE - stack + 1, HALO_MORE - 1, HALO_MORE, HALO_MORE + 1, INT_MAX - stack, INT_MAX};
    for (int at : places)
        for (int left = 0; left <= stack; ++left)
        {
            const int room  = haloRoom(at, left);
            const bool in   = at >= 0 && at < HALO_MORE;
            const int want  = in ? int(std::min<long long>(left, (long long)(HALO_MORE) - at)) : 0;
            const bool fits = room == 0 || (at >= 0 && (long long)(at) + room <= HALO_MORE);
            mismatches += room != want || !fits;
        }
    // 2^24 walks with a full stack each: their sum is 2.1 times the counter's range
    int length      = 0;
    long long taken = 0;
    for (int k = 0; k < 1 << 24; ++k)
    {
        const int at = length;
        if (haloListOpen(length)) length += stack;
        taken += haloRoom(at, stack);
    }
    mismatches += taken != HALO_MORE || length >= HALO_MORE + stack;
    std::printf("mismatches %lld\n", mismatches);
    return mismatches != 0;
}
