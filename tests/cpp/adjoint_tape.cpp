// Prints kept_segments for lines of "segments segment_bytes limit free".
#include "../../rrea_feedback_warpx_amrex_geant4_gb300/csrc/host/adjoint_tape.hpp"

#include <cstdio>

int main()
{
    long long s, b, l, f;
    while (std::scanf("%lld %lld %lld %lld", &s, &b, &l, &f) == 4) {
        std::printf("%d\n", rrea_host::kept_segments(s, b, l, f));
    }
    return 0;
}
