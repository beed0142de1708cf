// Prints, for every object size the entry points accept, the sizes whose chosen
// layout would not fit beside the static shared memory of the teams' or the
// batch's kernel; the last line is the number of layouts looked at.
#include <cstdio>

#include "fit_kernel.cuh"

int main()
{
    const size_t limit = 232448;  // sm_100: shared memory one block may have
    const size_t statics = sizeof(psb::TeamShared) > sizeof(psb::DevObject) + sizeof(psb::DevParams)
                               ? sizeof(psb::TeamShared)
                               : sizeof(psb::DevObject) + sizeof(psb::DevParams);
    const int layouts[3][2] = {{32, 1}, {32, 0}, {16, 0}};  // tile rows, curve statistics in shared memory
    long seen = 0;
    for (int nc = 1; nc <= 81; ++nc) {
        const int ma = nc + 8, rs = (ma + 2) & ~1, ncp = nc <= 16 ? 16 : (nc + 7) & ~7;
        for (int free = 0; free <= 6; ++free)
            for (int nf = 4; nf <= 1024; nf += 4)
                for (int curves = 1; curves <= 256; ++curves)
                    for (int mixed = 0; mixed <= (ncp <= psb::kMaxMixedNcp ? 1 : 0); ++mixed) {
                        const int mfit = ma - free;
                        if (mfit < 1) continue;
                        for (const auto &l : layouts) {
                            const size_t bytes =
                                psb::carve_bytes(nf, mfit, ncp, curves, rs, l[0], l[1], mixed, nullptr, nullptr);
                            if (bytes + psb::kStaticSmem > limit) continue;
                            ++seen;
                            if (bytes + statics > limit)
                                printf("nc %d mfit %d nf %d curves %d mixed %d\n", nc, mfit, nf, curves, mixed);
                            break;
                        }
                    }
    }
    printf("%ld\n", seen);
    return 0;
}
