// Host-side check of the four-phonon kernels' shared-memory sizes: for every branch count,
// both precisions and class counts up to far past what fits, none comes back smaller than
// the tables that it has to hold, also where all branches' tables are just past a multiple
// of 4 GB.  Exit status 0 when all hold.
#include <cstdio>

#include "../../fourphonon_b200/csrc/fp4_internal.h"

static long long checked = 0, bad = 0;

static void check(int nb, int mixed, long long npi) {
    fp4::DevSys S{};
    fp4::DevIfc F{};
    for (int d = 0; d < 3; d++) S.n[d] = 16;
    S.nptk = 4096;
    S.nb = nb;
    S.natoms = nb / 3;
    F.order = 4;
    F.npi = F.ntri = (int)npi;
    F.npt = 48;
    // one branch's tables and the clusters' factors
    const size_t least = (size_t)nb * npi * 9 * (mixed ? 8 : 16) + (size_t)npi * 16;
    const size_t size[3] = {fp4::k4_smem(2, 1, mixed, S, F), fp4::k4_smem(3, 1, mixed, S, F),
                            fp4::k4_multi_smem(mixed, S, F)};
    for (size_t s : size) {
        checked++;
        if (s < least && s < (size_t)INT32_MAX && bad++ < 10)
            printf("%d branches, %lld classes, mixed %d: %zu B for %zu B of tables\n", nb, npi, mixed, s, least);
    }
}

int main() {
    for (int nb = 3; nb <= fp4::kMaxNb; nb += 3)
        for (int mixed = 0; mixed < 2; mixed++) {
            for (long long npi = 1; npi <= 600000; npi += 1 + npi / 64) check(nb, mixed, npi);
            const size_t per = (size_t)nb * nb * 9 * (mixed ? 8 : 16) + 32;  // of a class, all branches
            for (size_t wrap = 1; wrap <= 4; wrap++)
                for (int x = -8; x <= 8; x++) check(nb, mixed, (long long)((wrap << 32) / per) + x);
        }
    printf("%lld sizes, %lld wrong\n", checked, bad);
    return bad ? 1 : 0;
}
