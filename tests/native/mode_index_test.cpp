// CPU check of the mode index of the per-mode update (csrc/mode_index.cuh): every mode of the
// largest plane that the z length given as argument can meet, against integer division.
#include <cstdio>
#include <cstdlib>
#include "mode_index.cuh"

int main(int argc, char** argv) {
    const int nz = argc > 1 ? atoi(argv[1]) : 0;
    if (nz < 1 || nz > pd::kMaxLength) return 2;
    const int nkk = 2 * (nz / 3) + 1, nkj = 2 * (pd::kMaxLength / 3) + 1;
    for (int q = 0; q < nkj * nkk; q++) {
        int j, k;
        pd::mode_row(q, nkk, j, k);
        if (j != q / nkk || k != q % nkk) {
            printf("nz %d q %d: %d %d\n", nz, q, j, k);
            return 1;
        }
    }
    printf("%d modes OK\n", nkj * nkk);
    return 0;
}
