// CPU check of the mode index of the per-mode update (csrc/mode_index.cuh): every mode of the
// largest plane that each z length can meet, against integer division.
#include <cstdio>
#include <initializer_list>
#include "mode_index.cuh"

int main() {
    int bad = 0, lengths = 0;
    for (int f : {1, 3, 5, 7})
        for (int nz = 8 * f; nz <= pd::kMaxLength; nz *= 2) {
            if (nz < 16) continue;
            lengths++;
            const int nkk = 2 * (nz / 3) + 1, nkj = 2 * (pd::kMaxLength / 3) + 1;
            for (int q = 0; q < nkj * nkk; q++) {
                int j, k;
                pd::mode_row(q, nkk, j, k);
                if (j != q / nkk || k != q % nkk) { bad++; printf("nz %d q %d: %d %d\n", nz, q, j, k); break; }
            }
        }
    printf("%d lengths %s\n", lengths, bad ? "FAIL" : "OK");
    return bad ? 1 : 0;
}
