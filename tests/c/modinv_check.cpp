// Reads 64-character hexadecimal numbers (below 2^256) from standard input, one per line, and
// prints the inverse mod 2^255 - 19 that modinv.cuh computes, as the kernels use it.
#include <stdint.h>
#include <stdio.h>

#include "../../meikey_b200/csrc/modinv.cuh"

int main() {
    uint32_t x[8], r[8];
    while (scanf("%8x%8x%8x%8x%8x%8x%8x%8x", x + 7, x + 6, x + 5, x + 4, x + 3, x + 2, x + 1, x) == 8) {
        mkinv::invert(x, r);
        for (int i = 7; i >= 0; i--) printf("%08x", r[i]);
        printf("\n");
    }
    return 0;
}
