// Test harness: the FP64 solver's staging buffer (csrc/fv2d_hostcopy.h) holds every transfer that goes
// through it: 8 doubles per cell, the face and incidence arrays, 4 doubles per block of the norm reduction.
#include "fv2d_hostcopy.h"
#include <cstdio>
int main() {
    const size_t blocks = 304;
    for (size_t cells : {1, 2, 9, 50, 128, 151, 152, 153, 4000}) {
        const size_t faces = 3 * cells + 1, inc = 2 * faces;
        const size_t have = fv2d::solver_staging_bytes(cells, faces, inc, blocks, sizeof(double));
        for (size_t need : {64 * cells, 4 * (cells + 1), 8 * faces, 4 * inc, 32 * blocks})
            if (have < need) { printf("%zu cells: %zu bytes, %zu needed\n", cells, have, need); return 1; }
    }
    return 0;
}
