// Host-only check of which value columns a lane of attn_rows_kernel reads (crabml_b200/csrc/attn_rows_lanes.cuh): every lane that loads stays inside the row, and
// every column of a row is read once for each group of heads and of keys.  Prints "dv heads outside missing" for the sizes given as arguments.  No CUDA call is made.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../crabml_b200/csrc/attn_rows_lanes.cuh"

int main(int argc, char** argv) {
    for (int a = 1; a < argc; a++) {
        const int dv = std::atoi(argv[a]);
        for (int HB = 1; HB <= 16; HB *= 2) {
            const int HG = HB / (HB < 8 ? HB : 8);
            long outside = 0, missing = 0;
            for (int cb = 0; cb * AR_COLS < dv; cb++) {
                const int first = cb * AR_COLS, cols = ar_cols(dv, cb), kgs = ar_lane(0, 0, ar_dvp(dv), cols, HG).kgs;
                std::vector<int> seen((size_t)HG * kgs * cols, 0);
                for (int w = 0; w < AR_WARPS; w++)
                    for (int lane = 0; lane < 32; lane++) {
                        const ArLane l = ar_lane(w, lane, ar_dvp(dv), cols, HG);
                        if (!l.loads) continue;
                        // rows of whole 16 bytes are read 4 columns at a time, others column by column: the first one whatever the row's length
                        const int last = first + l.col + (dv % 4 == 0 ? 3 : 0);
                        if (last >= dv) { outside++; continue; }
                        for (int c = l.col; c < cols && c < l.col + 4; c++) seen[((size_t)l.hg * kgs + l.kg) * cols + c]++;
                    }
                for (int n : seen) missing += n != 1;
            }
            std::printf("%d %d %ld %ld\n", dv, HB, outside, missing);
        }
    }
}
