// The arithmetic of kmc_exp64.cuh on the host: records of three doubles from
// standard input, results to standard output.  One argument, the function.
#include <cstdlib>

#include "device.h"
#include "kmc_exp64.cuh"

using namespace kmc;

int main(int, char **argv)
{
    double2 table[kExpTable];
    for (int j = 0; j < kExpTable; ++j) table[j] = exp_table_entry(j);
    double in[3], out[2];
    while (fread(in, sizeof(double), 3, stdin) == 3) {
        switch (std::atoi(argv[1])) {
        case 0: {       // exp(x + y) = out[0] 2^out[1]
            int k;
            out[0] = exp_split(in[0], in[1], table, k);
            out[1] = k;
            break;
        }
        case 1:         // x / kT and the rest
            out[0] = over_kT(in[0], in[1] == 1.0, in[1], 1.0 / in[1], out[1]);
            break;
        default:        // min(cap, g 2^ex)
            out[0] = scaled_min(in[0], static_cast<int>(in[1]), in[2]);
            out[1] = splittable(in[0]);
        }
        fwrite(out, sizeof(double), 2, stdout);
    }
    return 0;
}
