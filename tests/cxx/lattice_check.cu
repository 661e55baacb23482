// lattice_check.cu -- host checks of the lattice kernels' own source (dmftpack_gb300/csrc/schur.cuh).
// stdin: one case per line; stdout: one line each:
//   cps <untuned>     the CTAs per SM that the autotuner times
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "schur.cuh"

int main() {
    static char line[1 << 16];
    while (std::fgets(line, sizeof line, stdin)) {
        char op[32];
        int off = 0;
        if (std::sscanf(line, "%31s%n", op, &off) != 1) continue;
        std::vector<double> v;
        for (char *s = line + off, *end = nullptr;; s = end) {
            const double x = std::strtod(s, &end);
            if (end == s) break;
            v.push_back(x);
        }
        const std::string o(op);
        if (o == "cps") {
            int c[4];
            const int n = dg::schur_cps_candidates((int)v[0], c);
            for (int i = 0; i < n; i++) std::printf("%d ", c[i]);
        } else return 3;
        std::printf("\n");
    }
    return 0;
}
