// lattice_check.cu -- host checks of the lattice kernels' own source (dmftpack_gb300/csrc/schur.cuh).
// stdin: one case per line; stdout: one line each:
//   cps <untuned>                        the CTAs per SM that the autotuner times
//   inv2d <re im of a_00 a_01 a_10 a_11> the 2 x 2 inverse in FP64: singular or not, the four entries
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
        } else if (o == "inv2d") {
            double2 a[2][2];
            for (int e = 0; e < 4; e++) a[e / 2][e % 2] = cmk(v[2 * e], v[2 * e + 1]);
            std::printf("%d", (int)dg::thread_inverse<OpsD, 2>(a));
            for (int e = 0; e < 4; e++) std::printf(" %a %a", a[e / 2][e % 2].x, a[e / 2][e % 2].y);
        } else return 3;
        std::printf("\n");
    }
    return 0;
}
