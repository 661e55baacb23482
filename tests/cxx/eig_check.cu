// eig_check.cu -- host checks of the lattice eigensolver's own source (dmftpack_gb300/csrc/eig.cuh).
// stdin: one case per line, numbers in C99 hex (inf and nan as strtod reads them); stdout: one line each:
//   rank <n> <w_0> ... <w_n-1>       the places of the values in ascending order
//   tan <r> <d>                      the tangent of a rotation in FP64
//   tandf <r.h> <r.l> <d.h> <d.l>    in double-float (hi lo)
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "eig.cuh"

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
        if (o == "rank") {
            const int n = (int)v[0];
            for (int i = 0; i < n; i++) std::printf("%d ", eig_rank(v.data() + 1, n, i));
        } else if (o == "tan") {
            std::printf("%a", jacobi_tan(v[0], v[1]));
        } else if (o == "tandf") {
            const dfl t = jacobi_tan(dfl{(float)v[0], (float)v[1]}, dfl{(float)v[2], (float)v[3]});
            std::printf("%a %a", t.h, t.l);
        } else return 3;
        std::printf("\n");
    }
    return 0;
}
