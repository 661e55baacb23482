// eig_check.cu -- host checks of the lattice eigensolver's own source (dmftpack_gb300/csrc/eig.cuh).
// stdin: one case per line, "rank <n> <w_0> ... <w_n-1>" (C99 hex, inf and nan as strtod reads them); stdout: the places.
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
        if (std::string(op) != "rank") return 3;
        const int n = (int)v[0];
        for (int i = 0; i < n; i++) std::printf("%d ", eig_rank(v.data() + 1, n, i));
        std::printf("\n");
    }
    return 0;
}
