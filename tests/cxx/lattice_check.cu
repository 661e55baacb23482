// lattice_check.cu -- host checks of the lattice kernels' own source (dmftpack_gb300/csrc/schur.cuh, df.cuh, smallmat_df.cuh),
// built with -ffp-contract=off: every FP32 operation is then the IEEE one of its device instruction, but for the reciprocal and
// reciprocal root that the device approximates first and refines.
// stdin: one case per line; stdout: one line each:
//   cps <untuned>                        the CTAs per SM that the autotuner times
//   inv2d <re im of a_00 a_01 a_10 a_11> the 2 x 2 inverse in FP64: singular or not, the four entries
//   inv2p, inv3p <entries as doubles>    the 2 x 2 and 3 x 3 inverses in packed double-float, entries read as hi + lo
//   pack <a b c as (re.h re.l im.h im.l)> differences of OpsP's and OpsF's mul, mulc, fma, fms, add, sub: 0 where bits agree
//   rsqrt <h l>                          a^-1/2 in double-float
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "schur.cuh"
#include "smallmat_df.cuh"

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
        } else if (o == "inv2p" || o == "inv3p") {
            const int n = o == "inv2p" ? 2 : 3;
            pdf a2[2][2], a3[3][3];
            for (int e = 0; e < n * n; e++) (n == 2 ? a2[e / 2][e % 2] : a3[e / 3][e % 3]) = OpsP::from(cmk(v[2 * e], v[2 * e + 1]));
            std::printf("%d", n == 2 ? (int)dg::thread_inverse<OpsP, 2>(a2) : (int)dg::thread_inverse<OpsP, 3>(a3));
            for (int e = 0; e < n * n; e++) {
                const double2 z = OpsP::to(n == 2 ? a2[e / 2][e % 2] : a3[e / 3][e % 3]);
                std::printf(" %a %a", z.x, z.y);
            }
        } else if (o == "pack") {
            cdf f[3];
            pdf p[3];
            for (int i = 0; i < 3; i++) {
                f[i] = {{(float)v[4 * i], (float)v[4 * i + 1]}, {(float)v[4 * i + 2], (float)v[4 * i + 3]}};
                p[i] = OpsP::mk(f[i].re, f[i].im);
            }
            auto same = [](cdf x, pdf y) {
                return x.re.h == y.h.x && x.re.l == y.l.x && x.im.h == y.h.y && x.im.l == y.l.y ? 0 : 1;
            };
            std::printf("%d %d %d %d %d %d", same(OpsF::mul(f[0], f[1]), OpsP::mul(p[0], p[1])),
                        same(OpsF::mulc(f[0], f[1]), OpsP::mulc(p[0], p[1])),
                        same(OpsF::fma(f[0], f[1], f[2]), OpsP::fma(p[0], p[1], p[2])),
                        same(OpsF::fms(f[0], f[1], f[2]), OpsP::fms(p[0], p[1], p[2])),
                        same(OpsF::add(f[0], f[1]), OpsP::add(p[0], p[1])), same(OpsF::sub(f[0], f[1]), OpsP::sub(p[0], p[1])));
        } else if (o == "rsqrt") {
            const dfl y = df_rsqrt({(float)v[0], (float)v[1]});
            std::printf("%a %a", y.h, y.l);
        } else return 3;
        std::printf("\n");
    }
    return 0;
}
