// Host check of lsq_decide (csu_b200/csrc/cuda/lsqdd.cuh) against the x86-64 host's x87 long double: every gradient
// component it rounds equals the reference's formula (solverCalcGrad3, solver.c:1031-1074), bit for bit and sign of
// zero included, on random, strongly stretched, axis-aligned, one-directional, nearly uniform and uniform fields of
// three and four neighbours, over the exponents a solver meets. Prints counts; exit status 1 on any mismatch.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "../../csu_b200/csrc/cuda/lsqdd.cuh"

using namespace csu;

// k / det as the host layout builds it (layout.c): double-double product with the corrected reciprocal
static DD over(long double k, long double det)
{
    double dh = (double)det, dl = (double)(det - (long double)dh);
    double r = 1.0 / dh, e = fma(-dh, r, 1.0);
    e = e - dl * r;
    double re = e * r, rs = r + re, rl = re - (rs - r);
    double h = (double)k, l = (double)(k - (long double)h);
    double p = h * rs, t = fma(h, rs, -p) + (h * rl + l * rs), z = p + t;
    DD q = {z, t - (z - p)};
    return q;
}

int main(int argc, char** argv)
{
    long n = argc > 1 ? atol(argv[1]) : 200000;
    std::mt19937_64 rng(20240607);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    std::uniform_int_distribution<int> E(-40, 40);
    const int KINDS = 7;
    long tried[KINDS] = {}, decided[KINDS] = {}, bad = 0;
    for (long i = 0; i < n * KINDS; i++) {
        const int kind = i % KINDS, nn = 3 + (int)(rng() & 1);
        const double scale = ldexp(1.0, E(rng)), size = ldexp(1.0, E(rng) / 2), thin = kind == 1 ? 1e-5 : 1.0;
        double dx[4], dy[4], du[4];
        const double gx = U(rng), gy = kind == 3 ? 0.0 : U(rng);
        for (int j = 0; j < nn; j++) {
            const double a = 2 * M_PI * (j + 0.3 * U(rng)) / nn;
            dx[j] = size * cos(a);
            dy[j] = size * thin * sin(a);
            if (kind == 2) { // axis aligned: b is exactly zero
                dx[j] = (j & 1) ? 0.0 : size * (j ? -1 : 1);
                dy[j] = (j & 1) ? size * (j > 1 ? -1 : 1) : 0.0;
            }
            du[j] = scale * (gx * dx[j] + gy * dy[j] + 0.1 * size * U(rng));
            if (kind == 3) du[j] = scale * gx * dx[j];                       // a field of x alone
            if (kind == 4) du[j] = scale * ((rng() & 1) ? 0.0 : 1e-12 * U(rng));
            if (kind == 5) du[j] = 0.0;
            if (kind == 6) du[j] = (1.0 + 1e-9 * scale * U(rng)) - 1.0;      // differences of rounded values
        }
        long double a = 0, b = 0, c = 0, A = 0, B = 0;
        LsqSum X, Y;
        for (int j = 0; j < nn; j++) {
            a += dx[j] * dx[j];
            b += dx[j] * dy[j];
            c += dy[j] * dy[j];
            A += dx[j] * du[j];
            B += dy[j] * du[j];
            if (j == 1) {
                X = lsq_sum2(dx[0] * du[0], dx[1] * du[1]);
                Y = lsq_sum2(dy[0] * du[0], dy[1] * du[1]);
            } else if (j > 1) {
                lsq_sum_add(X, dx[j] * du[j]);
                lsq_sum_add(Y, dy[j] * du[j]);
            }
        }
        const long double det = a * c - b * b;
        const double want[2] = {(double)((c * A - b * B) / det), (double)((-b * A + a * B) / det)};
        const DD ka = over(a, det), kb = over(b, det), kc = over(c, det);
        for (int y = 0; y < 2; y++) {
            double q;
            tried[kind]++;
            if (!lsq_decide(y ? ka : kc, kb, y ? Y : X, y ? X : Y, &q)) continue;
            decided[kind]++;
            if (memcmp(&q, &want[y], 8) != 0) {
                if (bad++ < 10) printf("kind %d component %d: %.17g instead of %.17g\n", kind, y, q, want[y]);
            }
        }
    }
    printf("mismatches=%ld", bad);
    for (int k = 0; k < KINDS; k++) printf(" decided%d=%.5f", k, (double)decided[k] / tried[k]);
    printf("\n");
    return bad ? 1 : 0;
}
