// Both formulations of an item of the narrow phase (the reference's and the
// filter's, mizuba_b200/csrc/k_narrow.cu) operation for operation on the host,
// for random pairs: prints per order and kind of coefficients the largest
// difference of their Bernstein coefficients over the filter's margin.
//   filter_margin_harness ORDER PAIRS SEED
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "filter_margin.cuh"

using vec = std::vector<double>;
using pair_t = vec[2][3]; // [object][coordinate]

static double pairwise(vec t)
{
    while (t.size() > 1) {
        vec r;
        for (size_t k = 0; k < t.size(); k += 2) r.push_back(k + 1 < t.size() ? t[k] + t[k + 1] : t[k]);
        t = r;
    }
    return t[0];
}
static vec powers(double a, int op1)
{
    vec p(op1, 1.0);
    p[1] = a;
    for (int i = 2; i < op1; ++i) p[i] = i % 2 == 0 ? p[i / 2] * p[i / 2] : p[i / 2 + 1] * p[i / 2];
    return p;
}
static double binom(int n, int k)
{
    double b = 1;
    for (int i = 0; i < k; ++i) b = b * (n - i) / (i + 1);
    return b;
}
// The difference table of e: the Bernstein coefficients.
static vec differences(vec e)
{
    vec b{e[0]};
    while (e.size() > 1) {
        for (size_t j = 0; j + 1 < e.size(); ++j) e[j] = e[j] + e[j + 1];
        e.pop_back();
        b.push_back(e[0]);
    }
    return b;
}

static vec reference(const double *node, int op1, const pair_t &c, const double (&delta)[2], double rf)
{
    const int n = op1 - 1;
    vec f(op1), vs(op1);
    for (int r = 0; r < 6; ++r) {
        const int v = r >> 1, o = r & 1;
        vec tr = c[o][v];
        if (delta[o] != 0) {
            const vec ap = powers(delta[o], op1);
            for (int i = 0; i < op1; ++i) {
                vec t;
                for (int k = 0; i + k < op1; ++k) t.push_back((c[o][v][i + k] * binom(i + k, k)) * ap[k]);
                tr[i] = pairwise(t);
            }
        }
        for (int m = 0; m < op1; ++m) {
            const double x = node[m] * rf;
            double h = tr[n];
            for (int k = n - 1; k >= 0; --k) h = tr[k] + h * x;
            if (o == 0) {
                vs[m] = h;
            } else {
                const double d = vs[m] - h;
                f[m] = v == 0 ? d * d : f[m] + d * d;
            }
        }
    }
    for (int k = 0; k < n; ++k)
        for (int j = n; j > k; --j) f[j] = (f[j] - f[j - 1]) / (node[j] * rf - node[j - k - 1] * rf);
    for (int k = n - 1; k >= 0; --k)
        for (int j = k; j < n; ++j) f[j] = f[j] - (node[k] * rf) * f[j + 1];
    const vec dp = powers(rf, op1);
    for (int k = 0; k < op1; ++k) f[k] = (f[k] * dp[k]) / binom(n, k);
    return differences(f);
}

static vec filter(const mzb::filter_tables &t, int op1, const pair_t &c, const double (&delta)[2], double rf, double &M)
{
    const int n = op1 - 1;
    const double h = 0.5 * rf;
    vec f(op1);
    double P2 = 0, F = 0, Ms = 0;
    for (int v = 0; v < 3; ++v) {
        vec s[2] = {c[0][v], c[1][v]};
        double pc = 0;
        for (int o = 0; o < 2; ++o) {
            const double a = delta[o] + h, e = (delta[o] + rf) * 1.08;
            double p = std::fabs(s[o][n]);
            for (int k = n - 1; k >= 0; --k) p = std::fma(p, e, std::fabs(s[o][k]));
            pc += p;
            for (int i = 0; i < n; ++i)
                for (int k = n - 1; k >= i; --k) s[o][k] = std::fma(a, s[o][k + 1], s[o][k]);
        }
        P2 = std::fma(pc, pc, P2);
        double hp = h;
        vec g = s[0];
        g[0] = g[0] - s[1][0];
        for (int k = 1; k < op1; ++k) {
            g[k] = (g[k] - s[1][k]) * hp;
            hp *= h;
        }
        auto add = [&](int m, double d) { f[m] = v == 0 ? d * d : std::fma(d, d, f[m]); };
        const int ev = n & ~1, od = (n - 1) | 1;
        for (int m = 0; m < op1 / 2; ++m) {
            double even = g[ev], odd = g[od];
            for (int k = ev - 2; k >= 0; k -= 2) even = std::fma(even, t.y[m], g[k]);
            for (int k = od - 2; k >= 1; k -= 2) odd = std::fma(odd, t.y[m], g[k]);
            add(n - m, std::fma(t.x[m], odd, even));
            add(m, std::fma(-t.x[m], odd, even));
        }
        if (op1 & 1) add(n / 2, g[0]);
    }
    for (int m = 0; m < op1; ++m) F = std::fma(t.node_w[m], f[m], F);
    for (int k = 0; k < n; ++k)
        for (int j = n; j > k; --j) f[j] = (f[j] - f[j - 1]) * (1.0 / (t.node[j] - t.node[j - k - 1]));
    M = 1e-250;
    for (int k = 0; k < op1; ++k) M = std::fma(t.newton[k], std::fabs(f[k]), M);
    for (int k = n - 1; k >= 0; --k)
        for (int j = k; j < n; ++j) f[j] = std::fma(-t.node[k], f[j + 1], f[j]);
    for (int k = 0; k < op1; ++k) Ms += std::fabs(f[k]);
    M += Ms * t.mono + std::fma(t.value * std::sqrt(F), std::sqrt(P2), std::fma(t.square, F, t.norm * P2));
    for (int k = 0; k < op1; ++k) f[k] = f[k] * t.inv_binom[k];
    return differences(f);
}

int main(int argc, char **argv)
{
    if (argc != 4) return 2;
    const int n = std::atoi(argv[1]), op1 = n + 1, pairs = std::atoi(argv[2]);
    std::mt19937_64 gen(std::strtoull(argv[3], nullptr, 10));
    auto uni = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); };
    auto log_uni = [&](double a, double b) { return std::exp(uni(std::log(a), std::log(b))); };
    double node[mzb::FILTER_MAX_OP1];
    for (int m = 0; m < op1; ++m)
        node[n - m] = (std::cos((2. * m + 1.) / (2. * op1) * 3.14159265358979323846) + 1.) / 2.;
    const mzb::filter_tables t = mzb::make_filter_tables(node, op1);
    // Coefficients of one size, falling off, growing; shifted far against the
    // interval; two nearly equal objects over intervals of any length.
    for (int kind = 0; kind < 5; ++kind) {
        double worst = 0;
        for (int p = 0; p < pairs; ++p) {
            const double amp = log_uni(1.0, 1000.0);
            const double ratio = kind == 1 ? uni(0.3, 1.0) : kind == 2 ? uni(1.0, 2.0) : kind == 3 ? 0.5 : 1.0;
            const double rf = kind == 3 ? log_uni(1e-3, 2.0) : kind == 4 ? log_uni(1e-4, 1e3) : 1.0;
            double delta[2] = {0, 0};
            if (kind == 3) delta[0] = uni(0.0, 3.0), delta[1] = uni(0.0, 3.0);
            if (kind == 4) delta[0] = uni(0.0, 1.0) * rf, delta[1] = uni(0.0, 1e-3) * rf;
            const double base = kind == 4 ? 1.0 / (1.5 * rf) : ratio;
            pair_t c;
            for (int v = 0; v < 3; ++v)
                for (int o = 0; o < 2; ++o)
                    for (int k = 0; k < op1; ++k) {
                        const double x = amp * uni(0.3, 1.0) * (gen() & 1 ? 1.0 : -1.0) * std::pow(base, k);
                        c[o][v].push_back(kind == 4 && o == 1 ? c[0][v][k] * (1.0 + 1e-3 * uni(-1.0, 1.0)) : x);
                    }
            c[0][0][0] += amp * uni(0.0, 30.0);
            double M;
            const vec a = reference(node, op1, c, delta, rf), b = filter(t, op1, c, delta, rf, M);
            for (int i = 0; i < op1; ++i) worst = std::fmax(worst, std::fabs(a[i] - b[i]) / M);
        }
        std::printf("%d %.6g\n", kind, worst);
    }
    return 0;
}
