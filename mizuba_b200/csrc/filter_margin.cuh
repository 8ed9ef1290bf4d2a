// Constants of the narrow phase's filter (k_narrow.cu, which has the argument):
// nodes, the range of sub-interval lengths and the weights of the error margin
// per order.  Host code without CUDA.
#pragma once

#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

namespace mzb
{

constexpr int FILTER_MAX_OP1 = 33;

struct filter_tables {
    double x[FILTER_MAX_OP1 / 2], y[FILTER_MAX_OP1 / 2]; // nodes in (0, 1] of [-1, 1], descending, and their squares
    double node[FILTER_MAX_OP1];                         // nodes of [0, 1], ascending
    double inv_binom[FILTER_MAX_OP1];
    double node_w[FILTER_MAX_OP1];    // F = sum node_w[m] f_m
    double newton[FILTER_MAX_OP1];    // margin per Newton coefficient
    double value, square, norm, mono; // and per sqrt(F) P, F, P^2 and sum |f_k|
    double rf_lo, rf_hi;              // range of sub-interval lengths
};

// Where the filter's argument holds for order n: the reference formulation
// divides differences of f by node distances c rf_int, so its k-th divided
// differences are at most 2^k max f / (G_k rf_int^k), G_k the product of the
// smallest node distances at lags 1 to k; with max f <= 1e30 they stay below
// 1e280 for rf_int >= rf_lo, and neither rf_int^n nor its inverse leaves the
// exponent range for rf_int in [rf_lo, rf_hi].
inline void filter_range(filter_tables &t, int n)
{
    t.rf_lo = std::pow(10.0, -250.0 / n);
    t.rf_hi = std::pow(10.0, 200.0 / n);
    double log_g = 0;
    for (int k = 1; k <= n; ++k) {
        double gap = 1.0;
        for (int j = k; j <= n; ++j) gap = std::min(gap, t.node[j] - t.node[j - k]);
        log_g += std::log10(gap);
        t.rf_lo = std::max(t.rf_lo, std::pow(10.0, (k * std::log10(2.0) + 30.0 - log_g - 280.0) / k));
    }
}

// The weights of the margin M for order n.  Everything here is a
// linear map of the few dozen numbers of an item; the maps are applied to unit
// vectors in long double and the results' largest Bernstein coefficients taken.
inline void filter_margins(filter_tables &t, int n)
{
    using real = long double;
    using vec = std::vector<real>;
    const double *c = t.node;
    const size_t m = size_t(n) + 1;
    // p (s - r) and the degree elevation of p, in Bernstein form over [0, 1].
    auto times_root = [](const vec &p, real r) {
        const int d = int(p.size()) - 1;
        vec q(size_t(d) + 2, 0);
        for (int i = 0; i <= d + 1; ++i) {
            if (i <= d) q[i] -= r * (d + 1 - i) * p[i] / (d + 1);
            if (i > 0) q[i] += (1 - r) * i * p[i - 1] / (d + 1);
        }
        return q;
    };
    auto elevated = [n](vec p) {
        while (int(p.size()) <= n) {
            const int d = int(p.size()) - 1;
            vec q(size_t(d) + 2, 0);
            for (int i = 0; i <= d + 1; ++i)
                q[i] = ((i ? i * p[i - 1] : 0) + (i <= d ? (d + 1 - i) * p[i] : 0)) / (d + 1);
            p = std::move(q);
        }
        return p;
    };
    auto largest = [](const vec &p) {
        real a = 0;
        for (const real v : p) a = std::max(a, std::fabs(v));
        return a;
    };
    // Newton basis w_l = prod_{i < l} (s - c_i), also at degree n.
    std::vector<vec> w(m), wn(m);
    for (int l = 0; l <= n; ++l) {
        w[l] = l ? times_root(w[l - 1], c[l - 1]) : vec{1};
        wn[l] = elevated(w[l]);
    }
    // Bernstein coefficients from the divided differences of level k (entries
    // from k on; the ones before are zero).
    auto bernstein = [&](vec f, int k) {
        for (int q = k; q < n; ++q)
            for (int j = n; j > q; --j) f[j] = (f[j] - f[j - 1]) / (real(c[j]) - c[j - q - 1]);
        vec b(m, 0);
        for (int l = k; l <= n; ++l)
            for (int i = 0; i <= n; ++i) b[i] += f[l] * wn[l][i];
        return b;
    };
    // What a node's value can do to a Bernstein coefficient.
    real L = 0;
    for (int j = 0; j <= n; ++j) {
        vec e(m, 0);
        e[j] = 1;
        const real a = largest(bernstein(std::move(e), 0));
        t.node_w[j] = double(a);
        L += a;
    }
    // Divided difference j of level k: its relative rounding in both
    // formulations, and what an error of it does to the coefficients.
    std::vector<vec> dd(m, vec(m, 0));
    for (int k = 1; k <= n; ++k)
        for (int j = k; j <= n; ++j) {
            vec e(m, 0);
            e[j] = 1;
            dd[k][j] = (7 + (real(c[j]) + c[j - k]) / (real(c[j]) - c[j - k])) * largest(bernstein(std::move(e), k));
        }
    // Step k of Newton form -> monomials writes the coefficients of
    // s^(j - k) w_k: four roundings of at most the sum of magnitudes there.
    std::vector<vec> nm(m, vec(m, 0));
    for (int k = 0; k < n; ++k) {
        vec p = w[k];
        for (int j = k; j < n; ++j) {
            nm[k][j] = 4 * largest(elevated(p));
            p = times_root(p, 0);
        }
    }
    const real u = 1.1102230246251565e-16L, slack = 1.05L; // slack: second order and this function's own rounding
    for (int l = 0; l <= n; ++l) {
        real g = 0;
        vec f(m); // w_l at the nodes, then its divided differences level by level (none beyond l)
        for (int j = 0; j <= n; ++j) {
            f[j] = 1;
            for (int i = 0; i < l; ++i) f[j] *= real(c[j]) - c[i];
        }
        for (int k = 1; k <= l; ++k)
            for (int j = n; j >= k; --j) {
                f[j] = (f[j] - f[j - 1]) / (real(c[j]) - c[j - k]);
                g += dd[k][j] * std::fabs(f[j]);
            }
        vec a(m, 0); // magnitudes of the coefficients that w_l contributes to
        a[l] = 1;
        for (int k = n - 1; k >= 0; --k)
            for (int j = k; j < n; ++j) {
                a[j] += c[k] * a[j + 1];
                g += nm[k][j] * a[j];
            }
        t.newton[l] = double(slack * u * g);
    }
    t.value = double(slack * u * std::sqrt(L) * 78.4);
    t.square = double(slack * u * 10);
    t.norm = double(slack * u * u * L * 1537);
    t.mono = double(slack * u * (6 * n + 24));
}

// All of it for the op1 given nodes.
inline filter_tables make_filter_tables(const double *nodes, int op1)
{
    filter_tables t{};
    const int n = op1 - 1;
    double b = 1.0;
    for (int i = 0; i <= n; ++i) {
        t.node[i] = nodes[i];
        t.inv_binom[i] = 1.0 / b;
        b = b * (n - i) / (i + 1);
    }
    for (int m = 0; m < op1 / 2; ++m) {
        t.x[m] = 2.0 * nodes[n - m] - 1.0;
        t.y[m] = t.x[m] * t.x[m];
    }
    filter_range(t, n);
    filter_margins(t, n);
    return t;
}

} // namespace mzb
