// rules.cu — compressed quadrature rules of the far pass.
//
// The reference integrates a cell with the midpoint rule of its n x n split
// (integral_universal.h:38-220): n^2 equal sub-cells, one node each. Away from
// the cell the far integrands are smooth over it, so that sum is itself an
// integral (of a discrete measure) that a Gauss rule of that measure gives with
// far fewer nodes: a rule with m nodes per direction reproduces the n-node sum
// of every polynomial up to degree 2m - 1. The far kernels take, per (warp,
// cell), the shortest rule whose truncation error is below rounding, else the
// n^2-node table; the result is the reference's n x n sum to rounding.
//
//   Quads:     tensor products of the m-point Gauss rule of n equidistant
//              points (the discrete, Gram counterpart of Gauss-Legendre), by
//              the recurrence coefficients (Stieltjes procedure) and the roots
//              of the resulting polynomial. Nodes are mapped bilinearly and
//              weighted by the bilinear Jacobian, whose value at a sub-cell's
//              centre is that sub-cell's area.
//              Between them symmetric rules of total degree 5, 7, 9, 11 (8, 12,
//              20, 28 nodes; orbit structures of Burnside 1908, Tyler 1953 and, for
//              20 and 28 nodes, Rabinowitz & Richter, Math. Comp. 23, 1969), whose
//              orbit parameters are solved by Newton's method for the moments of the
//              n x n midpoints, from start values for the continuous measure.
//   Triangles: symmetric rules of degree 5, 6, 8, 10 and 12 (7, 12, 16, 25, 33
//              nodes; the orbit structures of Radon and of Dunavant, Int. J.
//              Numer. Meth. Eng. 21, 1985), solved the same way for the n^2
//              sub-triangle centroids; from n = 16 on also four copies on the
//              four sub-triangles, whose lattices make up the whole one.
//
// Where a rule may be used is decided by two numbers per cell and rule: a
// distance rmin and a wave number kmax. With theta = rho / r0 (rho: largest
// node distance from the centre, r0: distance of the point) and kappa = |k| rho,
// the error relative to sum w |F| is bounded by
//   sum_d D_d sum_{a + b = d} C_a theta^a kappa^b / b!,   C_a = (a+1)(a+2)/2,
// D_d the rule's error in the cell's own d-th moments (the largest over 32
// directions, measured per quad: it covers distorted, degenerate and
// non-planar cells, whose Jacobian is no polynomial). C_a is the growth of the
// Taylor coefficients of 1/r^3. rmin and kmax are where the terms of theta alone
// (b = 0) and of kappa alone (a = 0) reach the tolerance.
//   Real k: both may be at their limit; e^{ikr} turns the terms of different b
//   against each other. Measured there, over shapes (squares, rectangles to 6:1,
//   trapezoids to triangles, twisted and skew cells, triangles to needles) and
//   directions: at most 0.7 of the FP32 tolerance and 1.5 of the FP64 one.
//   Complex k: e^{-Im k r} makes them add. With both at their limit the error was up
//   to 34 (FP32) and 67 (FP64) times the tolerance, so the limits share it:
//   theta / theta_max + |Im k| / kmax <= 1. Because (C_a a!)^(1/a) grows with a, the
//   terms of each degree are then below those of a binomial (x + y)^d whose ends are
//   the two parts, hence below the part of them that the fractions take. Measured: 1.03
//   and 1.8.
// Moment differences below kRuleFloor count as none, so that much (an ulp or two) can
// come on top in FP64. Compared with the true error the theta part is 0.79 - 2 times it
// for the tensor rules (taken 1.6 times); for the total-degree rules, whose error is one
// angular harmonic that real directions see only in part, up to 2.1, 16, 8 and 140 times
// too small (taken 2.6, 20, 10 and 175 times). The kappa part (real directions) is 0.98 - 4
// times the error, taken 1.5 times. An affine triangle needs no measurement: its error is
// (alpha theta)^(D+1) and (beta kappa)^(D+1) with alpha, beta the largest over
// shapes (equilateral to needles of height 0.02) and directions.
#include <cmath>
#include <map>
#include <mutex>
#include <utility>

#include "internal.h"
#include "ops.cuh"

namespace bielcc_gpu {

// Truncation allowed by a rule, relative to sum w |F| of the pair: an order
// below the rounding of the FP32 node sum (1.1e-7 rms per pair, measured) and
// of the FP64 one.
#ifndef BIELCC_RULE_TOL32
#define BIELCC_RULE_TOL32 1e-8
#endif
constexpr double kRuleTol32 = BIELCC_RULE_TOL32, kRuleTol64 = 3e-17;
// Moments agree to rounding only; differences below this are rounding (of the
// nodes and weights: the sums of the low degrees are compensated).
constexpr double kRuleFloor = 4e-16;
constexpr int kRuleDeg = 18;       // moments D_0 .. D_17 are compared
constexpr int kRuleMaxNodes = 400;  // nodes of all levels of one (shape, n)
constexpr int kRuleMaxSym = 40;     // nodes of one symmetric rule

namespace {

struct RuleHost {
    int n_lev = 0, total = 0;
    int cnt[kMaxRules], off[kMaxRules];
    double factor[kMaxRules];  // quads: on the moment bound's theta part
    double tmax[kMaxRules][2], kmax[kMaxRules][2];  // theta and kappa limits (FP32, FP64): triangles' own, quads' caps
    double s[kRuleMaxNodes], t[kRuleMaxNodes], w[kRuleMaxNodes];
};

// m-point Gauss rule of the measure sum_i delta((i + 1/2) / n): abscissae in
// (0, 1), weights of sum 1. Recurrence coefficients by the Stieltjes procedure
// (the measure is symmetric about 1/2, so only the off-diagonal ones), roots by
// bisection between those of the previous polynomial, weights 1 / sum p_k^2 of
// the orthonormal polynomials.
void discrete_gauss(int n, int m, long double* x, long double* w) {
    typedef long double ld;
    std::vector<ld> t(n), p0(n, 0.0L), p1(n, 1.0L), b(m + 1, 0.0L), nrm(m + 1, 0.0L);
    for (int i = 0; i < n; i++) t[i] = (2.0L * i + 1.0L) / n - 1.0L;
    nrm[0] = n;
    for (int j = 1; j <= m; j++) {
        for (int i = 0; i < n; i++) {
            const ld q = t[i] * p1[i] - b[j - 1] * p0[i];
            p0[i] = p1[i];
            p1[i] = q;
        }
        ld s = 0;
        for (int i = 0; i < n; i++) s += p1[i] * p1[i];
        nrm[j] = s;
        b[j] = s / nrm[j - 1];
    }
    auto poly = [&](int d, ld z) {  // the monic polynomial of degree d
        ld a = 0, c = 1;
        for (int j = 1; j <= d; j++) {
            const ld q = z * c - (j > 1 ? b[j - 1] : 0.0L) * a;
            a = c;
            c = q;
        }
        return c;
    };
    std::vector<ld> r;
    for (int d = 1; d <= m; d++) {
        std::vector<ld> nx;
        for (int i = 0; i < d; i++) {
            ld lo = i == 0 ? -1.0L : r[i - 1], hi = i == d - 1 ? 1.0L : r[i];
            const bool up = poly(d, hi) > 0;
            for (int it = 0; it < 80; it++) {
                const ld mid = (lo + hi) / 2;
                if ((poly(d, mid) > 0) == up) hi = mid;
                else lo = mid;
            }
            nx.push_back((lo + hi) / 2);
        }
        r = nx;
    }
    for (int i = 0; i < m; i++) {
        ld a = 0, c = 1, s = 1.0L / nrm[0];
        for (int j = 1; j < m; j++) {
            const ld q = r[i] * c - (j > 1 ? b[j - 1] : 0.0L) * a;
            a = c;
            c = q;
            s += c * c / nrm[j];
        }
        x[i] = (r[i] + 1.0L) / 2.0L;
        w[i] = 1.0L / s / n;
    }
}

// Symmetric rules whose parameters are solved for the discrete moments; the
// start values are those of the continuous measure (n -> infinity).
// Triangles: orbits of 1 (centroid), 3 ((a, a) and images) and 6 points in
// barycentric (s, t). Squares, (x, y) in [-1, 1]^2: orbits of 4 on the axes
// (r, 0), 4 on the diagonals (r, r) and 8 (p, q).
struct SymRule {
    int nv, degree, o1, o2, o3;  // orbits: triangles 1 / 3 / 6 points, squares 4 (axes) / 4 (diagonals) / 8
    int min_n;                   // smallest n with positive weights and inner nodes
    // triangles: error (alpha theta)^(degree+1), (beta kappa)^(degree+1), the largest
    // over shapes and n; squares: alpha = factor on the moment bound's theta part
    double alpha, beta;
    double z[20];
    int fixed = -1;  // a parameter kept at its start value (one more unknown than invariants)
};
const SymRule kTri[5] = {
    {3, 5, 1, 2, 0, 4, 0.86, 0.164, {0.225, 0.470142064, 0.132394153, 0.101286507, 0.125939181}},
    {3, 6, 0, 2, 1, 5, 0.63, 0.111,
     {0.249286745, 0.116786276, 0.063089014, 0.050844906, 0.310352451, 0.636502499, 0.082851076}},
    {3, 8, 1, 3, 1, 6, 0.76, 0.097,
     {0.144315608, 0.459292588, 0.095091634, 0.170569308, 0.103217371, 0.050547228, 0.032458498, 0.008394777,
      0.263112830, 0.027230314}},
    {3, 10, 1, 2, 3, 7, 0.62, 0.077,
     {0.090817990, 0.485577633, 0.036725958, 0.109481575, 0.045321059, 0.307939839, 0.550352942, 0.072757917,
      0.246672561, 0.728323905, 0.028327243, 0.066803251, 0.923655934, 0.009421667}},
    {3, 12, 0, 5, 3, 8, 0.63, 0.068,
     {0.488217390, 0.025731066, 0.439724392, 0.043692545, 0.271210385, 0.062858224, 0.127576146, 0.034796113,
      0.021317350, 0.006166261, 0.275713270, 0.608943236, 0.040371558, 0.281325581, 0.695836087, 0.022356773,
      0.116251916, 0.858014034, 0.017316231}},
};
const SymRule kSquare[4] = {
    {4, 5, 1, 1, 0, 4, 2.6, 0, {0.683126086, 0.204079993, 0.881906473, 0.045920007}},
    {4, 7, 1, 2, 0, 5, 20., 0, {0.925807563, 0.060495214, 0.805971879, 0.059359933, 0.380549792, 0.130144854}},
    {4, 9, 1, 2, 1, 6, 10., 0,
     {0.488916289, 0.113536148, 0.690868012, 0.053547559, 0.939627180, 0.010685672, 0.918602638, 0.344865048,
      0.036115311}},
    {4, 11, 2, 3, 1, 7, 175., 0,
     {0.247539047, 0.035511857, 0.778945815, 0.060033938, 0.430728263, 0.064597081, 0.919085141, 0.011595508,
      0.723262697, 0.037763475, 0.430430969, 0.962181690, 0.020249070},
     4},
};
constexpr int kSymMax = 20;  // most parameters of a rule

typedef long double ld;

int sym_unknowns(const SymRule& r) {
    return r.nv == 3 ? r.o1 + 2 * r.o2 + 3 * r.o3 : 2 * (r.o1 + r.o2) + 3 * r.o3;
}

// Invariants of the shape's symmetry group up to `degree`: triangles, products of
// e2 = sum u^2 and e3 = u1 u2 u3 (u = barycentric - 1/3); squares, of x^2 + y^2
// and x^2 y^2. Returns their number (the rule's number of unknowns).
int sym_invariants(const SymRule& r, ld s, ld t, ld* out) {
    ld f[2];
    int step, k = 0;
    if (r.nv == 3) {
        const ld u = s - 1.0L / 3, v = t - 1.0L / 3, q = -u - v;
        f[0] = (u * u + v * v + q * q) * 1.5L;
        f[1] = u * v * q * 13.5L;
        step = 3;
    } else {
        f[0] = s * s + t * t;
        f[1] = 4 * s * s * t * t;
        step = 4;
    }
    for (int d = 0; d <= r.degree; d++)
        for (int c = 0; step * c <= d; c++)
            if ((d - step * c) % 2 == 0) {
                ld p = 1;
                for (int i = 0; i < c; i++) p *= f[1];
                for (int i = 0; i < (d - step * c) / 2; i++) p *= f[0];
                out[k++] = p;
            }
    return k;
}

// Points of the rule with parameters z: (s, t, w) triples; returns the count.
int sym_points(const SymRule& r, const ld* z, ld (*p)[3]) {
    int k = 0, c = 0;
    auto put = [&](ld s, ld t, ld w) {
        p[c][0] = s;
        p[c][1] = t;
        p[c++][2] = w;
    };
    if (r.nv == 3) {
        if (r.o1) put(1.0L / 3, 1.0L / 3, z[k++]);
        for (int o = 0; o < r.o2; o++, k += 2) {
            const ld a = z[k], b = 1 - 2 * a, w = z[k + 1];
            put(a, a, w);
            put(a, b, w);
            put(b, a, w);
        }
        for (int o = 0; o < r.o3; o++, k += 3) {
            const ld a = z[k], b = z[k + 1], g = 1 - a - b, w = z[k + 2];
            put(a, b, w);
            put(b, a, w);
            put(a, g, w);
            put(g, a, w);
            put(b, g, w);
            put(g, b, w);
        }
        return c;
    }
    for (int o = 0; o < r.o1 + r.o2; o++, k += 2) {
        const ld a = z[k], w = z[k + 1], b = o < r.o1 ? 0 : a;
        put(a, b, w);
        put(-a, -b, w);
        put(-b, a, w);
        put(b, -a, w);
    }
    for (int o = 0; o < r.o3; o++, k += 3)
        for (int f = 0; f < 8; f++) {
            const ld a = (f & 1) ? -z[k] : z[k], b = (f & 2) ? -z[k + 1] : z[k + 1];
            if (f & 4) put(b, a, z[k + 2]);
            else put(a, b, z[k + 2]);
        }
    return c;
}

// The rule matched to the n^2 midpoints of the n-split: Newton's method on the
// invariant moments. False when it does not converge to positive weights and
// inner nodes (the level is then left out).
bool sym_rule(const SymRule& r, int n, ld (*p)[3], int* count) {
    const int nz = sym_unknowns(r), nu = r.fixed < 0 ? nz : nz - 1;
    auto par = [&](int j) { return r.fixed >= 0 && j >= r.fixed ? j + 1 : j; };  // unknown -> parameter
    ld z[kSymMax], tgt[kSymMax] = {0}, inv[kSymMax], res[kSymMax], jac[kSymMax][kSymMax + 1];
    for (int i = 0; i < nz; i++) z[i] = r.z[i];
    for (int i = 0; i < n; i++)
        for (int j = 0; j < n; j++) {
            if (r.nv == 4) {
                sym_invariants(r, (2 * i + 1.0L) / n - 1, (2 * j + 1.0L) / n - 1, inv);
                for (int q = 0; q < nu; q++) tgt[q] += inv[q];
                continue;
            }
            for (int up = 0; up < 2; up++) {
                if (i + j + up >= n) continue;
                const ld o = up ? 2.0L / 3 : 1.0L / 3;
                sym_invariants(r, (i + o) / n, (j + o) / n, inv);
                for (int q = 0; q < nu; q++) tgt[q] += inv[q];
            }
        }
    for (int q = 0; q < nu; q++) tgt[q] /= (ld)n * n;
    auto moments = [&](const ld* zz, ld* out) {
        ld pts[kRuleMaxSym][3];
        const int c = sym_points(r, zz, pts);
        for (int q = 0; q < nu; q++) out[q] = 0;
        for (int i = 0; i < c; i++) {
            sym_invariants(r, pts[i][0], pts[i][1], inv);
            for (int q = 0; q < nu; q++) out[q] += inv[q] * pts[i][2];
        }
    };
    ld step = 1;
    for (int it = 0; it < 60 && step > 1e-14L; it++) {
        moments(z, res);
        for (int q = 0; q < nu; q++) jac[q][nu] = tgt[q] - res[q];
        for (int j = 0; j < nu; j++) {  // central differences: their error only slows the last steps
            ld& zj = z[par(j)];
            const ld h = 1e-7L, z0 = zj;
            ld a[kSymMax], b[kSymMax];
            zj = z0 + h;
            moments(z, a);
            zj = z0 - h;
            moments(z, b);
            zj = z0;
            for (int q = 0; q < nu; q++) jac[q][j] = (a[q] - b[q]) / (2 * h);
        }
        for (int c = 0; c < nu; c++) {  // Gauss elimination with row pivoting
            int pv = c;
            for (int q = c + 1; q < nu; q++)
                if (fabsl(jac[q][c]) > fabsl(jac[pv][c])) pv = q;
            if (!(fabsl(jac[pv][c]) > 0)) return false;
            for (int k = c; k <= nu; k++) std::swap(jac[c][k], jac[pv][k]);
            for (int q = 0; q < nu; q++)
                if (q != c) {
                    const ld f = jac[q][c] / jac[c][c];
                    for (int k = c; k <= nu; k++) jac[q][k] -= f * jac[c][k];
                }
        }
        step = 0;
        for (int q = 0; q < nu; q++) step = fmaxl(step, fabsl(jac[q][nu] / jac[q][q]));
        const ld damp = step > 0.05L ? 0.05L / step : 1.0L;
        for (int q = 0; q < nu; q++) z[par(q)] += damp * jac[q][nu] / jac[q][q];
    }
    // the last step was below 1e-14, so the next (quadratic but for the Jacobian's
    // difference quotient, 1e-11) would be below rounding
    moments(z, res);
    for (int q = 0; q < nu; q++)
        if (!(fabsl(res[q] - tgt[q]) < 1e-16L)) return false;
    *count = sym_points(r, z, p);
    for (int i = 0; i < *count; i++) {
        const ld s = p[i][0], t = p[i][1];
        const bool inside = r.nv == 3 ? s > 0 && t > 0 && s + t < 1 : fabsl(s) < 1 && fabsl(t) < 1;
        if (!(p[i][2] > 0) || !inside) return false;
    }
    return true;
}

// The levels of one (shape, n), shortest first: rules of at most 0.6 n^2 nodes
// (a longer one saves less than the table it displaces costs).
RuleHost make_rules(int nv, int n) {
    RuleHost h;
    if (n < 4) return h;
    const double tol[2] = {kRuleTol32, kRuleTol64};
    auto open = [&](int cnt) {
        if (h.n_lev == kMaxRules || cnt > 0.6 * n * n || h.total + cnt > kRuleMaxNodes) return false;
        h.cnt[h.n_lev] = cnt;
        h.off[h.n_lev] = h.total;
        h.factor[h.n_lev] = 1.6;
        return true;
    };
    // A node of the level opened last. The rounding of each weight goes into the next,
    // so that their sum is 1 to 1e-17: rounded on their own they left every cell up to
    // 1.4e-16 light or heavy, which does not average out over the cells.
    ld carry = 0;
    auto put = [&](int k, ld s, ld t, ld w) {
        const int q = h.total + k;
        if (k == 0) carry = 0;
        h.s[q] = (double)s;
        h.t[q] = (double)t;
        h.w[q] = (double)(w + carry);
        carry += w - (ld)h.w[q];
    };
    auto close = [&]() {
        h.total += h.cnt[h.n_lev];
        h.n_lev++;
    };
    ld p[kRuleMaxSym][3];
    int c;
    if (nv == 4) {
        // m > 0: the tensor rule of m^2 nodes; m < 0: kSquare[-m - 1]. The tensor rule of
        // 9 nodes stays exact on distorted cells, where the 8-node rule is not.
        const int order[11] = {-1, 3, -2, 4, -3, -4, 6, 7, 8, 10, 0};
        for (int i = 0; order[i]; i++) {
            const int m = order[i];
            if (n >= 16 && (m == 3 || m == 7)) continue;  // room for the long ones
            if (m > 0) {
                if (m >= n || !open(m * m)) continue;
                ld x[10], w[10];
                discrete_gauss(n, m, x, w);
                for (int a = 0; a < m; a++)
                    for (int b = 0; b < m; b++) put(a * m + b, x[a], x[b], w[a] * w[b]);
            } else {
                const SymRule& r = kSquare[-m - 1];
                if (n < r.min_n || !sym_rule(r, n, p, &c) || !open(c)) continue;
                h.factor[h.n_lev] = r.alpha;
                for (int k = 0; k < c; k++) put(k, (1 + p[k][0]) / 2, (1 + p[k][1]) / 2, p[k][2]);
            }
            // the compared moments end at degree 17: these limits keep the rest
            // of the series (and all of it for m = 10) below the tolerance
            h.tmax[h.n_lev][0] = 0.3;
            h.tmax[h.n_lev][1] = 0.2;
            h.kmax[h.n_lev][0] = 3.0;
            h.kmax[h.n_lev][1] = 2.0;
            close();
        }
        return h;
    }
    for (const SymRule& r : kTri) {
        if (n < r.min_n || !sym_rule(r, n, p, &c) || !open(c)) continue;
        for (int i = 0; i < c; i++) put(i, p[i][0], p[i][1], p[i][2]);
        for (int g = 0; g < 2; g++) {
            const double e = pow(tol[g], 1.0 / (r.degree + 1)) / 1.03;
            h.tmax[h.n_lev][g] = e / r.alpha;
            h.kmax[h.n_lev][g] = e / r.beta;
        }
        close();
    }
    if (n % 2 == 0 && n >= 16)
        for (int q = 2; q < 5; q++) {  // degrees 8, 10, 12 on the four halves
            if (!sym_rule(kTri[q], n / 2, p, &c) || !open(4 * c)) continue;
            for (int f = 0; f < 4; f++)
                for (int i = 0; i < c; i++) {
                    const ld s = p[i][0] / 2, t = p[i][1] / 2;
                    put(f * c + i, f == 3 ? 0.5L - s : s + (f == 1 ? 0.5L : 0.L),
                        f == 3 ? 0.5L - t : t + (f == 2 ? 0.5L : 0.L), p[i][2] / 4);
                }
            for (int g = 0; g < 2; g++) {
                // half the size, the nearest half up to rho / 2 nearer: alpha / 1.8, beta / 2 (measured:
                // 0.35 for degree 8)
                const double e = pow(tol[g], 1.0 / (kTri[q].degree + 1)) / 1.03;
                h.tmax[h.n_lev][g] = fmin(0.25, e / (0.56 * kTri[q].alpha));
                h.kmax[h.n_lev][g] = e / (0.56 * kTri[q].beta);
            }
            close();
        }
    return h;
}

// Rules depend on (shape, n) only: computed once per process for each split
// (n <= kRuleMaxN, so the cache is bounded).
constexpr int kRuleMaxN = 64;
const RuleHost& rules_for(int nv, int n) {
    static std::mutex mu;
    static std::map<std::pair<int, int>, RuleHost>* cache = new std::map<std::pair<int, int>, RuleHost>();
    static const RuleHost none = RuleHost();
    if (n > kRuleMaxN) return none;
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache->find({nv, n});
    if (it == cache->end()) it = cache->emplace(std::make_pair(nv, n), make_rules(nv, n)).first;
    return it->second;
}

}  // namespace

// Rule node k of a cell relative to its first vertex frame: y and the weight.
// Quads: (s, t) are the reference's (p, q) of quad_node; the Jacobian
// |y_p x y_q| is n^2 times the area of the sub-cell centred there.
BIELCC_D void rule_node(const double (*v)[3], int nv, double area, double s, double t, double w, double* y,
                        double* wt) {
    if (nv == 4) {
        double yp[3], yq[3], nr[3];
        for (int k = 0; k < 3; k++) {
            const double lo = t * v[1][k] + (1 - t) * v[0][k], hi = t * v[2][k] + (1 - t) * v[3][k];
            y[k] = s * hi + (1 - s) * lo;
            yp[k] = hi - lo;
            yq[k] = s * (v[2][k] - v[3][k]) + (1 - s) * (v[1][k] - v[0][k]);
        }
        cross3(yp, yq, nr);
        *wt = len3(nr) * w;
        return;
    }
    for (int k = 0; k < 3; k++) y[k] = v[0][k] + s * (v[1][k] - v[0][k]) + t * (v[2][k] - v[0][k]);
    *wt = area * w;
}

// One thread per (cell, rule node): FP64 (y, w) and FP32 (y - centre, w) rows.
__global__ void rule_nodes_kernel(const __grid_constant__ RuleHost h, const double* __restrict__ verts,
                                  const CellGeo* __restrict__ geo, int nv, int n_cells, double4* __restrict__ n64,
                                  float4* __restrict__ n32) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t c = i / h.total;
    if (c >= (size_t)n_cells) return;
    const int q = (int)(i - c * h.total);
    int l = 0;
    while (l + 1 < h.n_lev && q >= h.off[l + 1]) l++;
    double v[4][3];
    for (int a = 0; a < nv; a++)
        for (int g = 0; g < 3; g++) v[a][g] = verts[(c * nv + a) * 3 + g];
    double y[3], w;
    rule_node(v, nv, nv == 3 ? tri_area(v[0], v[1], v[2]) : 0., h.s[q], h.t[q], h.w[q], y, &w);
    const size_t o = (size_t)h.off[l] * n_cells + c * h.cnt[l] + (q - h.off[l]);
    const double* ctr = geo[c].c;
    if (n64) n64[o] = make_double4(y[0], y[1], y[2], w);
    if (n32) n32[o] = make_float4((float)(y[0] - ctr[0]), (float)(y[1] - ctr[1]), (float)(y[2] - ctr[2]), (float)w);
}

// FP32 weights of a row, rounded so that their sum is the FP64 sum's (the rounding
// of each goes into the next): 7 - 20 weights rounded on their own left a cell up to
// 2e-8 heavy, where the errors of 64 mostly cancel. One thread per (cell, level).
__global__ void rule_weights_kernel(const __grid_constant__ RuleHost h, const double* __restrict__ verts, int nv,
                                    int n_cells, float4* __restrict__ n32) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t c = i / h.n_lev;
    if (c >= (size_t)n_cells) return;
    const int l = (int)(i - c * h.n_lev);
    double v[4][3], y[3], w, carry = 0.;
    for (int a = 0; a < nv; a++)
        for (int g = 0; g < 3; g++) v[a][g] = verts[(c * nv + a) * 3 + g];
    const double area = nv == 3 ? tri_area(v[0], v[1], v[2]) : 0.;
    float4* row = n32 + (size_t)h.off[l] * n_cells + c * h.cnt[l];
    for (int q = 0; q < h.cnt[l]; q++) {
        const int k = h.off[l] + q;
        rule_node(v, nv, area, h.s[k], h.t[k], h.w[k], y, &w);
        w += carry;
        const float f = (float)w;
        row[q].w = f;
        carry = w - (double)f;
    }
}

// Triangles: the limits are the same for every cell up to its node radius. The node
// nearest a vertex is the centroid of a sub-triangle 1/n the size with that vertex.
__global__ void rule_limits_tri_kernel(const __grid_constant__ RuleHost h, const CellGeo* __restrict__ geo, int n_cells,
                                       int n, float2* __restrict__ thr) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_cells) return;
    const double r = geo[c].rho * (1.0 - 1.0 / n) * (1.0 + 1e-6);
    for (int g = 0; g < 2; g++)
        for (int l = 0; l < h.n_lev; l++)
            thr[((size_t)g * n_cells + c) * h.n_lev + l] =
                make_float2((float)(r / h.tmax[l][g] * (1.0 + 1e-5)), (float)(h.kmax[l][g] / r));
}

// Quads: one warp per cell. Lane = direction (16 in the cell's plane, 16 tilted
// by 45 degrees); each lane sums w (e . y / rho)^d, d < kRuleDeg, over the n^2
// nodes and over every rule's nodes, all relative to the centre so that the
// differences carry no cancellation from the cell's position. The largest
// difference over the lanes is D_d; the limits are then read off a grid of 32
// theta (kappa) values, one per lane, refined once.
__global__ void rule_limits_quad_kernel(const __grid_constant__ RuleHost h, const double* __restrict__ verts,
                                        const CellGeo* __restrict__ geo, int n_cells, int n,
                                        float2* __restrict__ thr) {
    const int c = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (c >= n_cells) return;  // whole warps
    const CellGeo& gg = geo[c];
    double v[4][3], e[3];
    for (int a = 0; a < 4; a++)
        for (int g = 0; g < 3; g++) v[a][g] = verts[((size_t)c * 4 + a) * 3 + g] - gg.c[g];
    {
        double sa, ca;
        sincospi((lane & 15) / 16.0, &sa, &ca);
        const double tilt = lane < 16 ? 0. : ((lane & 1) ? 1. : -1.);
        const double sc = lane < 16 ? 1. : 0.70710678118654752;
        for (int g = 0; g < 3; g++) e[g] = (ca * gg.t1[g] + sa * gg.t2[g] + tilt * gg.n[g]) * sc;
    }
    __shared__ double4 s_node[4][32];  // a chunk of nodes (y, weight), one per lane
    double4* buf = s_node[(threadIdx.x >> 5) & 3];
    const double inv_n = 1.0 / n;
    double rho = 0., y[3], w;
    for (int q = lane; q < n * n; q += 32) {
        rule_node(v, 4, 0., (q / n + 0.5) * inv_n, (q % n + 0.5) * inv_n, 1.0, y, &w);
        rho = fmax(rho, len3(y));
    }
    for (int o = 16; o > 0; o >>= 1) rho = fmax(rho, __shfl_xor_sync(0xffffffffu, rho, o));
    const double ir = 1.0 / rho;
    // Power sums of the n^2 nodes and of a rule's: the low degrees, whose differences
    // count most, with a running correction (Neumaier), the others plainly.
    constexpr int kComp = 4;
    double full[kRuleDeg], fc[kComp];
    auto clear = [&](double (&m)[kRuleDeg], double (&cc)[kComp]) {
#pragma unroll
        for (int d = 0; d < kRuleDeg; d++) m[d] = 0.;
#pragma unroll
        for (int d = 0; d < kComp; d++) cc[d] = 0.;
    };
    auto add = [&](double (&m)[kRuleDeg], double (&cc)[kComp], double wt, double t) {
#pragma unroll
        for (int d = 0; d < kRuleDeg; d++) {
            if (d < kComp) {
                const double sum = __dadd_rn(m[d], wt), b = __dsub_rn(sum, m[d]);
                cc[d] += __dadd_rn(__dsub_rn(m[d], __dsub_rn(sum, b)), __dsub_rn(wt, b));
                m[d] = sum;
            } else {
                m[d] += wt;
            }
            wt *= t;
        }
    };
    // Sums over `count` nodes: the lanes evaluate 32 of them side by side, then each
    // adds them all in its direction.
    auto sums = [&](double (&m)[kRuleDeg], double (&cc)[kComp], int count, auto node) {
        clear(m, cc);
        for (int q0 = 0; q0 < count; q0 += 32) {
            __syncwarp();
            if (q0 + lane < count) {
                node(q0 + lane);
                buf[lane] = make_double4(y[0], y[1], y[2], w);
            }
            __syncwarp();
            const int m32 = min(32, count - q0);
#pragma unroll 4
            for (int q = 0; q < m32; q++) {
                const double4 b = buf[q];
                add(m, cc, b.w, (b.x * e[0] + b.y * e[1] + b.z * e[2]) * ir);
            }
        }
    };
    sums(full, fc, n * n, [&](int q) {
        rule_node(v, 4, 0., (q / n + 0.5) * inv_n, (q % n + 0.5) * inv_n, inv_n * inv_n, y, &w);
    });
    const double tol[2] = {kRuleTol32, kRuleTol64};
    const double grid[2] = {pow(0.87, (double)lane), pow(0.84, (double)lane)};  // theta, kappa: times the limit
    for (int l = 0; l < h.n_lev; l++) {
        double dm[kRuleDeg], dc[kComp];
        sums(dm, dc, h.cnt[l], [&](int q) {
            q += h.off[l];
            rule_node(v, 4, 0., h.s[q], h.t[q], h.w[q], y, &w);
        });
#pragma unroll
        for (int d = 0; d < kRuleDeg; d++) {
            double x = dm[d] - full[d];
            if (d < kComp) x += dc[d] - fc[d];
            x = fabs(x) / full[0];
            // a NaN (a cell without area) must reach every lane: fmax would drop it
            for (int o = 16; o > 0; o >>= 1) {
                const double z = __shfl_xor_sync(0xffffffffu, x, o);
                x = (x >= z || x != x) ? x : z;
            }
            dm[d] = x - kRuleFloor > 0. || x != x ? x - kRuleFloor : 0.;
        }
        for (int g = 0; g < 2; g++) {
            auto theta_ok = [&](double th) {
                double s = 0., p = 1.;
#pragma unroll
                for (int d = 0; d < kRuleDeg; d++) {
                    s += 0.5 * (d + 1) * (d + 2) * p * dm[d];
                    p *= th;
                }
                return h.factor[l] * s <= tol[g];
            };
            auto kappa_ok = [&](double ka) {
                double s = 0., p = 1.;
#pragma unroll
                for (int d = 0; d < kRuleDeg; d++) {
                    s += p * dm[d];
                    p *= ka * (1.0 / (d + 1));
                }
                return 1.5 * s <= tol[g];
            };
            double lim[2];
            for (int which = 0; which < 2; which++) {
                const double top = which ? h.kmax[l][g] : h.tmax[l][g], ratio = which ? 0.84 : 0.87;
                const double a = top * grid[which];
                const unsigned m = __ballot_sync(0xffffffffu, which ? kappa_ok(a) : theta_ok(a));
                if (!m) {
                    lim[which] = -1.;
                    continue;
                }
                const int f = __ffs(m) - 1;
                lim[which] = top;
                if (f > 0) {  // between grid value f (kept) and f - 1 (not)
                    const double lo = __shfl_sync(0xffffffffu, a, f), hi = lo / ratio;
                    const double b = hi + (lo - hi) * (lane + 1) / 32.0;  // lane 31: lo
                    const unsigned m2 = __ballot_sync(0xffffffffu, which ? kappa_ok(b) : theta_ok(b));
                    lim[which] = m2 ? hi + (lo - hi) * __ffs(m2) / 32.0 : lo;
                }
            }
            if (lane == 0) {
                const bool ok = lim[0] > 0. && lim[1] > 0.;
                thr[((size_t)g * n_cells + c) * h.n_lev + l] =
                    ok ? make_float2((float)(rho / lim[0] * (1.0 + 1e-5)), (float)(lim[1] / rho))
                       : make_float2(__int_as_float(0x7f800000), -1.f);
            }
        }
    }
}

// Device bytes of h's levels with FP64 rows, FP32 rows or both, and their limits.
static size_t level_bytes(const RuleHost& h, int n_cells, bool f64, bool f32, bool limits) {
    return (size_t)n_cells * (h.total * ((f64 ? sizeof(double4) : 0) + (f32 ? sizeof(float4) : 0)) +
                              (limits ? 2 * h.n_lev * sizeof(float2) : 0));
}

size_t rules_bytes(int nv, int n, int n_cells, bool f64, bool f32, const FarRules& out) {
    f64 = f64 && !out.n64;
    f32 = f32 && !out.n32;
    return f64 || f32 ? level_bytes(rules_for(nv, n), n_cells, f64, f32, !out.n_lev) : 0;
}

// Builds the levels of h in `mem` ([FP64 rows][FP32 rows][limits]).
static cudaError_t build_levels(const RuleHost& h, const double* verts, const CellGeo* geo, int nv, int n_cells, int n,
                                bool f64, bool f32, void* mem, FarRules* out, cudaStream_t s) {
    const bool limits = !out->n_lev;
    double4* n64 = f64 ? (double4*)mem : nullptr;
    char* end = (char*)mem + (f64 ? (size_t)h.total * n_cells * sizeof(double4) : 0);
    float4* n32 = f32 ? (float4*)end : nullptr;
    float2* thr = (float2*)(end + (f32 ? (size_t)h.total * n_cells * sizeof(float4) : 0));
    const size_t nodes = (size_t)h.total * n_cells;
    rule_nodes_kernel<<<(unsigned)((nodes + 127) / 128), 128, 0, s>>>(h, verts, geo, nv, n_cells, n64, n32);
    if (f32)
        rule_weights_kernel<<<(unsigned)(((size_t)n_cells * h.n_lev + 127) / 128), 128, 0, s>>>(h, verts, nv, n_cells,
                                                                                                n32);
    if (limits) {
        if (nv == 4) rule_limits_quad_kernel<<<(n_cells + 3) / 4, 128, 0, s>>>(h, verts, geo, n_cells, n, thr);
        else rule_limits_tri_kernel<<<(n_cells + 127) / 128, 128, 0, s>>>(h, geo, n_cells, n, thr);
        out->n_lev = h.n_lev;
        for (int l = 0; l < h.n_lev; l++) {
            out->cnt[l] = h.cnt[l];
            out->off[l] = h.off[l];
        }
        out->thr32 = thr;
        out->thr64 = thr + (size_t)n_cells * h.n_lev;
    }
    if (f64) out->n64 = n64;
    if (f32) out->n32 = n32;
    return cudaGetLastError();
}

cudaError_t launch_rules(const double* verts, const CellGeo* geo, int nv, int n_cells, int n, bool f64, bool f32,
                         void* mem, FarRules* out, cudaStream_t s) {
    const RuleHost& h = rules_for(nv, n);
    f64 = f64 && !out->n64;
    f32 = f32 && !out->n32;
    if (!h.n_lev || n_cells <= 0 || !(f64 || f32)) return cudaSuccess;
    return build_levels(h, verts, geo, nv, n_cells, n, f64, f32, mem, out, s);
}

cudaError_t launch_rules_within(const double* verts, const CellGeo* geo, int nv, int n_cells, int n,
                                bool mixed, void* mem, size_t bytes, FarRules* out, cudaStream_t s) {
    *out = FarRules();
    RuleHost h = rules_for(nv, n);
    while (h.n_lev > 0 && level_bytes(h, n_cells, !mixed, mixed, true) > bytes) {
        h.n_lev--;
        h.total = h.off[h.n_lev];
    }
    if (!h.n_lev || n_cells <= 0) return cudaSuccess;
    return build_levels(h, verts, geo, nv, n_cells, n, !mixed, mixed, mem, out, s);
}

}  // namespace bielcc_gpu
