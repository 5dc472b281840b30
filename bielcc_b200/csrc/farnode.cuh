// farnode.cuh — the per-node far-field integrand shared by the far kernels
// (field.cu, batch.cu): F_RotRotSimplePot_H (kernel_lib.h:453-492) and
// F_GradSimplePot_H (kernel_lib.h:295-313) evaluated together at one
// quadrature node and accumulated as J-independent moments of one cell:
//   A1 = sum w e f1,  T = sum w e f2 d^ d^T (6),  G = sum w e (ikr - 1)/r^3 d (3)
// so that K_RotRot_Far = (A1 J + T J)/4pi and R_Rot_Colloc = (G x J)/4pi.
// FP64 and FP32 (phase split relative to the cell centre) forms.
//
// Real k: with alpha = 1/r^3 - i k/r^2 and u = k^2/r,
//   f1 = u - alpha, f2 = 3 alpha - u, (ikr - 1)/r^3 = -alpha.
// The node loop accumulates S = sum w e alpha in place of A1 and T/3 in place
// of T; since |d|^2 = r^2, tr T = 3 S - sum w e u, so A1 = 2 S - tr T, which
// finish_real_k recovers once per cell (two accumulators and the k^2/r
// product leave the per-node work).
#pragma once
#include "common.cuh"
#include "internal.h"

namespace bielcc_gpu {

// Near decision of get_field.h:58 with the reference's rounding: sqrt_rn(s) < t
// for the rounded sum of squares s of x - c and t = analytic_calc * diam. The
// rounded root is monotone, so this is s < T with T the smallest FP64 number
// whose rounded root reaches t: found once per staged cell from t^2 by a step or
// two up or down, it leaves one comparison per pair.
BIELCC_D double near_square(double t) {
    if (!(t > 0.)) return t != t ? t : 0.;  // no distance is below a t <= 0 (or NaN)
    double T = __dmul_rn(t, t);
    while (T > 0. && __dsqrt_rn(__longlong_as_double(__double_as_longlong(T) - 1)) >= t)
        T = __longlong_as_double(__double_as_longlong(T) - 1);
    while (__dsqrt_rn(T) < t) T = __longlong_as_double(__double_as_longlong(T) + 1);
    return T;
}
// cell row for near_exact: centre and T
BIELCC_D double4 near_cell(const CellGeo& g, double analytic_calc) {
    return make_double4(g.c[0], g.c[1], g.c[2], near_square(__dmul_rn(analytic_calc, g.diam)));
}
BIELCC_D bool near_exact(const double* x, const double4& cell, double (&d)[3], double* s) {
    d[0] = __dsub_rn(x[0], cell.x);
    d[1] = __dsub_rn(x[1], cell.y);
    d[2] = __dsub_rn(x[2], cell.z);
    *s = __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])), __dmul_rn(d[2], d[2]));
    return *s < cell.w;
}

// sqrt(s) in FP64 from the FP32 reciprocal root and one third-order step (about
// an ulp; EXACT: with a correction, half an ulp and a bit); outside the FP32
// range (and for NaN) the library root.
template <bool EXACT = true>
BIELCC_D double dist_from_sq(double s) {
    const float sf = (float)s;
    if (!(sf > 1e-30f && sf < 1e30f)) return sqrt(s);
    double y = (double)rsqrtf(sf);
    const double e = fma(-s * y, y, 1.0);
    y = fma(y * e, fma(e, 0.375, 0.5), y);
    const double d = s * y;
    return EXACT ? fma(fma(-d, d, s), 0.5 * y, d) : d;
}

// e^{i 2 pi t} for FP32 use, t in turns: the quarter turn is taken off in FP64
// (magic-number rounding; exact), sine and cosine of the rest, |a| <= pi / 4, from
// their Taylor series (truncation below 2e-9), in FP64, scaled by `amp`.
BIELCC_D void turn_f32(double t, double amp, float* c, float* s) {
    const double big = fma(t, 4.0, 6755399441055744.0);  // 1.5 2^52: rounds to an integer
    const int j = __double2loint(big);
    const double a = fma(-0.25, big - 6755399441055744.0, t) * 6.283185307179586477;
    const double q = a * a;
    const double ps = fma(fma(fma(fma(q, 1.0 / 362880, -1.0 / 5040), q, 1.0 / 120), q, -1.0 / 6), q, 1.0);
    const double pc =
        fma(fma(fma(fma(fma(q, -1.0 / 3628800, 1.0 / 40320), q, -1.0 / 720), q, 1.0 / 24), q, -0.5), q, 1.0);
    const float sf = (float)(a * ps * amp), cf = (float)(pc * amp);
    const float c0 = (j & 1) ? sf : cf, s0 = (j & 1) ? cf : sf;
    *c = ((j + 1) & 2) ? -c0 : c0;
    *s = (j & 2) ? -s0 : s0;
}
constexpr double kInvTwoPi = 0.15915494309189533577;

// The same decision from the root itself, which *d_out receives.
BIELCC_D bool is_near(const double* x, const double* c, double diam, double analytic_calc, double* d_out) {
    double d = dist3_rn(x, c);
    *d_out = d;
    return d < __dmul_rn(analytic_calc, diam);
}

// Rows of the far pass's quadrature (rules.cu): level l < n_lev is a compressed
// rule, level n_lev the full n^2-node table. The CTA keeps base and length of
// every level in shared memory.
template <typename NodeT>
struct RuleTab {
    const NodeT* base[kMaxRules + 1];
    int cnt[kMaxRules + 1];
    int n_lev;
    // one thread fills it; the caller synchronises
    BIELCC_D void fill(const FarRules& r, const NodeT* rows, const NodeT* full, int nn, int n_cells) {
        n_lev = r.n_lev;
        for (int l = 0; l < r.n_lev; l++) {
            base[l] = rows + (size_t)r.off[l] * n_cells;
            cnt[l] = r.cnt[l];
        }
        base[r.n_lev] = full;
        cnt[r.n_lev] = nn;
    }
};
BIELCC_D const float4* rule_rows(const FarRules& r, float4) { return r.n32; }
BIELCC_D const double4* rule_rows(const FarRules& r, double4) { return r.n64; }
BIELCC_D const float2* rule_limits(const FarRules& r, float4) { return r.thr32; }
BIELCC_D const float2* rule_limits(const FarRules& r, double4) { return r.thr64; }
// A node of a row in global memory (the same address for the whole warp).
BIELCC_D double4 ldg_node(const double4* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldg(q), b = __ldg(q + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}
// |k| and |Im k| as the limits take them, and a limit's smallest distance at that k.
// A limit holds theta = rho / r0 and kappa = |k| rho each at its own largest value.
// For real k both may be at it. Growth or decay adds the mixed terms of the product
// of the two series (rules.cu), which the sum of the two fractions bounds: theta /
// theta_max + |Im k| / kmax <= 1.
struct RuleK {
    float abs, im;
};
BIELCC_D RuleK rule_k(cplx k) {
    return {(float)(sqrt(cabs2(k)) * (1.0 + 1e-6)), (float)(fabs(k.im) * (1.0 + 1e-6))};
}
BIELCC_D float rule_rmin_real(float2 lim, RuleK k) { return k.abs <= lim.y ? lim.x : __int_as_float(0x7f800000); }
BIELCC_D float rule_rmin(float2 lim, RuleK k) {
    const float r = rule_rmin_real(lim, k);
    return k.im > 0.f ? r / fmaxf(1.f - k.im / lim.y, 0.f) : r;
}

// Smallest of the warp's values (all >= 0): every lane calls.
BIELCC_D float warp_min_pos(float v) { return __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(v))); }
// A lane's distance as that minimum takes it: infinity for a lane that does not
// take part; finite otherwise (a NaN or infinite distance takes part, so that it
// reaches the result: 0 asks for the full row).
BIELCC_D float rule_key(bool far, double d) {
    return far ? fminf(fmaxf((float)d, 0.f), 3e38f) : __int_as_float(0x7f800000);
}
// Shortest row usable from distance r (a warp's smallest, so the level is
// uniform over the warp): the first l < n_lev with r >= rmin[l], else the whole
// table (n_lev). A longer level need not reach nearer: on distorted cells the
// total-degree rules' limits fall behind those of shorter tensor rules, and a
// level that a cell cannot use at all has rmin = infinity.
BIELCC_D int rule_level(const float* rmin, int n_lev, float r) {
    int l = 0;
    while (l < n_lev && !(r >= rmin[l])) l++;
    return l;
}
// The same for two cells that take rows of one level: the first that both allow
// (a level that only one of them allows may be one that the other cannot use).
// An infinite distance (no lane far from that cell) allows every level.
BIELCC_D int rule_level2(const float* rmin_a, float ra, const float* rmin_b, float rb, int n_lev) {
    int l = 0;
    while (l < n_lev && !(ra >= rmin_a[l] && rb >= rmin_b[l])) l++;
    return l;
}

// Per-thread moment accumulators of one cell.
template <typename F>
struct Moments {
    F a1r, a1i;
    F t[6][2];  // xx, xy, xz, yy, yz, zz
    F g[3][2];
    static constexpr bool kNegG = sizeof(F) == 4;  // far_node_f32's real-k loop leaves -G
    BIELCC_D void zero() {
        a1r = a1i = 0;
        for (int i = 0; i < 6; i++) t[i][0] = t[i][1] = 0;
        for (int i = 0; i < 3; i++) g[i][0] = g[i][1] = 0;
    }
    BIELCC_D void finish_real_k();
};

// Real-k node loops leave (S, T/3) in (a1, t): turn them into (A1, T).
template <typename F>
BIELCC_D void finish_real_k(F& a1r, F& a1i, F (&t)[6][2]) {
    const F trr = t[0][0] + t[3][0] + t[5][0], tri = t[0][1] + t[3][1] + t[5][1];
    a1r = F(2) * a1r - F(3) * trr;
    a1i = F(2) * a1i - F(3) * tri;
#pragma unroll
    for (int q = 0; q < 6; q++) {
        t[q][0] *= F(3);
        t[q][1] *= F(3);
    }
}

template <typename F>
BIELCC_D void Moments<F>::finish_real_k() {
    bielcc_gpu::finish_real_k<F>(a1r, a1i, t);
    if (kNegG) {
#pragma unroll
        for (int q = 0; q < 3; q++) {
            g[q][0] = -g[q][0];
            g[q][1] = -g[q][1];
        }
    }
}

// FP32 wavenumber constants of one launch (or one job).
struct KF32 {
    float kr, ki;    // k
    float k2r, k2i;  // k^2
    float ikr;       // 1 / Re k, 1e30 for Re k = 0 (phase k (r - r0) = q / ((r + r0) ikr) then rounds to 0)
    float k2r3;      // -Re k^2 / 3
    static BIELCC_D KF32 make(double kre, double kim) {
        KF32 f;
        const double k2r = kre * kre - kim * kim;
        f.kr = (float)kre;
        f.ki = (float)kim;
        f.k2r = (float)k2r;
        f.k2i = (float)(2.0 * kre * kim);
        f.ikr = kre != 0.0 ? (float)(1.0 / kre) : 1e30f;
        f.k2r3 = (float)(-k2r / 3.0);
        return f;
    }
};

// Largest |Re k| |r - r0| and |Im k| |r - r0| over a cell of radius rho.
BIELCC_D double phase_range64(cplx k, double rho) { return fmax(fabs(k.re), fabs(k.im)) * rho * (1.0 + 1e-6); }

// One far node, FP64. dx = x - y; w = node weight. Real k (CK = false) or
// complex k. F_RotRotSimplePot_H (kernel_lib.h:453-492) and
// F_GradSimplePot_H (kernel_lib.h:295-313) share r, 1/r and e^{ikr}.
// SPLIT: the phase is taken relative to r0 = |x - centre| (the moments are
// multiplied by e^{ik r0} once per cell) and e^{ik (r - r0)} comes from the
// Taylor series, where |Re k| rho and |Im k| rho stay below 1/2 (phase_range64);
// otherwise e^{ikr} from sincos (and exp) per node. Complex k,
// 3200 quads x 2000 points, mixed call with its FP64 error sample: 0.77 ms with sincos
// and exp per node, 0.74 so.
template <bool CK, bool SPLIT, int TD = 0>
BIELCC_D void far_node_f64(Moments<double>& m, double dx, double dy, double dz, double w, cplx k, double k2r,
                           double k2i, double r0) {
    double r2 = dx * dx + dy * dy + dz * dz;
    double ir = rsqrt(r2);
    double r = r2 * ir;
    double s, c;
    if (SPLIT) {
        const double dr = r - r0;
        sincos_taylor64<TD>(k.re * dr, &s, &c);
        if (CK) {
            const double a = exp_taylor64<TD>(-k.im * dr);
            s *= a;
            c *= a;
        }
    } else {
        sincos(k.re * r, &s, &c);
        if (CK) {
            double a = exp(-k.im * r);
            s *= a;
            c *= a;
        }
    }
    double ir2 = ir * ir, ir3 = ir2 * ir;
    double er = w * c, ei = w * s;
    if (!CK) {
        // real k: S += e alpha, T/3 += e (alpha - u/3)/r^2 d d^T, G -= e alpha d
        const double beta = k.re * ir2;
        const double ear = fma(ei, beta, er * ir3), eai = fma(-er, beta, ei * ir3);
        if (r >= kMachineZero) {  // F_RotRotSimplePot_H is 0 below MACHINE_ZERO
            m.a1r += ear;
            m.a1i += eai;
            const double u3 = k2r * (1.0 / 3.0) * ir3;
            const double a2r = fma(ear, ir2, -er * u3), a2i = fma(eai, ir2, -ei * u3);
            const double dd[6] = {dx * dx, dx * dy, dx * dz, dy * dy, dy * dz, dz * dz};
#pragma unroll
            for (int q = 0; q < 6; q++) {
                m.t[q][0] += a2r * dd[q];
                m.t[q][1] += a2i * dd[q];
            }
        }
        m.g[0][0] -= ear * dx;
        m.g[0][1] -= eai * dx;
        m.g[1][0] -= ear * dy;
        m.g[1][1] -= eai * dy;
        m.g[2][0] -= ear * dz;
        m.g[2][1] -= eai * dz;
        return;
    }
    if (r >= kMachineZero) {  // F_RotRotSimplePot_H is 0 below MACHINE_ZERO
        double f1r, f1i, f2r, f2i;
        if (CK) {
            f1r = k2r * ir - ir3 - k.im * ir2;
            f1i = k.re * ir2 + k2i * ir;
            f2r = 3.0 * ir3 + 3.0 * k.im * ir2 - k2r * ir;
            f2i = -3.0 * k.re * ir2 - k2i * ir;
        } else {
            f1r = k2r * ir - ir3;
            f1i = k.re * ir2;
            f2r = 3.0 * ir3 - k2r * ir;
            f2i = -3.0 * k.re * ir2;
        }
        m.a1r += er * f1r - ei * f1i;
        m.a1i += er * f1i + ei * f1r;
        double a2r = (er * f2r - ei * f2i) * ir2, a2i = (er * f2i + ei * f2r) * ir2;
        double dd[6] = {dx * dx, dx * dy, dx * dz, dy * dy, dy * dz, dz * dz};
#pragma unroll
        for (int q = 0; q < 6; q++) {
            m.t[q][0] += a2r * dd[q];
            m.t[q][1] += a2i * dd[q];
        }
    }
    // (ikr - 1) with ikr = (-k.im r, k.re r)
    double ur = CK ? (-k.im * r - 1.0) : -1.0, ui = k.re * r;
    double gr = (er * ur - ei * ui) * ir3, gi = (er * ui + ei * ur) * ir3;
    m.g[0][0] += gr * dx;
    m.g[0][1] += gi * dx;
    m.g[1][0] += gr * dy;
    m.g[1][1] += gi * dy;
    m.g[2][0] += gr * dz;
    m.g[2][1] += gi * dz;
}

// Taylor sine / cosine on |t| <= 1 (truncation below 2.6e-8), FP32.
BIELCC_D void sincos_poly(float t, float* s, float* c) {
    float t2 = t * t;
    float ps = fmaf(t2, 2.7557319e-6f, -1.9841270e-4f);
    ps = fmaf(t2, ps, 8.3333333e-3f);
    ps = fmaf(t2, ps, -1.6666667e-1f);
    ps = fmaf(t2, ps, 1.0f);
    *s = t * ps;
    float pc = fmaf(t2, -2.7557319e-7f, 2.4801587e-5f);
    pc = fmaf(t2, pc, -1.3888889e-3f);
    pc = fmaf(t2, pc, 4.1666667e-2f);
    pc = fmaf(t2, pc, -0.5f);
    *c = fmaf(t2, pc, 1.0f);
}

// Short Taylor sine / cosine for |t| <= 0.25 (truncation below 1.3e-8).
BIELCC_D void sincos_short(float t, float* s, float* c) {
    float t2 = t * t;
    float ps = fmaf(t2, 8.3333333e-3f, -1.6666667e-1f);
    *s = t * fmaf(t2, ps, 1.0f);
    float pc = fmaf(t2, -1.3888889e-3f, 4.1666667e-2f);
    pc = fmaf(t2, pc, -0.5f);
    *c = fmaf(t2, pc, 1.0f);
}

// e^{i theta} for a per-cell bound on |theta| (uniform over the CTA, so the
// mode is a template argument of the node loop): 0 -> |theta| <= 0.25 short
// polynomial; 1 -> <= 1; 2 -> <= 2 (half angle, one doubling); 3 -> <= 4 (two
// doublings); 4 -> accurate sincosf.
template <int MODE>
BIELCC_D void phase_f32(float th, float* s, float* c) {
    if constexpr (MODE == 0) {
        sincos_short(th, s, c);
    } else if constexpr (MODE == 4) {
        sincosf(th, s, c);
    } else {
        constexpr int H = MODE - 1;
        float ss, cc;
        sincos_poly(th * (H == 0 ? 1.f : (H == 1 ? 0.5f : 0.25f)), &ss, &cc);
#pragma unroll
        for (int h = 0; h < H; h++) {
            float ns = 2.f * ss * cc;
            cc = fmaf(cc, cc, -ss * ss);
            ss = ns;
        }
        *s = ss;
        *c = cc;
    }
}

BIELCC_HD int phase_mode(float th) {
    return th <= 0.25f ? 0 : (th <= 1.f ? 1 : (th <= 2.f ? 2 : (th <= 4.f ? 3 : 4)));
}

// A row's chunk of staged nodes, one of every warp's buffers. FP32 nodes are held
// as the packed arithmetic of far_node_f32 reads them: negated and doubled
// (-x, -x, -y, -y), (-z, -z, w, |y - centre|^2), |.|^2 computed once per node.
constexpr int kRowChunk = 32;
struct NodeF32 {
    float4 a, b;
};
BIELCC_D NodeF32 node_f32(float4 n) {  // n = (y - centre, w)
    return {make_float4(-n.x, -n.x, -n.y, -n.y),
            make_float4(-n.z, -n.z, n.w, fmaf(n.x, n.x, fmaf(n.y, n.y, n.z * n.z)))};
}
template <typename NodeT>
struct RowBuf {
    NodeT nd[kRowChunk];
    BIELCC_D void put(int i, const NodeT& v) { nd[i] = v; }
    BIELCC_D NodeT get(int i) const { return nd[i]; }
};
template <>
struct RowBuf<float4> {
    float4 a[kRowChunk], b[kRowChunk];
    BIELCC_D void put(int i, float4 v) {
        const NodeF32 n = node_f32(v);
        a[i] = n.a;
        b[i] = n.b;
    }
    BIELCC_D NodeF32 get(int i) const { return {a[i], b[i]}; }
};

// Per-pair FP32 state of the mixed far node, relative to the cell centre:
// X = x - centre (each component twice), X2 = 2 X, r0 = |X| (FP64 rounded), r0sq = r0^2, r0k = r0 / Re k.
struct PairF32 {
    float2 X[3];
    float X2[3], r0, r0sq, r0k;
    // from x - centre (FP64), |x - centre|^2 and |x - centre|
    BIELCC_D void set(const double (&dx)[3], double s, double d, const KF32& kf) {
#pragma unroll
        for (int g = 0; g < 3; g++) {
            const float v = (float)dx[g];
            X[g] = make_float2(v, v);
            X2[g] = v + v;
        }
        r0 = (float)d;
        r0sq = (float)s;
        r0k = r0 * kf.ikr;
    }
};

// a / b by the approximate reciprocal alone (b positive and normal here, so the
// scaling that __fdividef adds for large divisors is not needed).
BIELCC_D float fast_div(float a, float b) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    return a * r;
}

// Two FP32 values at a time (add, mul and fma .f32x2: one issue slot each).
BIELCC_D float2 dup2(float v) { return make_float2(v, v); }

// Shared head of the FP32 far node: n = the node, yy = |y - centre|^2.
// q = |x - y|^2 - r0^2 = yy - 2 (y - centre).X carries no cancellation.
// Returns 1/r and sets r, the weighted phase factor e = w e^{ik(r - r0)} and the
// components of d = x - y, each twice.
template <bool CK, int MODE>
BIELCC_D float far_head_f32(const PairF32& p, const NodeF32& n, const KF32& kf, float& r_out, float2& e, float2& dx,
                            float2& dy, float2& dz) {
    const float q = fmaf(n.a.x, p.X2[0], fmaf(n.a.z, p.X2[1], fmaf(n.b.x, p.X2[2], n.b.w)));
    const float r2 = p.r0sq + q;
    const float ir = rsqrtf(r2);
    const float r = r2 * ir;
    float s, c, w = n.b.z;
    if (CK) {
        const float dr = fast_div(q, r + p.r0);  // r - r0 without cancellation
        phase_f32<MODE>(kf.kr * dr, &s, &c);
        w *= __expf(-kf.ki * dr);
    } else {
        phase_f32<MODE>(fast_div(q, fmaf(r, kf.ikr, p.r0k)), &s, &c);  // k (r - r0)
    }
    dx = __fadd2_rn(p.X[0], make_float2(n.a.x, n.a.y));
    dy = __fadd2_rn(p.X[1], make_float2(n.a.z, n.a.w));
    dz = __fadd2_rn(p.X[2], make_float2(n.b.x, n.b.y));
    e = make_float2(w * c, w * s);
    r_out = r;
    return ir;
}

// acc += v * w, acc an (re, im) pair of the moments.
BIELCC_D void fma_into(float (&acc)[2], float2 v, float2 w) {
    const float2 o = __ffma2_rn(v, w, make_float2(acc[0], acc[1]));
    acc[0] = o.x;
    acc[1] = o.y;
}

// T += b d^T over the 6 symmetric entries, b = a2 d (complex a2).
BIELCC_D void acc_sym6(float (&t)[6][2], float2 a2, float2 dx, float2 dy, float2 dz) {
    const float2 bx = __fmul2_rn(a2, dx), by = __fmul2_rn(a2, dy), bz = __fmul2_rn(a2, dz);
    fma_into(t[0], bx, dx);
    fma_into(t[1], bx, dy);
    fma_into(t[2], bx, dz);
    fma_into(t[3], by, dy);
    fma_into(t[4], by, dz);
    fma_into(t[5], bz, dz);
}

// One far node, FP32 (E and H moments; GRAD false: the K moments alone, for the
// collocation matrix). Real k leaves (S, T/3, -G) in (a1, t, g): the caller runs
// finish_real_k once the cell's nodes are summed. Re and im parts go through the
// packed forms, each with the roundings of the scalar one (64 + 2 instructions per
// real-k node in scalar form, about 48 so; the pipe time is the same, but the far
// kernels are bound by issue slots). Field of 8192 cells x 20,000 points 7.08 ->
// 6.82 ms, 6.55 with 128 registers.
template <bool CK, int MODE, bool GRAD = true>
BIELCC_D void far_node_f32(Moments<float>& m, const PairF32& p, const NodeF32& n, const KF32& kf) {
    float r;
    float2 e, dx, dy, dz;
    const float ir = far_head_f32<CK, MODE>(p, n, kf, r, e, dx, dy, dz);
    const float ir2 = ir * ir, ir3 = ir2 * ir;
    if (!CK) {
        const float beta = kf.kr * ir2;
        const float2 ea = make_float2(fmaf(e.y, beta, e.x * ir3), fmaf(-e.x, beta, e.y * ir3));  // e alpha
        const float2 S = __fadd2_rn(make_float2(m.a1r, m.a1i), ea);
        m.a1r = S.x;
        m.a1i = S.y;
        const float u3 = kf.k2r3 * ir3;  // -k^2 / (3 r^3)
        // e (alpha - u/3) / r^2
        acc_sym6(m.t, __ffma2_rn(ea, dup2(ir2), __fmul2_rn(e, dup2(u3))), dx, dy, dz);
        if (GRAD) {
            fma_into(m.g[0], ea, dx);
            fma_into(m.g[1], ea, dy);
            fma_into(m.g[2], ea, dz);
        }
        return;
    }
    const float f1r = kf.k2r * ir - ir3 - kf.ki * ir2;
    const float f1i = kf.kr * ir2 + kf.k2i * ir;
    const float f2r = 3.f * ir3 + 3.f * kf.ki * ir2 - kf.k2r * ir;
    const float f2i = -3.f * kf.kr * ir2 - kf.k2i * ir;
    m.a1r = fmaf(e.x, f1r, fmaf(-e.y, f1i, m.a1r));
    m.a1i = fmaf(e.x, f1i, fmaf(e.y, f1r, m.a1i));
    acc_sym6(m.t, make_float2((e.x * f2r - e.y * f2i) * ir2, (e.x * f2i + e.y * f2r) * ir2), dx, dy, dz);
    if (GRAD) {
        const float ur = -kf.ki * r - 1.f, ui = kf.kr * r;
        const float2 gg = make_float2((e.x * ur - e.y * ui) * ir3, (e.x * ui + e.y * ur) * ir3);
        fma_into(m.g[0], gg, dx);
        fma_into(m.g[1], gg, dy);
        fma_into(m.g[2], gg, dz);
    }
}

}  // namespace bielcc_gpu
