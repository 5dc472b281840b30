// assemble.cu — collocation-matrix assembly of the K operator:
//   A[(i,a),(j,b)] = tau_a(i) . K[cell_j, tau_b(j)](c_i),  c_i = centre of cell i
// (layout TAU2, 2N x 2N) or the full 3x3 blocks (layout FULL3, 3N x 3N).
// K is linear in the cell current, so each (i, j) block is the 3x3 operator
// matrix projected on the tangent bases (CellFill, mesh/cell.cpp).
//   far  (|c_i - c_j| >= analytic_calc * diam_j): K_RotRot_Far (K.h:288-301)
//        = (A1 I + T) / 4pi from the precomputed node tables; FP64 or FP32
//        (phase split as in field.cu);
//   near: K_RotRot_HS_Colloc (K.h:179-204) in FP64 = I_hs k^2/4pi I + M / 4pi,
//        I_hs = IntegralSurf_SimplePot_H_HS (integrals_analytic.h:136-164),
//        M = -sum_e ks_e nu_e^T from the unsmoothed K0 (K0.h:36-86).
// Every entry is written exactly once (far kernel skips near pairs).
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "farnode.cuh"
#include "grid.h"
#include "internal.h"
#include "ops.cuh"
#include "scan.cuh"

namespace bielcc_gpu {

constexpr int kAsmThreads = 128;
constexpr int kAsmStageCells = 32;  // column cells staged at a time: one mask word
constexpr int kAsmWays = 4;         // warps that share the columns on small matrices
constexpr size_t kAsmOutBytes = (size_t)(kAsmThreads / 32) * 2 * 32 * 8 * 16;  // staged blocks of a CTA (32 KB)

struct AsmArgs {
    const CellGeo* geo;
    int n_cells;
    const double4* nodes64;
    const float4* nodes32;
    const float* rho32;
    int nn;
    FarRules rules;
    cplx k;
    double analytic_calc;
    int cols_per_split;
    int ways;  // 1, or kAsmWays: the CTA's warps share the columns, 32 rows per CTA
    int m;  // 2 (tau) or 3 (full)
    int c64;
    void* A;
    unsigned* mask;  // [ceil(N/32)][N] near bits of (row i, column word) written by the far kernel, or null
};

// p_max >= 3, the far kernel's marks-reading variant: mark[b] [ceil(N/32)][N]
// is set for the (row, column) blocks whose column-b integral failed the
// convergence test at the second pass; take_marked 0 writes the columns that
// passed, 1 the ones that failed. (A separate type, so that the plain
// variants keep AsmArgs' parameter block.)
struct AsmArgsMarks : AsmArgs {
    const unsigned* mark;
    int take_marked;
};
template <bool MARKS>
using AsmArgsOf = typename std::conditional<MARKS, AsmArgsMarks, AsmArgs>::type;

BIELCC_D bool asm_is_near(const double* x, const CellGeo& g, double analytic_calc, double* d) {
    *d = dist3_rn(x, g.c);
    return *d < __dmul_rn(analytic_calc, g.diam);
}

// The M x M block of (row cell i, column cell j) from the 3x3 complex operator
// matrix K (already / 4pi): M = 2 projects on tau1, tau2 of both cells, M = 3 keeps
// the Cartesian block. M is a template argument so that the block stays in registers.
template <int M>
BIELCC_D void block_f64(const double (&Kr)[3][3], const double (&Ki)[3][3], const double* ti1, const double* ti2,
                        const double* tj1, const double* tj2, double (&o)[M][M][2]) {
#pragma unroll
    for (int aa = 0; aa < M; aa++) {
#pragma unroll
        for (int b = 0; b < M; b++) {
            double vr = 0., vi = 0.;
            if constexpr (M == 3) {
                vr = Kr[aa][b];
                vi = Ki[aa][b];
            } else {
                const double* ta = aa == 0 ? ti1 : ti2;
                const double* tb = b == 0 ? tj1 : tj2;
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    double kr = Kr[p][0] * tb[0] + Kr[p][1] * tb[1] + Kr[p][2] * tb[2];
                    double ki = Ki[p][0] * tb[0] + Ki[p][1] * tb[1] + Ki[p][2] * tb[2];
                    vr += ta[p] * kr;
                    vi += ta[p] * ki;
                }
            }
            o[aa][b][0] = vr;
            o[aa][b][1] = vi;
        }
    }
}

// Writes a block; cols: bit b writes column b (the convergence-test passes of
// p_max >= 3; all otherwise).
template <int M, typename F>
BIELCC_D void store_block(const AsmArgs& a, int i, int j, const F (&o)[M][M][2], unsigned cols) {
    const size_t dim = (size_t)M * a.n_cells;
#pragma unroll
    for (int aa = 0; aa < M; aa++) {
        const size_t off = ((size_t)i * M + aa) * dim + (size_t)j * M;
        if (a.c64) {
            float2* dst = reinterpret_cast<float2*>(a.A) + off;
#pragma unroll
            for (int b = 0; b < M; b++)
                if ((cols >> b) & 1u) dst[b] = make_float2((float)o[aa][b][0], (float)o[aa][b][1]);
        } else {
            double2* dst = reinterpret_cast<double2*>(a.A) + off;
#pragma unroll
            for (int b = 0; b < M; b++)
                if ((cols >> b) & 1u) dst[b] = make_double2(o[aa][b][0], o[aa][b][1]);
        }
    }
}

template <int M>
BIELCC_D void write_block_m(const AsmArgs& a, int i, int j, const double (&Kr)[3][3], const double (&Ki)[3][3],
                            const double* ti1, const double* ti2, const double* tj1, const double* tj2,
                            unsigned cols = ~0u) {
    double o[M][M][2];
    block_f64<M>(Kr, Ki, ti1, ti2, tj1, tj2, o);
    store_block<M, double>(a, i, j, o, cols);
}

// The mixed form's far block, in FP32 (the moments are FP32 sums already):
// K = A1 I + T with T symmetric (xx, xy, xz, yy, yz, zz), projected on the two
// cells' tangents (M = 2: u_b = K t_b, A_ab = t_a . u_b) or kept Cartesian
// (M = 3), times ph = e^{ik r0} / 4pi.
template <int M>
BIELCC_D void block_f32(float a1r, float a1i, const float (&t)[6][2], float phr, float phi, const float (&ti)[2][3],
                        const float* tj1, const float* tj2, float (&out)[M][M][2]) {
    const int sym[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    float kr[6], ki[6];
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const bool diag = q == 0 || q == 3 || q == 5;
        kr[q] = diag ? t[q][0] + a1r : t[q][0];
        ki[q] = diag ? t[q][1] + a1i : t[q][1];
    }
    if constexpr (M == 3) {
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int q = 0; q < 3; q++) {
                out[p][q][0] = kr[sym[p][q]] * phr - ki[sym[p][q]] * phi;
                out[p][q][1] = kr[sym[p][q]] * phi + ki[sym[p][q]] * phr;
            }
    } else {
        const float tb[2][3] = {{tj1[0], tj1[1], tj1[2]}, {tj2[0], tj2[1], tj2[2]}};
#pragma unroll
        for (int b = 0; b < 2; b++) {
            float ur[3], ui[3];
#pragma unroll
            for (int p = 0; p < 3; p++) {
                ur[p] = kr[sym[p][0]] * tb[b][0] + kr[sym[p][1]] * tb[b][1] + kr[sym[p][2]] * tb[b][2];
                ui[p] = ki[sym[p][0]] * tb[b][0] + ki[sym[p][1]] * tb[b][1] + ki[sym[p][2]] * tb[b][2];
            }
#pragma unroll
            for (int aa = 0; aa < 2; aa++) {
                const float vr = ti[aa][0] * ur[0] + ti[aa][1] * ur[1] + ti[aa][2] * ur[2];
                const float vi = ti[aa][0] * ui[0] + ti[aa][1] * ui[1] + ti[aa][2] * ui[2];
                out[aa][b][0] = vr * phr - vi * phi;
                out[aa][b][1] = vr * phi + vi * phr;
            }
        }
    }
}

template <int M>
BIELCC_D void write_block_f32(const AsmArgs& a, int i, int j, float a1r, float a1i, const float (&t)[6][2], float phr,
                              float phi, const float (&ti)[2][3], const float* tj1, const float* tj2,
                              unsigned cols = ~0u) {
    float out[M][M][2];
    block_f32<M>(a1r, a1i, t, phr, phi, ti, tj1, tj2, out);
    store_block<M, float>(a, i, j, out, cols);
}

BIELCC_D void write_block(const AsmArgs& a, int i, int j, const double (&Kr)[3][3], const double (&Ki)[3][3],
                          const double* ti1, const double* ti2, const double* tj1, const double* tj2,
                          unsigned cols = ~0u) {
    if (a.m == 2) write_block_m<2>(a, i, j, Kr, Ki, ti1, ti2, tj1, tj2, cols);
    else write_block_m<3>(a, i, j, Kr, Ki, ti1, ti2, tj1, tj2, cols);
}

// Minimum resident CTAs per SM asked of the real-k mixed far kernel (0: the
// compiler's own register choice, which the other variants keep). 5 gives 96
// registers without spills (20,480 triangles 20.0 ms; 4: 20.1; 6: 20.6).
#ifndef BIELCC_ASM_MINB
#define BIELCC_ASM_MINB 5
#endif
// A warp (32 rows, one per lane) takes each column cell's row of nodes from the
// shortest rule that its nearest far row cell allows (rules.cu), staged as in
// far_kernel. ways = 1: 128 rows per CTA, every warp all columns; ways = 4, for
// matrices too small to fill the GPU: 32 rows, each warp every fourth column.
// STAGE (TAU2, ways = 1): a lane's 2 x 2 block is 16 bytes (complex64) of two
// matrix rows, so writing it directly touches 64 lines per warp and cell for
// half a sector each. Blocks go to shared memory instead (row chunks of 128 bytes,
// rotated by the lane so that neither side conflicts) and are written eight
// (complex128: four) columns at a time in whole lines; near blocks are written
// too (as zeros) and overwritten by asm_near_kernel, which always follows.
// 20,480 triangles, mixed, complex64, whole call: 65.6 ms with all 64 nodes and
// direct writes, 28.2 with the rules, 20.0 with rows staged per warp and whole-line
// writes (this kernel 16 of it: node loops 8, the pairs' set-up and projection 6,
// writes 1; bound by issue slots, 72 % active; 13.4 GB written). Now 18.7 with the
// near blocks' short forms.
// ways = 4: 80 triangles, FP64, 0.70 -> 0.28 ms.
template <bool CK, bool MIXED, bool MARKS = false, bool STAGE = false>
__global__ void __launch_bounds__(kAsmThreads, (!CK && MIXED) ? BIELCC_ASM_MINB : 0)
    assemble_far_kernel(const __grid_constant__ AsmArgsOf<MARKS> a) {
    using NodeT = typename std::conditional<MIXED, float4, double4>::type;
    constexpr int kWarps = kAsmThreads / 32;
    static_assert(kWarps == kAsmWays, "ways = 4 gives every warp its share of the columns");
    __shared__ __align__(16) RowBuf<NodeT> s_rows[kWarps];
    __shared__ RuleTab<NodeT> s_tab;
    using F = typename std::conditional<MIXED, float, double>::type;
    __shared__ F s_tau[kAsmStageCells][6];      // the column cells' tangents
    __shared__ double4 s_cell[kAsmStageCells];  // centre, near square
    __shared__ int s_mode[kAsmStageCells];      // mixed: phase polynomial; FP64: 1 phase split, 0 sincos per node
    __shared__ float s_rmin[kAsmStageCells][kMaxRules];
    __shared__ unsigned s_near[kWarps][32];
    extern __shared__ __align__(16) uint4 s_out[];  // STAGE: [warp][2][32][8] 16-byte pieces

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool split_cols = !STAGE && a.ways > 1;
    const int i = split_cols ? blockIdx.x * 32 + lane : blockIdx.x * kAsmThreads + threadIdx.x;
    const bool live = i < a.n_cells;
    const CellGeo& gi = a.geo[live ? i : 0];
    const double x[3] = {gi.c[0], gi.c[1], gi.c[2]};
    const int cb = blockIdx.y * a.cols_per_split;  // a multiple of 32
    const int ce = min(a.n_cells, cb + a.cols_per_split);
    const double k2r = a.k.re * a.k.re - a.k.im * a.k.im, k2i = 2.0 * a.k.re * a.k.im;
    const int n_lev = a.rules.n_lev;
    if (threadIdx.x == 0) {
        const NodeT* full;
        if constexpr (MIXED) full = a.nodes32;
        else full = a.nodes64;
        s_tab.fill(a.rules, rule_rows(a.rules, NodeT()), full, a.nn, a.n_cells);
    }

    unsigned cols = ~0u;  // MARKS: the block columns this pass writes
    const KF32 kf = KF32::make(a.k.re, a.k.im);
    // the row cell's tangents in FP32 (mixed-form block projection)
    float tif[2][3];
    if constexpr (MIXED) {
#pragma unroll
        for (int g = 0; g < 3; g++) {
            tif[0][g] = (float)gi.t1[g];
            tif[1][g] = (float)gi.t2[g];
        }
    }
    const int group = a.c64 ? 8 : 4;  // STAGE: columns per 128-byte row chunk
    uint4* out = STAGE ? s_out + warp * 512 : nullptr;

    for (int c0 = cb; c0 < ce; c0 += kAsmStageCells) {
        const int nc = min(kAsmStageCells, ce - c0);
        unsigned nbits = 0;  // near bits of this 32-column word
        __syncthreads();
        for (int q = threadIdx.x; q < nc * 6; q += kAsmThreads) {
            const CellGeo& gg = a.geo[c0 + q / 6];
            s_tau[q / 6][q % 6] = (F)(q % 6 < 3 ? gg.t1[q % 6] : gg.t2[q % 6 - 3]);
        }
        for (int q = threadIdx.x; q < nc; q += kAsmThreads) {
            s_cell[q] = near_cell(a.geo[c0 + q], a.analytic_calc);
            if constexpr (MIXED) s_mode[q] = phase_mode((float)fabs(a.k.re) * a.rho32[c0 + q]);
            else s_mode[q] = phase_range64(a.k, (double)a.rho32[c0 + q]) <= 0.5;
        }
        {
            const RuleK rk = rule_k(a.k);
            const float2* lim = rule_limits(a.rules, NodeT()) + (size_t)c0 * n_lev;
            for (int q = threadIdx.x; q < nc * n_lev; q += kAsmThreads)
                s_rmin[q / n_lev][q % n_lev] = CK ? rule_rmin(lim[q], rk) : rule_rmin_real(lim[q], rk);
        }
        __syncthreads();
        for (int cc = split_cols ? warp : 0; cc < nc; cc += split_cols ? kWarps : 1) {
            double dx[3], s2;
            const bool nr = near_exact(x, s_cell[cc], dx, &s2);
            const double d = dist_from_sq<!MIXED>(s2);
            bool far = live && !nr;
            nbits |= (nr ? 1u : 0u) << cc;
            if constexpr (MARKS) {
                if (far) {
                    const int c = c0 + cc;
                    const size_t wi = (size_t)(c >> 5) * a.n_cells + i;
                    const size_t plane = (size_t)((a.n_cells + 31) >> 5) * a.n_cells;
                    cols = 0u;
                    for (int b = 0; b < a.m; b++)
                        if ((((a.mark[b * plane + wi] >> (c & 31)) & 1u) != 0) == (a.take_marked != 0)) cols |= 1u << b;
                    far = cols != 0u;
                }
            }
            const float dmin = warp_min_pos(rule_key(far, d));
            const bool any = dmin < __int_as_float(0x7f800000);
            const F *tj1 = s_tau[cc], *tj2 = s_tau[cc] + 3;
            double Kr[3][3], Ki[3][3];     // FP64 form: the operator matrix
            Moments<float> m;              // mixed form: moments (A1, T)
            float phr = 0, phi = 0;        // and phase / 4pi
            m.zero();
            if (any) {
                const int lev = rule_level(s_rmin[cc], n_lev, dmin);
                const int cnt = s_tab.cnt[lev], mode = s_mode[cc];
                const NodeT* row = s_tab.base[lev] + (size_t)(c0 + cc) * cnt;
                NodeT v{};
                if (lane < cnt) v = row[lane];  // on its way during the pair's set-up
                PairF32 pf{};
                Moments<double> mm;
                double P0r = 1., P0i = 0.;
                if constexpr (MIXED) {
                    pf.set(dx, s2, d, kf);
                    turn_f32(d * (a.k.re * kInvTwoPi), CK ? exp(-a.k.im * d) * kInvFourPi : kInvFourPi, &phr, &phi);
                } else {
                    mm.zero();
                    if (mode) {
                        sincos(a.k.re * d, &P0i, &P0r);
                        if (CK) {
                            const double am = exp(-a.k.im * d);
                            P0r *= am;
                            P0i *= am;
                        }
                    }
                }
                for (int k0 = 0; k0 < cnt; k0 += kRowChunk) {
                    const int kc = min(kRowChunk, cnt - k0);
                    RowBuf<NodeT>& rb = s_rows[warp];
                    if (k0 && lane < kc) v = row[k0 + lane];
                    __syncwarp();  // the previous chunk has been read
                    rb.put(lane, v);
                    __syncwarp();
                    if (!far) continue;
                    if constexpr (MIXED) {
#define BIELCC_ASM_LOOP(MODE_)                                                \
    _Pragma("unroll 4") for (int q = 0; q < kc; q++)                          \
        far_node_f32<CK, MODE_, false>(m, pf, rb.get(q), kf);
                        switch (mode) {
                            case 0: BIELCC_ASM_LOOP(0) break;
                            case 1: BIELCC_ASM_LOOP(1) break;
                            case 2: BIELCC_ASM_LOOP(2) break;
                            case 3: BIELCC_ASM_LOOP(3) break;
                            default: BIELCC_ASM_LOOP(4) break;
                        }
#undef BIELCC_ASM_LOOP
                    } else if (mode) {
                        // FP64: the field kernel's node (phase relative to r0 with the Taylor
                        // series when |k| rho <= 0.5); its grad-F moments are unused here
#pragma unroll 2
                        for (int q = 0; q < kc; q++) {
                            const double4 y = rb.get(q);
                            far_node_f64<CK, true>(mm, x[0] - y.x, x[1] - y.y, x[2] - y.z, y.w, a.k, k2r, k2i, d);
                        }
                    } else {
#pragma unroll 2
                        for (int q = 0; q < kc; q++) {
                            const double4 y = rb.get(q);
                            far_node_f64<CK, false>(mm, x[0] - y.x, x[1] - y.y, x[2] - y.z, y.w, a.k, k2r, k2i, d);
                        }
                    }
                }
                if constexpr (MIXED) {
                    if constexpr (!CK) finish_real_k<float>(m.a1r, m.a1i, m.t);
                } else {
                    if (!CK) mm.finish_real_k();
                    // K = (A1 I + T) * P0 / 4pi
                    const int ti[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
#pragma unroll
                    for (int p = 0; p < 3; p++)
#pragma unroll
                        for (int q = 0; q < 3; q++) {
                            const double vr = mm.t[ti[p][q]][0] + (p == q ? mm.a1r : 0.);
                            const double vi = mm.t[ti[p][q]][1] + (p == q ? mm.a1i : 0.);
                            Kr[p][q] = (vr * P0r - vi * P0i) * kInvFourPi;
                            Ki[p][q] = (vr * P0i + vi * P0r) * kInvFourPi;
                        }
                }
            }
            if constexpr (STAGE) {
                const int g = cc & (group - 1);
                // 16-byte pieces of matrix row r (0, 1) of this lane: complex64, piece g is the
                // column cell's pair; complex128, pieces 2 g and 2 g + 1 its two entries
                if constexpr (MIXED) {
                    float o[2][2][2];
                    block_f32<2>(m.a1r, m.a1i, m.t, phr, phi, tif, tj1, tj2, o);
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        uint4* w = out + (r * 32 + lane) * 8;
                        if (a.c64) {
                            *reinterpret_cast<float4*>(w + ((g + lane) & 7)) =
                                make_float4(o[r][0][0], o[r][0][1], o[r][1][0], o[r][1][1]);
                        } else {
#pragma unroll
                            for (int b = 0; b < 2; b++)
                                *reinterpret_cast<double2*>(w + ((2 * g + b + lane) & 7)) =
                                    make_double2(o[r][b][0], o[r][b][1]);
                        }
                    }
                } else {
                    double o[2][2][2] = {};
                    if (any) block_f64<2>(Kr, Ki, gi.t1, gi.t2, tj1, tj2, o);
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        uint4* w = out + (r * 32 + lane) * 8;
                        if (a.c64) {
                            *reinterpret_cast<float4*>(w + ((g + lane) & 7)) = make_float4(
                                (float)o[r][0][0], (float)o[r][0][1], (float)o[r][1][0], (float)o[r][1][1]);
                        } else {
#pragma unroll
                            for (int b = 0; b < 2; b++)
                                *reinterpret_cast<double2*>(w + ((2 * g + b + lane) & 7)) =
                                    make_double2(o[r][b][0], o[r][b][1]);
                        }
                    }
                }
                if (g == group - 1 || cc == nc - 1) {  // the group's columns, four matrix rows at a time
                    __syncwarp();
                    const int pieces = a.c64 ? g + 1 : 2 * (g + 1), piece = lane & 7;
                    const size_t pitch = (size_t)2 * a.n_cells * (a.c64 ? 8 : 16);  // bytes of a matrix row
                    char* base = (char*)a.A + (size_t)(c0 + cc - g) * (a.c64 ? 16 : 32) + 16 * piece;
                    const int i0 = blockIdx.x * kAsmThreads + warp * 32;
#pragma unroll 4
                    for (int it = 0; it < 16; it++) {
                        const int r = it >> 3, l = ((it & 7) << 2) + (lane >> 3);  // matrix row r of row cell i0 + l
                        if (piece < pieces && i0 + l < a.n_cells)
                            *reinterpret_cast<uint4*>(base + (size_t)(2 * (i0 + l) + r) * pitch) =
                                out[(r * 32 + l) * 8 + ((piece + l) & 7)];
                    }
                    __syncwarp();
                }
            } else if (far) {
                if constexpr (MIXED) {
                    if (a.m == 2) write_block_f32<2>(a, i, c0 + cc, m.a1r, m.a1i, m.t, phr, phi, tif, tj1, tj2, cols);
                    else write_block_f32<3>(a, i, c0 + cc, m.a1r, m.a1i, m.t, phr, phi, tif, tj1, tj2, cols);
                } else {
                    write_block(a, i, c0 + cc, Kr, Ki, gi.t1, gi.t2, tj1, tj2, cols);
                }
            }
        }
        if (split_cols) {
            s_near[warp][lane] = nbits;
            __syncthreads();
            if (warp == 0) {
#pragma unroll
                for (int w = 1; w < kWarps; w++) nbits |= s_near[w][lane];
            }
        }
        if (live && a.mask && (!split_cols || warp == 0)) a.mask[(size_t)(c0 >> 5) * a.n_cells + i] = nbits;
    }
}

// ---------------------------------------------------------------- adaptive far blocks (p_max >= 3)
// The reference runs one refinement loop per matrix column: K_RotRot_Far
// (K.h:288-301) of the column's basis current J_b (tau_b of the column cell, or
// e_b) at the row cell's centre, which stops at the first pass after the first
// whose squared change is below eps^2 (integral_universal.h:58-119), else
// returns its last pass. asm_refine_decide_kernel runs the test at the second
// pass for every far block and column from the FP64 node tables at n_start and
// 2 n_start, writes the near mask, and marks the failing columns in
// mark[b]. The marks-reading far kernel then writes the columns that passed
// from the 2 n_start tables and, with p_max = 3, the failing ones from the
// 4 n_start tables; with p_max > 3 the failing ones run the whole loop in
// assemble_far_refine_kernel.

// One FP64 pass over a cell's node table row (the field kernels' FP64 node,
// K moments only), finished and ready for K = (A1 I + T) J.
template <bool CK>
BIELCC_D void asm_pass_f64(Moments<double>& m, const double4* __restrict__ nd, int nn, const double* x, cplx k,
                           double k2r, double k2i, double r0, bool split) {
    m.zero();
    if (split) {
#pragma unroll 8
        for (int q = 0; q < nn; q++) {
            const double4 v = ldg_node(nd + q);
            far_node_f64<CK, true>(m, x[0] - v.x, x[1] - v.y, x[2] - v.z, v.w, k, k2r, k2i, r0);
        }
    } else {
#pragma unroll 8
        for (int q = 0; q < nn; q++) {
            const double4 v = ldg_node(nd + q);
            far_node_f64<CK, false>(m, x[0] - v.x, x[1] - v.y, x[2] - v.z, v.w, k, k2r, k2i, r0);
        }
    }
    if (!CK) m.finish_real_k();
}

// The squared change of column b's raw integral (A1 J + T J) P0 between two
// passes, |.| taken first as in integral_universal.h:96-99.
BIELCC_D double asm_delta2(const Moments<double>& m0, const Moments<double>& m1, const double* J, double pr,
                           double pi) {
    const int ti[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    double d = 0.;
    for (int p = 0; p < 3; p++) {
        double e0r = m0.a1r * J[p], e0i = m0.a1i * J[p], e1r = m1.a1r * J[p], e1i = m1.a1i * J[p];
        for (int q = 0; q < 3; q++) {
            e0r += m0.t[ti[p][q]][0] * J[q];
            e0i += m0.t[ti[p][q]][1] * J[q];
            e1r += m1.t[ti[p][q]][0] * J[q];
            e1i += m1.t[ti[p][q]][1] * J[q];
        }
        const cplx k0 = mk(e0r, e0i) * mk(pr, pi), k1 = mk(e1r, e1i) * mk(pr, pi);
        const double t = sqrt(cabs2(k1 - k0));
        d += t * t;
    }
    return d;
}

// Each pass takes the shortest row its table's rules allow (rules.cu, FP64 limits).
__global__ void asm_refine_decide_kernel(const __grid_constant__ AsmArgs a, const __grid_constant__ FarRules rules_lo,
                                         const double4* __restrict__ lo, int nn_lo, double eps2,
                                         unsigned* __restrict__ mark) {
    __shared__ RuleTab<double4> s_lo, s_hi;
    __shared__ float s_rmin[2][kAsmStageCells][kMaxRules];
    const int i = blockIdx.x * kAsmThreads + threadIdx.x;
    const bool live = i < a.n_cells;
    const CellGeo gi = a.geo[live ? i : 0];
    const double* x = gi.c;
    const int cb = blockIdx.y * a.cols_per_split;  // a multiple of 32
    const int ce = min(a.n_cells, cb + a.cols_per_split);
    const bool ck = a.k.im != 0.0;
    const double k2r = a.k.re * a.k.re - a.k.im * a.k.im, k2i = 2.0 * a.k.re * a.k.im;
    const size_t plane = (size_t)((a.n_cells + 31) >> 5) * a.n_cells;
    const int nlo = rules_lo.n_lev, nhi = a.rules.n_lev;
    if (threadIdx.x == 0) {
        s_lo.fill(rules_lo, rules_lo.n64, lo, nn_lo, a.n_cells);
        s_hi.fill(a.rules, a.rules.n64, a.nodes64, a.nn, a.n_cells);
    }
    unsigned nbits = 0, mb[3] = {0u, 0u, 0u};
    for (int j = cb; j < ce; j++) {
        if ((j & 31) == 0) {
            const int nc = min(kAsmStageCells, ce - j);
            const RuleK rk = rule_k(a.k);
            __syncthreads();  // the previous columns' limits are no longer read
            for (int q = threadIdx.x; q < nc * nlo; q += kAsmThreads)
                s_rmin[0][q / nlo][q % nlo] = rule_rmin(rules_lo.thr64[(size_t)j * nlo + q], rk);
            for (int q = threadIdx.x; q < nc * nhi; q += kAsmThreads)
                s_rmin[1][q / nhi][q % nhi] = rule_rmin(a.rules.thr64[(size_t)j * nhi + q], rk);
            __syncthreads();
        }
        const CellGeo& gj = a.geo[j];
        double d;
        const bool nr = asm_is_near(x, gj, a.analytic_calc, &d);
        const bool far = live && !nr;
        const float dmin = warp_min_pos(rule_key(far, d));
        const int llo = rule_level(s_rmin[0][j & 31], nlo, dmin), lhi = rule_level(s_rmin[1][j & 31], nhi, dmin);
        if (far) {
            const int n_lo = s_lo.cnt[llo], n_hi = s_hi.cnt[lhi];
            const double4* row_lo = s_lo.base[llo] + (size_t)j * n_lo;
            const double4* row_hi = s_hi.base[lhi] + (size_t)j * n_hi;
            const bool split = !ck && fabs(a.k.re) * (double)a.rho32[j] * (1.0 + 1e-6) <= 0.5;
            double pr = 1.0, pi = 0.0;
            if (split) sincos(a.k.re * d, &pi, &pr);
            Moments<double> m0, m1;
            if (ck) {
                asm_pass_f64<true>(m0, row_lo, n_lo, x, a.k, k2r, k2i, d, false);
                asm_pass_f64<true>(m1, row_hi, n_hi, x, a.k, k2r, k2i, d, false);
            } else {
                asm_pass_f64<false>(m0, row_lo, n_lo, x, a.k, k2r, k2i, d, split);
                asm_pass_f64<false>(m1, row_hi, n_hi, x, a.k, k2r, k2i, d, split);
            }
            for (int b = 0; b < a.m; b++) {
                double J[3];
                for (int g = 0; g < 3; g++) J[g] = a.m == 3 ? (g == b ? 1. : 0.) : (b == 0 ? gj.t1[g] : gj.t2[g]);
                if (!(asm_delta2(m0, m1, J, pr, pi) < eps2)) mb[b] |= 1u << (j & 31);
            }
        }
        nbits |= (nr ? 1u : 0u) << (j & 31);
        if ((j & 31) == 31 || j == ce - 1) {
            const size_t wi = (size_t)(j >> 5) * a.n_cells + i;
            if (live) {
                if (a.mask) a.mask[wi] = nbits;
                for (int b = 0; b < a.m; b++) mark[b * plane + wi] = mb[b];
            }
            nbits = 0;
            mb[0] = mb[1] = mb[2] = 0u;
        }
    }
}

// p_max > 3: the marked (row, column, basis) far entries through the whole
// loop (integral_cell, ops.cuh: nodes on the fly).
__global__ void assemble_far_refine_kernel(AsmArgs a, const unsigned* __restrict__ mark, const double* __restrict__ verts,
                                           int nv, DNP np) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n_cells) return;
    const CellGeo gi = a.geo[i];
    const int cb = blockIdx.y * a.cols_per_split;
    const int ce = min(a.n_cells, cb + a.cols_per_split);
    const int m = a.m;
    const size_t plane = (size_t)((a.n_cells + 31) >> 5) * a.n_cells;
    for (int j = cb; j < ce; j++) {
        const size_t wi = (size_t)(j >> 5) * a.n_cells + i;
        unsigned cols = 0u;
        for (int b = 0; b < m; b++) cols |= ((mark[b * plane + wi] >> (j & 31)) & 1u) << b;
        if (!cols) continue;
        const CellGeo& gj = a.geo[j];
        DCell cl;
        cl.nv = nv;
        for (int v = 0; v < nv; v++)
            for (int g = 0; g < 3; g++) cl.v[v][g] = verts[((size_t)j * nv + v) * 3 + g];
        cplx v[3][3];  // v[b] = K[J_b], J_b = tau_b(j) (TAU2) or e_b (FULL3)
        for (int b = 0; b < m; b++) {
            if (!((cols >> b) & 1u)) continue;
            DKP kp;
            dkp_zero(kp);
            kp.smoothR = kMachineZero;
            kp.smoothRMin = kMachineZero;
            kp.k = a.k;
            for (int g = 0; g < 3; g++)
                kp.current[g] = mk(m == 3 ? (g == b ? 1. : 0.) : (b == 0 ? gj.t1[g] : gj.t2[g]), 0.);
            integral_cell<cplx>(F_ROTROTSIMPLEPOT_H, gi.c, cl, kp, 3, np.n_start, np.p_max, np.eps, v[b]);
        }
        const size_t dim = (size_t)m * a.n_cells;
        for (int aa = 0; aa < m; aa++) {
            size_t off = ((size_t)i * m + aa) * dim + (size_t)j * m;
            for (int b = 0; b < m; b++) {
                if (!((cols >> b) & 1u)) continue;
                cplx e = m == 3 ? v[b][aa]
                                : (aa == 0 ? v[b][0] * gi.t1[0] + v[b][1] * gi.t1[1] + v[b][2] * gi.t1[2]
                                           : v[b][0] * gi.t2[0] + v[b][1] * gi.t2[1] + v[b][2] * gi.t2[2]);
                e = e * kInvFourPi;
                if (a.c64) reinterpret_cast<float2*>(a.A)[off + b] = make_float2((float)e.re, (float)e.im);
                else reinterpret_cast<double2*>(a.A)[off + b] = make_double2(e.re, e.im);
            }
        }
    }
}

// Near pairs from the far kernel's bit mask (row i, word w: the near test of
// get_field.h:58 for columns 32w..32w+31, evaluated there with the same
// non-contracted FP64 arithmetic): counts per row, then the (row, column)
// pairs in ascending column order.
__global__ void asm_mask_count_kernel(const unsigned* __restrict__ mask, int n_words, int n_cells,
                                      long long* __restrict__ counts) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_cells) return;
    long long n = 0;
    for (int w = 0; w < n_words; w++) n += __popc(mask[(size_t)w * n_cells + i]);
    counts[i] = n;
}

__global__ void asm_mask_fill_kernel(const unsigned* __restrict__ mask, int n_words, int n_cells,
                                     const long long* __restrict__ offs, int* __restrict__ pr, int* __restrict__ pc) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_cells) return;
    long long o = offs[i];
    for (int w = 0; w < n_words; w++) {
        unsigned b = mask[(size_t)w * n_cells + i];
        while (b) {
            const int bit = __ffs(b) - 1;
            b &= b - 1;
            pr[o] = i;
            pc[o] = w * 32 + bit;
            o++;
        }
    }
}

// K_RotRot_HS_Colloc (electrodynamics/K.h:179-204) at x as a 3x3 operator, FP64.
BIELCC_D void near_operator(const DCell& cl, const double* x, cplx k, const DNP& np, double (&Kr)[3][3],
                            double (&Ki)[3][3]) {
    cplx I = surf_simplepot_h_hs_dev(cl, x, np.analytic_calc, np.n_start, np.p_max, np.eps, k);
    cplx sI = I * k * k / kFourPi;
    DKP ps;
    dkp_zero(ps);
    ps.smoothR = kMachineZero;
    ps.smoothRMin = kMachineZero;
    ps.k = k;
    cplx M[3][3], dummy[3];
    K0_dev(F_GRADSIMPLEPOT_H, nullptr, x, cl, ps, np.n_start_seg, np.p_max_seg, np.eps, dummy, M);
    for (int p = 0; p < 3; p++)
        for (int r = 0; r < 3; r++) {
            cplx v = M[p][r] / kFourPi;
            if (p == r) v += sI;
            Kr[p][r] = v.re;
            Ki[p][r] = v.im;
        }
}

// Near entries: K_RotRot_HS_Colloc as a 3x3 operator, FP64.
template <int G>
__global__ void asm_near_kernel(AsmArgs a, const double* __restrict__ verts, int nv, const int* __restrict__ pr,
                                const int* __restrict__ pc, long long n_pairs, DNP np) {
    const Lanes<G> g = Lanes<G>::make();
    const long long q = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G;
    if (q >= n_pairs) return;  // whole groups
    int i = pr[q], j = pc[q];
    const CellGeo &gi = a.geo[i], &gj = a.geo[j];
    DCell cl;
    cl.nv = nv;
    for (int v = 0; v < nv; v++)
        for (int h = 0; h < 3; h++) cl.v[v][h] = verts[((size_t)j * nv + v) * 3 + h];
    const double x[3] = {gi.c[0], gi.c[1], gi.c[2]};
    cplx K[3][3];
    group_hs_colloc<G>(g, x, cl, a.k, np, K);
    if (g.l != 0) return;
    double Kr[3][3], Ki[3][3];
    for (int p = 0; p < 3; p++)
        for (int r = 0; r < 3; r++) {
            Kr[p][r] = K[p][r].re;
            Ki[p][r] = K[p][r].im;
        }
    write_block(a, i, j, Kr, Ki, gi.t1, gi.t2, gj.t1, gj.t2);
}

// Error sample of a mixed assembly: rows of the cells i_r = r N / R
// (r < R), every column, recomputed in FP64 with the per-pair operators
// (K_RotRot_HS_Colloc near, K_RotRot_Far far, electrodynamics/K.h) and
// projected as the stored entries are; each block sums |stored - FP64|^2
// and |FP64|^2 of its (row, column) pairs into part[block] (fixed order).
__global__ void asm_error_sample_kernel(AsmArgs a, const double* __restrict__ verts, int nv, int R, DNP np,
                                        double2* __restrict__ part) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int N = a.n_cells, M = a.m;
    double num = 0., den = 0.;
    if (q < (long long)R * N) {
        const int r = (int)(q / N), j = (int)(q - (long long)r * N);
        const int i = (int)((long long)r * N / R);
        const CellGeo gi = a.geo[i], gj = a.geo[j];
        DCell cl;
        cl.nv = nv;
        for (int v = 0; v < nv; v++)
            for (int g = 0; g < 3; g++) cl.v[v][g] = verts[((size_t)j * nv + v) * 3 + g];
        const double* x = gi.c;
        double d;
        double Kr[3][3], Ki[3][3];
        if (asm_is_near(x, gj, a.analytic_calc, &d)) {
            near_operator(cl, x, a.k, np, Kr, Ki);
        } else if (np.p_max <= 2) {
            // one FP64 pass at the far pass's split (p_max = 2: 2 n_start) over nodes of its
            // own, with the phase of each: neither the mesh's tables nor a rule, whose errors
            // the sample is there to see. 20,480 triangles, 16 rows, whole call: 18.7 ms, as
            // over the rows of the table's rules (18.8); K_far_dev per column (p_max > 2) took
            // 2.46 ms for the sample alone.
            const int n = np.p_max == 2 ? 2 * np.n_start : np.n_start;
            const double area = nv == 3 ? tri_area(cl.v[0], cl.v[1], cl.v[2]) / n / n : 1.;
            const double k2r = a.k.re * a.k.re - a.k.im * a.k.im, k2i = 2.0 * a.k.re * a.k.im;
            Moments<double> mm;
            mm.zero();
            const bool ck = a.k.im != 0.;
            cell_nodes<1>(Lanes<1>::make(), cl, n, [&](const double* y, double w) {
                if (ck) far_node_f64<true, false>(mm, x[0] - y[0], x[1] - y[1], x[2] - y[2], w * area, a.k, k2r, k2i, d);
                else far_node_f64<false, false>(mm, x[0] - y[0], x[1] - y[1], x[2] - y[2], w * area, a.k, k2r, k2i, d);
            });
            if (!ck) mm.finish_real_k();
            const int ti[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
            for (int p = 0; p < 3; p++)
                for (int r = 0; r < 3; r++) {
                    const cplx v = mk(mm.t[ti[p][r]][0] + (p == r ? mm.a1r : 0.),
                                      mm.t[ti[p][r]][1] + (p == r ? mm.a1i : 0.)) * kInvFourPi;
                    Kr[p][r] = v.re;
                    Ki[p][r] = v.im;
                }
        } else {
            for (int b = 0; b < 3; b++) {  // K_RotRot_Far is linear in the current: one column per basis vector
                cplx e[3] = {mk(b == 0, 0.), mk(b == 1, 0.), mk(b == 2, 0.)}, col[3];
                K_far_dev(e, x, cl, np, a.k, col);
                for (int p = 0; p < 3; p++) {
                    Kr[p][b] = col[p].re;
                    Ki[p][b] = col[p].im;
                }
            }
        }
        const size_t dim = (size_t)M * N;
        for (int aa = 0; aa < M; aa++)
            for (int b = 0; b < M; b++) {
                double vr = 0., vi = 0.;
                if (M == 3) {
                    vr = Kr[aa][b];
                    vi = Ki[aa][b];
                } else {
                    const double* ta = aa == 0 ? gi.t1 : gi.t2;
                    const double* tb = b == 0 ? gj.t1 : gj.t2;
                    for (int p = 0; p < 3; p++) {
                        vr += ta[p] * (Kr[p][0] * tb[0] + Kr[p][1] * tb[1] + Kr[p][2] * tb[2]);
                        vi += ta[p] * (Ki[p][0] * tb[0] + Ki[p][1] * tb[1] + Ki[p][2] * tb[2]);
                    }
                }
                const size_t off = ((size_t)i * M + aa) * dim + (size_t)j * M + b;
                double sr, si;
                if (a.c64) {
                    const float2 v = reinterpret_cast<const float2*>(a.A)[off];
                    sr = v.x;
                    si = v.y;
                } else {
                    const double2 v = reinterpret_cast<const double2*>(a.A)[off];
                    sr = v.x;
                    si = v.y;
                }
                num += (sr - vr) * (sr - vr) + (si - vi) * (si - vi);
                den += vr * vr + vi * vi;
            }
    }
    __shared__ double sn[128], sd[128];
    sn[threadIdx.x] = num;
    sd[threadIdx.x] = den;
    __syncthreads();
    for (int w = 64; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            sn[threadIdx.x] += sn[threadIdx.x + w];
            sd[threadIdx.x] += sd[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = make_double2(sn[0], sd[0]);
}

__global__ void asm_error_sum_kernel(const double2* __restrict__ part, int n, double* __restrict__ sums) {
    double a = 0., b = 0.;
    for (int i = 0; i < n; i++) {
        a += part[i].x;
        b += part[i].y;
    }
    sums[0] = a;
    sums[1] = b;
}

static size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

// Column blocks of the (row, column word) marks of p_max >= 3: one per basis vector.
static int asm_mark_planes(const AssembleLaunch& a) { return far_adaptive(a.np) ? (a.layout == 1 ? 3 : 2) : 0; }

size_t assemble_ws_base_bytes(const AssembleLaunch& a) {
    size_t N = a.mesh->n_cells;
    return 2 * al256((N + 1) * sizeof(long long)) + al256((N + 31) / 32 * N * sizeof(unsigned)) + 256 +
           al256((size_t)asm_mark_planes(a) * ((N + 31) / 32) * N * sizeof(unsigned));
}

static AsmArgs make_args(const AssembleLaunch& a) {
    const MeshDev& m = *a.mesh;
    AsmArgs g;
    g.geo = m.geo;
    g.n_cells = m.n_cells;
    g.nodes64 = m.nodes64;
    g.nodes32 = m.nodes32;
    g.rho32 = m.rho32;
    g.rules = rules_read(m.rules, a.precision != 1);
    g.nn = far_split_n(a.np) * far_split_n(a.np);
    g.k = a.k;
    g.analytic_calc = a.np.analytic_calc;
    g.ways = 1;
    g.m = a.layout == 1 ? 3 : 2;
    g.c64 = a.out_c64;
    g.A = a.A;
    g.mask = nullptr;
    return g;
}

// Resident CTAs (whole GPU) of the far assembly kernel variant.
static int asm_slots(bool ck, bool mixed, bool stage) {
    static std::atomic<int> cache[2][2][2];
    std::atomic<int>& c = cache[ck][mixed][stage];
    int v = c.load(std::memory_order_relaxed);
    if (v) return v;
    int dev = 0, sms = 148, per = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
#define BIELCC_AK(C, M) \
    (stage ? (const void*)assemble_far_kernel<C, M, false, true> : (const void*)assemble_far_kernel<C, M, false, false>)
    const void* fn = ck ? (mixed ? BIELCC_AK(true, true) : BIELCC_AK(true, false))
                        : (mixed ? BIELCC_AK(false, true) : BIELCC_AK(false, false));
#undef BIELCC_AK
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, kAsmThreads, stage ? kAsmOutBytes : 0);
    v = std::max(1, sms * std::max(1, per));
    c.store(v, std::memory_order_relaxed);
    return v;
}

cudaError_t assemble_stage1(const AssembleLaunch& a, void* ws, long long* d_total, cudaStream_t s) {
    const MeshDev& m = *a.mesh;
    const int N = m.n_cells;
    long long* counts = (long long*)ws;
    long long* offs = (long long*)((char*)ws + al256((size_t)(N + 1) * sizeof(long long)));
    unsigned* mask = (unsigned*)((char*)offs + al256((size_t)(N + 1) * sizeof(long long)));
    const int n_words = (N + 31) / 32;
    AsmArgs g = make_args(a);
    g.mask = mask;  // written by the far kernel (p_max <= 2) or the decision kernel (p_max >= 3)
    int tiles = (N + kAsmThreads - 1) / kAsmThreads;
    bool ck = a.k.im != 0.;
    // column splits in whole 32-column words, so every mask word has one writer
    if (m.table_n != far_split_n(a.np))
        return cudaErrorInvalidValue;  // node tables of another split: the caller builds far_split_n's
    if (far_adaptive(a.np) && (m.table_lo_n != a.np.n_start || !m.nodes64_lo))
        return cudaErrorInvalidValue;  // no n_start table for the convergence test
    if (far_third_pass(a.np) && (m.table_hi_n != 4 * a.np.n_start || !m.nodes64_hi))
        return cudaErrorInvalidValue;  // no 4 n_start tables for the third pass
    // staged blocks are written 16 bytes at a time: a complex64 matrix may start
    // between 16-byte boundaries, which the direct writes take
    const bool stage = g.m == 2 && !far_adaptive(a.np) && (reinterpret_cast<uintptr_t>(a.A) & 15) == 0;
    const int slots = asm_slots(ck, a.precision == 1, stage);
    // fewer 128-row CTAs than slots at one mask word (32 columns) per split: the
    // warps share the columns (not under the marks of p_max >= 3, whose decision
    // kernel sets the grid)
    g.ways = !far_adaptive(a.np) && (size_t)tiles * n_words < (size_t)slots ? kAsmWays : 1;
    const int far_tiles = g.ways > 1 ? (N + 31) / 32 : tiles;
    const int splits = choose_cell_splits(far_tiles, N, slots, N);
    g.cols_per_split = round_cells_per_split(N, splits);
    const dim3 grid(far_tiles, splits);
    if (far_adaptive(a.np)) {
        unsigned* mark = (unsigned*)((char*)mask + al256((size_t)n_words * N * sizeof(unsigned)) + 256);
        const int nn_lo = a.np.n_start * a.np.n_start;
        AsmArgs gd = g;
        gd.rules = rules_read(m.rules, true);  // FP64 rows in either precision
        asm_refine_decide_kernel<<<grid, kAsmThreads, 0, s>>>(gd, rules_read(m.rules_lo, true), m.nodes64_lo, nn_lo,
                                                              a.np.eps * a.np.eps, mark);
        AsmArgsMarks gm;
        static_cast<AsmArgs&>(gm) = g;
        gm.mask = nullptr;  // written by the decision kernel
        gm.mark = mark;
        gm.take_marked = 0;  // the columns that passed: the pass at 2 n_start
        if (a.precision == 1) {
            if (ck) assemble_far_kernel<true, true, true><<<grid, kAsmThreads, 0, s>>>(gm);
            else assemble_far_kernel<false, true, true><<<grid, kAsmThreads, 0, s>>>(gm);
        } else {
            if (ck) assemble_far_kernel<true, false, true><<<grid, kAsmThreads, 0, s>>>(gm);
            else assemble_far_kernel<false, false, true><<<grid, kAsmThreads, 0, s>>>(gm);
        }
        if (far_third_pass(a.np)) {  // p_max = 3: the failing columns return the pass at 4 n_start
            gm.nodes64 = m.nodes64_hi;
            gm.nodes32 = m.nodes32_hi;
            gm.rho32 = m.rho32_hi;
            gm.rules = rules_read(m.rules_hi, a.precision != 1);
            gm.nn = 16 * a.np.n_start * a.np.n_start;
            gm.take_marked = 1;
            if (a.precision == 1) {
                if (ck) assemble_far_kernel<true, true, true><<<grid, kAsmThreads, 0, s>>>(gm);
                else assemble_far_kernel<false, true, true><<<grid, kAsmThreads, 0, s>>>(gm);
            } else {
                if (ck) assemble_far_kernel<true, false, true><<<grid, kAsmThreads, 0, s>>>(gm);
                else assemble_far_kernel<false, false, true><<<grid, kAsmThreads, 0, s>>>(gm);
            }
        } else {
            DNP np{a.np.eps, a.np.rs, a.np.rs_seg, a.np.analytic_calc, a.np.n_start, a.np.n_start_seg, a.np.p_max,
                   a.np.p_max_seg};
            assemble_far_refine_kernel<<<grid, kAsmThreads, 0, s>>>(g, mark, m.verts, m.nv, np);
        }
    } else if (stage && g.ways == 1) {
        if (a.precision == 1) {
            if (ck) assemble_far_kernel<true, true, false, true><<<grid, kAsmThreads, kAsmOutBytes, s>>>(g);
            else assemble_far_kernel<false, true, false, true><<<grid, kAsmThreads, kAsmOutBytes, s>>>(g);
        } else {
            if (ck) assemble_far_kernel<true, false, false, true><<<grid, kAsmThreads, kAsmOutBytes, s>>>(g);
            else assemble_far_kernel<false, false, false, true><<<grid, kAsmThreads, kAsmOutBytes, s>>>(g);
        }
    } else if (a.precision == 1) {
        if (ck) assemble_far_kernel<true, true><<<grid, kAsmThreads, 0, s>>>(g);
        else assemble_far_kernel<false, true><<<grid, kAsmThreads, 0, s>>>(g);
    } else {
        if (ck) assemble_far_kernel<true, false><<<grid, kAsmThreads, 0, s>>>(g);
        else assemble_far_kernel<false, false><<<grid, kAsmThreads, 0, s>>>(g);
    }
    asm_mask_count_kernel<<<tiles, kAsmThreads, 0, s>>>(mask, n_words, N, counts);
    scan_kernel<<<1, 1024, 0, s>>>(counts, N, offs, d_total);
    return cudaGetLastError();
}

cudaError_t assemble_stage2(const AssembleLaunch& a, void* ws, long long n_near, void* pair_ws, cudaStream_t s) {
    if (n_near <= 0) return cudaSuccess;
    const MeshDev& m = *a.mesh;
    const int N = m.n_cells;
    long long* offs = (long long*)((char*)ws + al256((size_t)(N + 1) * sizeof(long long)));
    const unsigned* mask = (const unsigned*)((char*)offs + al256((size_t)(N + 1) * sizeof(long long)));
    int* pr = (int*)pair_ws;
    int* pc = pr + n_near;
    int tiles = (N + kAsmThreads - 1) / kAsmThreads;
    asm_mask_fill_kernel<<<tiles, kAsmThreads, 0, s>>>(mask, (N + 31) / 32, N, offs, pr, pc);
    AsmArgs g = make_args(a);
    DNP np{a.np.eps, a.np.rs, a.np.rs_seg, a.np.analytic_calc, a.np.n_start, a.np.n_start_seg, a.np.p_max,
           a.np.p_max_seg};
    const int lanes = near_lanes(n_near, np), blocks = (int)((n_near * lanes + 127) / 128);
    const auto near_blocks = lanes == 1 ? asm_near_kernel<1> : (lanes == 8 ? asm_near_kernel<8> : asm_near_kernel<32>);
    near_blocks<<<blocks, 128, 0, s>>>(g, m.verts, m.nv, pr, pc, n_near, np);
    return cudaGetLastError();
}

size_t assemble_error_ws_bytes(const AssembleLaunch& a, int R) {
    return al256((size_t)(((long long)R * a.mesh->n_cells + 127) / 128) * sizeof(double2)) + 256;
}

cudaError_t assemble_error_sample(const AssembleLaunch& a, int R, void* ws, double* sums, cudaStream_t s) {
    const MeshDev& m = *a.mesh;
    const long long tot = (long long)R * m.n_cells;
    const int blocks = (int)((tot + 127) / 128);
    AsmArgs g = make_args(a);
    DNP np{a.np.eps, a.np.rs, a.np.rs_seg, a.np.analytic_calc, a.np.n_start, a.np.n_start_seg, a.np.p_max,
           a.np.p_max_seg};
    double2* part = (double2*)ws;
    asm_error_sample_kernel<<<blocks, 128, 0, s>>>(g, m.verts, m.nv, R, np, part);
    asm_error_sum_kernel<<<1, 1, 0, s>>>(part, blocks, sums);
    return cudaGetLastError();
}

}  // namespace bielcc_gpu
