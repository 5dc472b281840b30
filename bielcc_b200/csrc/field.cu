// field.cu — E/H field over every observation-point x cell pair: the
// GetFieldE_Ideal driver (electrodynamics/get_field.h:35-78) and its H
// counterpart (examples/field/main0_field_test.cpp:237-311) on sm_100a.
//
// Pipeline (one stream, deterministic summation order):
//   1. far kernel   — one observation point per thread, cells split across
//                     gridDim.y (the split count is chosen per launch so that
//                     the last wave of CTAs fills the GPU: grid.h) and, on
//                     problems too small for that, across the CTA's warps;
//                     far cells only (near cells skipped). Per cell
//                     the J-independent moments A1 = sum w e f1,
//                     T = sum w e f2 d^d^T, G = sum w grad F are accumulated over
//                     the nodes of the shortest quadrature row that reproduces
//                     the n x n sum to rounding at this distance (rules.cu) and
//                     contracted with each right-hand side once per cell:
//                       K_RotRot_Far  (K.h:288-301)  = (A1 J + T J) / 4pi
//                       R_Rot_Colloc  (R.h:89-111)   = (G x J) / 4pi
//                     FP64 form: FP64 everywhere. Mixed form: nodes relative to
//                     the cell centre in FP32, phase split e^{ikr} =
//                     e^{ik r0} e^{ik (r - r0)} with r0 = |x - centre| and
//                     e^{ik r0} in FP64, r - r0 = q / (r + r0) with
//                     q = |delta|^2 - 2 delta.X (no cancellation), FP32 cell sums,
//                     FP64 accumulation across cells.
//   2. near count + scan + fill — per point, the cells with
//                     |x - centre| < analytic_calc * diam (get_field.h:58), in
//                     cell order.
//   3. near pair kernel — FP64, a group of lanes per pair: the J-independent parts of
//                     K_RotRot_Near_Smooth (K.h:47-79) and R_Rot_Smooth
//                     (R.h:46-61) with the reference's adaptive quadrature.
//   4. near sums    — one warp per (point, RHS): the point's near pairs
//                     contracted with J, lane-strided in cell order, fixed
//                     butterfly across the lanes.
//   5. finalize     — per (point, RHS): far partials over splits (in order) +
//                     the near sum, x mult, + incident field.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "farnode.cuh"
#include "grid.h"
#include "internal.h"
#include "ops.cuh"
#include "scan.cuh"

namespace bielcc_gpu {

#ifndef BIELCC_FAR_THREADS
#define BIELCC_FAR_THREADS 128
#endif
constexpr int kFarThreads = BIELCC_FAR_THREADS;
// Unrolling of the mixed node loop (rows of 8 - 20 nodes mostly; 8192 cells x
// 20,000 points, whole call: x2 7.23, x3 7.50, x4 7.26, x8 7.29 ms).
#ifndef BIELCC_FAR_UNROLL
#define BIELCC_FAR_UNROLL 4
#endif
#define BIELCC_FAR_STR(x) #x
#define BIELCC_FAR_PRAGMA(x) _Pragma(BIELCC_FAR_STR(unroll x))
#define BIELCC_FAR_UNROLL_PRAGMA BIELCC_FAR_PRAGMA(BIELCC_FAR_UNROLL)
// Unrolling of the FP64 split node loop (far points only: 5120 triangles x 6001 points
// x2 4.95, x3 4.94, x4 4.86 ms; 8192 quads x 2000 points 3.04, 3.04, 2.97; with the
// cells over the warps, where the warps are at different places in the code, 80
// triangles x 100 points 0.087, 0.086, 0.085, but x8 cost 70 % more than x2 in
// instruction-cache misses).
#ifndef BIELCC_FAR64_UNROLL
#define BIELCC_FAR64_UNROLL 4
#endif
#define BIELCC_FAR64_UNROLL_PRAGMA BIELCC_FAR_PRAGMA(BIELCC_FAR64_UNROLL)
// Minimum resident CTAs per SM asked of the 1-RHS real-k mixed far kernel
// (0: none, the compiler's own register choice, which the other variants
// keep). 4 allows 128 registers, no spills; 8192 cells x 20,000 points 6.55 ms
// (5: 96 registers, 6.82 ms).
#ifndef BIELCC_FAR_MINB
#define BIELCC_FAR_MINB 4
#endif
// The same for the 1-RHS real-k FP64 far kernel: 4 (128 registers) measured
// slower than the compiler's own 168 (5120 triangles x 6001 points 9.6 against
// 7.6 ms).
#ifndef BIELCC_FAR64_MINB
#define BIELCC_FAR64_MINB 0
#endif
#define BIELCC_FAR_BOUNDS(NRHS_, CK_, MIXED_) \
    __launch_bounds__(kFarThreads, NRHS_ == 1 && !CK_ ? (MIXED_ ? BIELCC_FAR_MINB : BIELCC_FAR64_MINB) : 0)
constexpr int kStageCells = 32;  // cells staged at a time: one near-mask word
constexpr int kFarWays = 4;      // warps that share a split's cells on small problems

struct FarArgs {
    const double* pts;
    int n_pts;
    const CellGeo* geo;
    int n_cells;
    const double4* nodes64;
    const float4* nodes32;
    const float* rho32;
    int nn;  // nodes per cell
    FarRules rules;
    const cplx* J;  // [S][N][3]
    int n_rhs, rhs0;
    cplx k;
    double analytic_calc;
    int cells_per_split;  // a multiple of 32, or 16 or 8: a split's cells never straddle near-mask words in part
    int ways;             // 1, or kFarWays: the CTA's warps share the cells, 32 points per CTA
    double* partial;      // [split][S][12][P]
    unsigned* nearmask;   // [ceil(N/32)][P]: bit c%32 of word c/32 set iff (p, c) is near
};
// p_max >= 3, the far kernel's marks-reading variant: the integrals that failed
// the convergence test at the second pass, grad F per pair [ceil(N/32)][P] and
// F . J per RHS [S][ceil(N/32)][P]; take_marked 1 adds the integrals that
// failed (the third pass, at 4 n_start), 0 the ones that passed (which the
// decision kernel adds itself on the field path). (A separate type: the plain variants keep
// FarArgs' parameter block, whose size the FP64 kernel's register allocation
// follows.)
struct FarArgsMarks : FarArgs {
    const unsigned* markG;
    const unsigned* markK;
    int take_marked;
};
template <bool MARKS>
using FarArgsOf = typename std::conditional<MARKS, FarArgsMarks, FarArgs>::type;

// Contract one cell's moments with the RHS currents times the phase P = pr + i pi
// and add into the FP64 accumulators acc[r][12] = (Ex, Ey, Ez, Hx, Hy, Hz) x
// (re, im): E = W J P with W = A1 I + T, H = G x J P. Real k: m holds (S, T/3)
// (farnode.cuh), so W_aa = 2 S - 3 (the other two diagonal entries of T/3) and
// W_ab = 3 (T/3)_ab. sj: the currents of the cell, (re, im) of x, y, z per RHS.
// takeE: bit r adds RHS r's E; takeH: the H of every RHS (convergence-test
// marks, p_max >= 3; all set otherwise).
template <int NRHS, bool CK, typename F>
BIELCC_D void contract(const Moments<F>& m, F pr, F pi, const F (*sj)[6], bool zeroR, double (*acc)[12],
                       unsigned takeE = ~0u, bool takeH = true) {
    const int ti[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    F W[6][2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const F a1 = c ? m.a1i : m.a1r;
        if (CK) {
#pragma unroll
            for (int q = 0; q < 6; q++) W[q][c] = m.t[q][c] + (q == 0 || q == 3 || q == 5 ? a1 : F(0));
        } else {
            const F s2 = a1 + a1;
            W[0][c] = fma(F(-3), m.t[3][c] + m.t[5][c], s2);
            W[3][c] = fma(F(-3), m.t[0][c] + m.t[5][c], s2);
            W[5][c] = fma(F(-3), m.t[0][c] + m.t[3][c], s2);
            W[1][c] = F(3) * m.t[1][c];
            W[2][c] = F(3) * m.t[2][c];
            W[4][c] = F(3) * m.t[4][c];
        }
    }
#pragma unroll
    for (int rr = 0; rr < NRHS; rr++) {
        F jr[3], ji[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const F re = sj[rr][2 * a], im = sj[rr][2 * a + 1];
            jr[a] = re * pr - im * pi;
            ji[a] = re * pi + im * pr;
        }
#pragma unroll
        for (int a = 0; a < 3; a++) {
            F er = 0, ei = 0;
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const F* t = W[ti[a][b]];
                er += t[0] * jr[b] - t[1] * ji[b];
                ei += t[0] * ji[b] + t[1] * jr[b];
            }
            if ((takeE >> rr) & 1u) {
                acc[rr][2 * a] += (double)er;
                acc[rr][2 * a + 1] += (double)ei;
            }
        }
        if (!zeroR && takeH) {
#pragma unroll
            for (int a = 0; a < 3; a++) {
                // (G x J)_a = G_b J_c - G_c J_b, b = a + 1, c = a + 2 (the other way round for -G)
                constexpr int o = !CK && Moments<F>::kNegG ? 2 : 1;
                const int b = (a + o) % 3, c = (a + 3 - o) % 3;
                const F hr = (m.g[b][0] * jr[c] - m.g[b][1] * ji[c]) - (m.g[c][0] * jr[b] - m.g[c][1] * ji[b]);
                const F hi = (m.g[b][0] * ji[c] + m.g[b][1] * jr[c]) - (m.g[c][0] * ji[b] + m.g[c][1] * jr[b]);
                acc[rr][6 + 2 * a] += (double)hr;
                acc[rr][6 + 2 * a + 1] += (double)hi;
            }
        }
    }
}

// The far kernel. MIXED = false: FP64 nodes; true: FP32 nodes. MARKS: the
// convergence-test marks of p_max >= 3 select the integrals this pass adds
// (FarArgs::markG / markK); the other variants read no marks.
// Per cell a warp takes the shortest row that its nearest far point allows
// (rules.cu); lane i loads node i of a chunk of 32 into the warp's buffer, which
// all lanes then walk (a broadcast load per node). The load is issued before the
// pair's set-up, so its latency is covered without a second buffer (a pipelined
// cp.async pair of buffers cost 100 instructions per cell and was slower).
// Bound: issue slots. 8192 cells x 20,000 points, mixed, whole call: 26.0 ms with
// all 64 nodes -> 8.3 with the rules -> 7.2 with the total-degree rules and a
// shorter set-up (near test on the squared distance, e^{ik r0} in turns, phase
// applied to J instead of the moments) -> 6.55 with packed node arithmetic; ncu on
// 8000 points: 804 warp instructions per (warp, cell), 67 % issue-active. FP64,
// 5120 triangles x 6001 points: 11.9 -> 7.6 ms, FP64 pipe 68 %.
// ways = 1: a CTA holds 128 points and every warp takes all cells of the split,
// so that the warps run the same code at about the same time (with each warp at a
// cell of its own the same sums took 10.2 instead of 8.4 ms: 2.0 instead of 0.1
// no-instruction stalls per issue). ways = 4: 32 points per CTA, each warp every
// fourth cell, the warps' sums added in warp order: 80 triangles x 100 points in
// FP64, a whole host call, 1216 -> 240 us.
template <int NRHS, bool CK, bool MIXED, bool MARKS = false>
__global__ void BIELCC_FAR_BOUNDS(NRHS, CK, MIXED) far_kernel(const __grid_constant__ FarArgsOf<MARKS> a) {
    using NodeT = typename std::conditional<MIXED, float4, double4>::type;
    using F = typename std::conditional<MIXED, float, double>::type;
    constexpr int kWarps = kFarThreads / 32;
    static_assert(kWarps == kFarWays, "ways = 4 gives every warp its share of the cells");
    __shared__ __align__(16) RowBuf<NodeT> s_rows[kWarps];
    __shared__ RuleTab<NodeT> s_tab;
    __shared__ double4 s_cell[kStageCells];  // centre xyz, near distance
    __shared__ F s_j[kStageCells][NRHS][6];
    __shared__ int s_mode[kStageCells];  // mixed: phase polynomial; FP64: Taylor length of the phase split, -1 none
    __shared__ float s_rmin[kStageCells][kMaxRules];
    __shared__ unsigned s_near[kWarps][32];
    __shared__ double s_sum[kWarps][12][32];

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool split_cells = a.ways > 1;
    const int p = split_cells ? blockIdx.x * 32 + lane : blockIdx.x * kFarThreads + threadIdx.x;
    const bool live = p < a.n_pts;
    double x[3] = {0., 0., 0.};
    if (live)
        for (int g = 0; g < 3; g++) x[g] = a.pts[3 * (size_t)p + g];
    const int cb = blockIdx.y * a.cells_per_split;  // a stage never crosses a 32-cell mask word
    const int ce = min(a.n_cells, cb + a.cells_per_split);
    const double k2r = a.k.re * a.k.re - a.k.im * a.k.im, k2i = 2.0 * a.k.re * a.k.im;
    const double kturn = a.k.re * kInvTwoPi;
    const int n_lev = a.rules.n_lev;
    if (threadIdx.x == 0) {
        const NodeT* full;
        if constexpr (MIXED) full = a.nodes32;
        else full = a.nodes64;
        s_tab.fill(a.rules, rule_rows(a.rules, NodeT()), full, a.nn, a.n_cells);
    }

    double acc[NRHS][12];
#pragma unroll
    for (int r = 0; r < NRHS; r++)
#pragma unroll
        for (int q = 0; q < 12; q++) acc[r][q] = 0.;

    const KF32 kf = KF32::make(a.k.re, a.k.im);
    // near bits of the stage at c0: a whole word, or the stage's bytes of it when a
    // split is shorter than a word (the split of the last cell clears the rest)
    auto write_mask = [&](int c0, unsigned bits) {
        if (!live || !a.nearmask) return;
        unsigned* word = a.nearmask + (size_t)(c0 >> 5) * a.n_pts + p;
        if (a.cells_per_split >= 32) {
            *word = bits;
        } else {
            const int b0 = (c0 & 31) >> 3, b1 = ce == a.n_cells ? 4 : ((c0 & 31) + a.cells_per_split) >> 3;
            for (int b = b0; b < b1; b++) reinterpret_cast<unsigned char*>(word)[b] = (bits >> (8 * b)) & 0xffu;
        }
    };

    for (int c0 = cb; c0 < ce; c0 += kStageCells) {
        const int nc = min(kStageCells, ce - c0);
        __syncthreads();
        for (int i = threadIdx.x; i < nc; i += kFarThreads) {
            s_cell[i] = near_cell(a.geo[c0 + i], a.analytic_calc);
            if constexpr (MIXED) {
                s_mode[i] = phase_mode((float)fabs(a.k.re) * a.rho32[c0 + i]);
            } else {  // FP64 phase split when the cell's phase range is small (farnode.cuh sincos_taylor64)
                const double th = phase_range64(a.k, (double)a.rho32[c0 + i]);
                s_mode[i] = !(th <= 0.5) ? -1 : (th <= 0.125 ? 2 : (th <= 0.25 ? 1 : 0));
            }
        }
        {
            const RuleK rk = rule_k(a.k);
            const float2* lim = rule_limits(a.rules, NodeT()) + (size_t)c0 * n_lev;
            for (int i = threadIdx.x; i < nc * n_lev; i += kFarThreads)
                s_rmin[i / n_lev][i % n_lev] = CK ? rule_rmin(lim[i], rk) : rule_rmin_real(lim[i], rk);
        }
        for (int i = threadIdx.x; i < nc * NRHS * 6; i += kFarThreads) {
            const int cc = i / (NRHS * 6), rem = i - cc * NRHS * 6, rr = rem / 6, g = rem - rr * 6;
            const int rhs = min(a.rhs0 + rr, a.n_rhs - 1);
            s_j[cc][rr][g] = (F)reinterpret_cast<const double*>(a.J)[((size_t)rhs * a.n_cells + (c0 + cc)) * 6 + g];
        }
        __syncthreads();
        unsigned nbits = 0;  // near bits of this warp's cells
        for (int cc = split_cells ? warp : 0; cc < nc; cc += a.ways) {
            double dx[3], s2;
            const bool nr = near_exact(x, s_cell[cc], dx, &s2);
            bool far = !nr && live;
            nbits |= (nr ? 1u : 0u) << ((c0 + cc) & 31);
            unsigned takeE = ~0u;  // convergence-test marks (p_max >= 3): the RHS whose E this pass adds
            bool takeH = true;     // and whether it adds H
            if constexpr (MARKS) {
                if (far) {  // each integral's convergence test decides which pass adds it
                    const int c = c0 + cc, nw = (a.n_cells + 31) >> 5;
                    const size_t wi = (size_t)(c >> 5) * a.n_pts + p;
                    const bool want = a.take_marked != 0;
                    takeH = (((a.markG[wi] >> (c & 31)) & 1u) != 0) == want;
                    takeE = 0u;
                    for (int rr = 0; rr < NRHS && a.rhs0 + rr < a.n_rhs; rr++) {
                        const unsigned mk = a.markK[(size_t)(a.rhs0 + rr) * nw * a.n_pts + wi];
                        if ((((mk >> (c & 31)) & 1u) != 0) == want) takeE |= 1u << rr;
                    }
                    far = takeE != 0u || takeH;
                }
            }
            const double d = dist_from_sq<!MIXED>(s2);
            const float dmin = warp_min_pos(rule_key(far, d));
            if (!(dmin < __int_as_float(0x7f800000))) continue;  // no lane takes part
            const int lev = rule_level(s_rmin[cc], n_lev, dmin);
            const int cnt = s_tab.cnt[lev];
            const NodeT* row = s_tab.base[lev] + (size_t)(c0 + cc) * cnt;
            NodeT v{};
            if (lane < cnt) v = row[lane];  // on its way during the pair's set-up
            Moments<F> m;
            m.zero();
            PairF32 pf{};
            F P0r = 1, P0i = 0;
            const int mode = s_mode[cc];
            if constexpr (MIXED) {  // the phase taken out of the nodes: e^{ik r0}
                pf.set(dx, s2, d, kf);
                turn_f32(d * kturn, CK ? exp(-a.k.im * d) : 1.0, &P0r, &P0i);
            } else if (mode >= 0) {
                sincos(a.k.re * d, &P0i, &P0r);
                if (CK) {
                    const double am = exp(-a.k.im * d);
                    P0r *= am;
                    P0i *= am;
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
#define BIELCC_NODE_LOOP(MODE_)                                           \
    BIELCC_FAR_UNROLL_PRAGMA for (int i = 0; i < kc; i++)                 \
        far_node_f32<CK, MODE_>(m, pf, rb.get(i), kf);
                    switch (mode) {
                        case 0: BIELCC_NODE_LOOP(0) break;
                        case 1: BIELCC_NODE_LOOP(1) break;
                        case 2: BIELCC_NODE_LOOP(2) break;
                        case 3: BIELCC_NODE_LOOP(3) break;
                        default: BIELCC_NODE_LOOP(4) break;
                    }
#undef BIELCC_NODE_LOOP
                } else if (mode >= 0) {
#define BIELCC_NODE64_LOOP(TD_)                                                                         \
    BIELCC_FAR64_UNROLL_PRAGMA for (int i = 0; i < kc; i++) {                                            \
        const double4 y = rb.get(i);                                                                      \
        far_node_f64<CK, true, TD_>(m, x[0] - y.x, x[1] - y.y, x[2] - y.z, y.w, a.k, k2r, k2i, d);       \
    }
                    switch (mode) {
                        case 2: BIELCC_NODE64_LOOP(2) break;
                        case 1: BIELCC_NODE64_LOOP(1) break;
                        default: BIELCC_NODE64_LOOP(0) break;
                    }
#undef BIELCC_NODE64_LOOP
                } else {
#pragma unroll 2
                    for (int i = 0; i < kc; i++) {
                        const double4 y = rb.get(i);
                        far_node_f64<CK, false>(m, x[0] - y.x, x[1] - y.y, x[2] - y.z, y.w, a.k, k2r, k2i, d);
                    }
                }
            }
            if (far) {
                const bool zeroR = d < kMachineZero;  // R_Rot_Colloc: R = 0 at the cell centre
                contract<NRHS, CK, F>(m, P0r, P0i, s_j[cc], zeroR, acc, takeE, takeH);
            }
        }
        if (split_cells) {
            s_near[warp][lane] = nbits;
            __syncthreads();
            if (warp == 0) {
#pragma unroll
                for (int w = 1; w < kWarps; w++) nbits |= s_near[w][lane];
                write_mask(c0, nbits);
            }
        } else {
            write_mask(c0, nbits);
        }
    }
    const size_t P = a.n_pts;
#pragma unroll
    for (int r = 0; r < NRHS; r++) {
        if (a.rhs0 + r >= a.n_rhs) break;
        double* dst = a.partial + (((size_t)blockIdx.y * a.n_rhs + (a.rhs0 + r)) * 12) * P + p;
        if (!split_cells) {
            if (live) {
#pragma unroll
                for (int q = 0; q < 12; q++) dst[(size_t)q * P] = acc[r][q];
            }
            continue;
        }
        // the warps' sums in warp order: warp w adds components 3 w .. 3 w + 2
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 12; q++) s_sum[warp][q][lane] = acc[r][q];
        __syncthreads();
        if (live) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const int q = 3 * warp + j;
                double v = s_sum[0][q][lane];
#pragma unroll
                for (int w = 1; w < kWarps; w++) v += s_sum[w][q][lane];
                dst[(size_t)q * P] = v;
            }
        }
    }
}

// ---------------------------------------------------------------- adaptive far pairs (p_max >= 3)
// The reference's loop (integral_universal.h:58-119) stops at the first pass
// after the first whose squared L2 change is below eps^2, else returns its last
// pass. far_refine_decide_kernel runs that test between the passes at n_start
// and 2 n_start for every far pair, from node tables: K_RotRot_Far's integral
// of F_RotRotSimplePot_H . J for every right-hand side (K.h:288-301) and
// R_Rot_Colloc's integral of grad F (R.h:89-111; none at the cell centre).
// Each integral is tested on its own, as the reference runs one loop per
// integral: an integral that passes returns the pass at 2 n_start, which the
// decision kernel has just run for the test and adds to the split sums itself
// (in FP64, in the mixed form too); one that fails is marked (markG per pair,
// markK per pair and RHS) and takes the pass at 4 n_start when p_max = 3
// (far_kernel with take_marked = 1 on those tables), else the whole loop in
// far_refine_sum_kernel.

// Unrolling of the decision kernel's node loops (the node rows come from
// global memory: unrolled, their loads issue ahead of the arithmetic). 3200 cells
// x 1000 points at p_max = 3, FP64, whole call: x1 13.7, x3 11.3, x5 12.2 ms.
#ifndef BIELCC_DECIDE_UNROLL
#define BIELCC_DECIDE_UNROLL 3
#endif

// One pass of the FP64 far node loop over a cell's node table row (far_kernel's
// FP64 arithmetic: the phase split below |k| rho = 0.5, else sincos per node).
template <bool CK>
BIELCC_D void far_pass_f64(Moments<double>& m, const double4* __restrict__ nd, int nn, const double* x, cplx k,
                           double k2r, double k2i, double r0, bool split, int td) {
    m.zero();
    if (split) {
#define BIELCC_PASS64(TD_)                                                                              \
    BIELCC_FAR_PRAGMA(BIELCC_DECIDE_UNROLL) for (int i = 0; i < nn; i++) {                              \
        const double4 v = ldg_node(nd + i);                                                             \
        far_node_f64<CK, true, TD_>(m, x[0] - v.x, x[1] - v.y, x[2] - v.z, v.w, k, k2r, k2i, r0);       \
    }
        switch (td) {
            case 2: BIELCC_PASS64(2) break;
            case 1: BIELCC_PASS64(1) break;
            default: BIELCC_PASS64(0) break;
        }
#undef BIELCC_PASS64
    } else {
        BIELCC_FAR_PRAGMA(BIELCC_DECIDE_UNROLL) for (int i = 0; i < nn; i++) {
            const double4 v = ldg_node(nd + i);
            far_node_f64<CK, false>(m, x[0] - v.x, x[1] - v.y, x[2] - v.z, v.w, k, k2r, k2i, r0);
        }
    }
    if (!CK) m.finish_real_k();
}

// Raw integrals of one pass (before the 1/4pi of K_RotRot_Far / R_Rot_Colloc),
// times the phase P: K = A1 J + T J, G = grad F.
BIELCC_D void far_raw_K(const Moments<double>& m, double pr, double pi, const cplx* j, cplx* K) {
    const int ti[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    for (int a = 0; a < 3; a++) {
        cplx e = mk(m.a1r, m.a1i) * j[a];
        for (int b = 0; b < 3; b++) e = e + mk(m.t[ti[a][b]][0], m.t[ti[a][b]][1]) * j[b];
        K[a] = e * mk(pr, pi);
    }
}

// The reference's squared change: sum of |res - prev|^2 with |.| taken first
// (integral_universal.h:96-99).
BIELCC_D double far_delta2(const cplx* a, const cplx* b) {
    double d = 0.;
    for (int g = 0; g < 3; g++) {
        const double t = sqrt(cabs2(a[g] - b[g]));
        d += t * t;
    }
    return d;
}

// markK and this split's slot of a.partial must be zero on entry (set bits
// only; the passing integrals are added); markG is written in full. Each pass
// takes the shortest row its table's rules allow (rules.cu, FP64 limits).
__global__ void far_refine_decide_kernel(const __grid_constant__ FarArgs a, const __grid_constant__ FarRules rules_lo,
                                         const double4* __restrict__ lo, int nn_lo, double eps2,
                                         unsigned* __restrict__ markG, unsigned* __restrict__ markK) {
    __shared__ RuleTab<double4> s_lo, s_hi;
    __shared__ float s_rmin[2][kStageCells][kMaxRules];
    const int p = blockIdx.x * kFarThreads + threadIdx.x;
    const bool live = p < a.n_pts;
    double x[3] = {0., 0., 0.};
    if (live)
        for (int g = 0; g < 3; g++) x[g] = a.pts[3 * (size_t)p + g];
    const int cb = blockIdx.y * a.cells_per_split;  // a multiple of 32
    const int ce = min(a.n_cells, cb + a.cells_per_split);
    const bool ck = a.k.im != 0.0;
    const double k2r = a.k.re * a.k.re - a.k.im * a.k.im, k2i = 2.0 * a.k.re * a.k.im;
    const int nw = (a.n_cells + 31) >> 5;
    const size_t P = a.n_pts;
    const int nlo = rules_lo.n_lev, nhi = a.rules.n_lev;
    if (threadIdx.x == 0) {
        s_lo.fill(rules_lo, rules_lo.n64, lo, nn_lo, a.n_cells);
        s_hi.fill(a.rules, a.rules.n64, a.nodes64, a.nn, a.n_cells);
    }
    unsigned nbits = 0, gbits = 0;
    for (int c = cb; c < ce; c++) {
        if ((c & 31) == 0) {
            const int nc = min(kStageCells, ce - c);
            const RuleK rk = rule_k(a.k);
            __syncthreads();  // the previous cells' limits are no longer read
            for (int i = threadIdx.x; i < nc * nlo; i += kFarThreads)
                s_rmin[0][i / nlo][i % nlo] = rule_rmin(rules_lo.thr64[(size_t)c * nlo + i], rk);
            for (int i = threadIdx.x; i < nc * nhi; i += kFarThreads)
                s_rmin[1][i / nhi][i % nhi] = rule_rmin(a.rules.thr64[(size_t)c * nhi + i], rk);
            __syncthreads();
        }
        const CellGeo& gg = a.geo[c];
        double d;
        const bool nr = is_near(x, gg.c, gg.diam, a.analytic_calc, &d);
        bool gfail = false;
        const bool far = !nr && live;
        const float dmin = warp_min_pos(rule_key(far, d));
        const int llo = rule_level(s_rmin[0][c & 31], nlo, dmin), lhi = rule_level(s_rmin[1][c & 31], nhi, dmin);
        if (far) {
            const int n_lo = s_lo.cnt[llo], n_hi = s_hi.cnt[lhi];
            const double4* row_lo = s_lo.base[llo] + (size_t)c * n_lo;
            const double4* row_hi = s_hi.base[lhi] + (size_t)c * n_hi;
            const double th64 = fabs(a.k.re) * (double)a.rho32[c] * (1.0 + 1e-6);
            const bool split = !ck && th64 <= 0.5;
            const int td = th64 <= 0.125 ? 2 : (th64 <= 0.25 ? 1 : 0);
            double pr = 1.0, pi = 0.0;
            if (split) sincos(a.k.re * d, &pi, &pr);
            Moments<double> m0, m1;
            if (ck) {
                far_pass_f64<true>(m0, row_lo, n_lo, x, a.k, k2r, k2i, d, false, 0);
                far_pass_f64<true>(m1, row_hi, n_hi, x, a.k, k2r, k2i, d, false, 0);
            } else {
                far_pass_f64<false>(m0, row_lo, n_lo, x, a.k, k2r, k2i, d, split, td);
                far_pass_f64<false>(m1, row_hi, n_hi, x, a.k, k2r, k2i, d, split, td);
            }
            const bool zeroR = d < kMachineZero;  // R_Rot_Colloc integrates grad F away from the centre only
            cplx g1[3];
            if (!zeroR) {
                cplx g0[3];
                for (int q = 0; q < 3; q++) {
                    g0[q] = mk(m0.g[q][0], m0.g[q][1]) * mk(pr, pi);
                    g1[q] = mk(m1.g[q][0], m1.g[q][1]) * mk(pr, pi);
                }
                gfail = !(far_delta2(g1, g0) < eps2);
            }
            for (int s = 0; s < a.n_rhs; s++) {
                const cplx* j = a.J + ((size_t)s * a.n_cells + c) * 3;
                const cplx jj[3] = {j[0], j[1], j[2]};
                cplx k0[3], k1[3];
                far_raw_K(m0, pr, pi, jj, k0);
                far_raw_K(m1, pr, pi, jj, k1);
                const bool kfail = !(far_delta2(k1, k0) < eps2);
                if (kfail) atomicOr(markK + ((size_t)s * nw + (c >> 5)) * a.n_pts + p, 1u << (c & 31));
                // the integrals that passed return the pass at 2 n_start: added
                // here, in cell order, to this split's raw sums (the thread owns them)
                double* dst = a.partial + ((size_t)blockIdx.y * a.n_rhs + s) * 12 * P + p;
                if (!kfail)
                    for (int q = 0; q < 3; q++) {
                        dst[(size_t)(2 * q) * P] += k1[q].re;
                        dst[(size_t)(2 * q + 1) * P] += k1[q].im;
                    }
                if (!zeroR && !gfail)
                    for (int q = 0; q < 3; q++) {  // (G x J)_q = G_b J_c - G_c J_b
                        const int b = (q + 1) % 3, cc = (q + 2) % 3;
                        const cplx h = g1[b] * jj[cc] - g1[cc] * jj[b];
                        dst[(size_t)(6 + 2 * q) * P] += h.re;
                        dst[(size_t)(6 + 2 * q + 1) * P] += h.im;
                    }
            }
        }
        nbits |= (nr ? 1u : 0u) << (c & 31);
        gbits |= (gfail ? 1u : 0u) << (c & 31);
        if ((c & 31) == 31 || c == ce - 1) {
            if (live) {
                if (a.nearmask) a.nearmask[(size_t)(c >> 5) * a.n_pts + p] = nbits;
                markG[(size_t)(c >> 5) * a.n_pts + p] = gbits;
            }
            nbits = gbits = 0;
        }
    }
}

// p_max > 3: the integrals that failed the test, through the whole loop
// (integral_cell, ops.cuh: the reference's passes, test and budget), one warp
// per (point, RHS, range of mask words): F . J where markK is set, grad F where
// markG is set. In round r lane l takes the range's marked cell of rank
// 32 r + l (cell order; each lane walks the mask words with its own cursor), so
// the lanes run their loops side by side; lane sums are in cell order and
// combined by a fixed xor butterfly. The marked cells gather on the few
// near-field points, so gridDim.z ranges per point give the GPU that many more
// warps. Writes the raw E, H sums (before 1/4pi) of every point and range,
// zero without marked cells, into partial-sum slot blockIdx.z of `out`
// [gridDim.z][S][12][P].
__global__ void far_refine_sum_kernel(FarArgs a, const unsigned* __restrict__ markG, const unsigned* __restrict__ markK,
                                      const double* __restrict__ verts, int nv, DNP np, double* __restrict__ out) {
    const int p = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    const int s = blockIdx.y;
    if (p >= a.n_pts) return;  // whole warps
    const size_t P = a.n_pts;
    const int n_words = (a.n_cells + 31) / 32;
    // this warp's range of mask words (blockIdx.z of gridDim.z parts) and output slot
    const int wpp = (n_words + gridDim.z - 1) / gridDim.z;
    const int w_end = min(n_words, (int)(blockIdx.z + 1) * wpp);
    out += (size_t)blockIdx.z * a.n_rhs * 12 * P;
    const unsigned* mK = markK + (size_t)s * n_words * P;
    const double x[3] = {a.pts[3 * (size_t)p], a.pts[3 * (size_t)p + 1], a.pts[3 * (size_t)p + 2]};
    double v[12];
#pragma unroll
    for (int q = 0; q < 12; q++) v[q] = 0.;
    int w = blockIdx.z * wpp;
    unsigned bits = w < w_end ? (markG[(size_t)w * P + p] | mK[(size_t)w * P + p]) : 0u;
    long long base = 0;  // rank (within the range) of the first flagged cell of word w
    for (long long t = lane;; t += 32) {
        while (w < w_end && base + __popc(bits) <= t) {
            base += __popc(bits);
            w++;
            bits = w < w_end ? (markG[(size_t)w * P + p] | mK[(size_t)w * P + p]) : 0u;
        }
        const bool have = w < w_end;
        if (!__any_sync(0xffffffffu, have)) break;
        if (!have) continue;
        unsigned b = bits;
        for (long long r = base; r < t; r++) b &= b - 1;  // drop the lower-ranked cells of the word
        const int c = w * 32 + __ffs(b) - 1;
        const bool doK = (mK[(size_t)w * P + p] >> (c & 31)) & 1u, doG = (markG[(size_t)w * P + p] >> (c & 31)) & 1u;
        DCell cl;
        cl.nv = nv;
        for (int vv = 0; vv < nv; vv++)
            for (int g = 0; g < 3; g++) cl.v[vv][g] = verts[((size_t)c * nv + vv) * 3 + g];
        const cplx* j = a.J + ((size_t)s * a.n_cells + c) * 3;
        DKP kp;
        dkp_zero(kp);
        kp.smoothR = kMachineZero;
        kp.smoothRMin = kMachineZero;
        kp.k = a.k;
        for (int g = 0; g < 3; g++) kp.current[g] = j[g];
        if (doK) {
            cplx K[3];
            integral_cell<cplx>(F_ROTROTSIMPLEPOT_H, x, cl, kp, 3, np.n_start, np.p_max, np.eps, K);
            for (int g = 0; g < 3; g++) {
                v[2 * g] += K[g].re;
                v[2 * g + 1] += K[g].im;
            }
        }
        double d;
        is_near(x, a.geo[c].c, a.geo[c].diam, a.analytic_calc, &d);
        if (doG && !(d < kMachineZero)) {  // R_Rot_Colloc: 0 at the cell centre
            DKP kr;
            dkp_zero(kr);
            kr.smoothR = kMachineZero;
            kr.smoothRMin = kMachineZero;
            kr.k = a.k;
            cplx G[3], h[3], jj[3] = {j[0], j[1], j[2]};
            integral_cell<cplx>(F_GRADSIMPLEPOT_H, x, cl, kr, 3, np.n_start, np.p_max, np.eps, G);
            ccross_cc(G, jj, h);
            for (int g = 0; g < 3; g++) {
                v[6 + 2 * g] += h[g].re;
                v[7 + 2 * g] += h[g].im;
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int q = 0; q < 12; q++) v[q] += __shfl_xor_sync(0xffffffffu, v[q], off);
    if (lane < 12) {
        double r = v[0];
#pragma unroll
        for (int q = 1; q < 12; q++)
            if (lane == q) r = v[q];
        out[((size_t)s * 12 + lane) * P + p] = r;
    }
}

// ---------------------------------------------------------------- near classification
// The far kernels record, per point, which cells failed the far test
// (get_field.h:58) in a bit mask; these two kernels turn it into per-point
// counts and the cell lists in ascending cell order.
__global__ void near_count_kernel(const unsigned* __restrict__ mask, int n_words, int n_pts,
                                  long long* __restrict__ counts) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_pts) return;
    long long n = 0;
    for (int w = 0; w < n_words; w++) n += __popc(mask[(size_t)w * n_pts + p]);
    counts[p] = n;
}

// Near list of a point in ascending cell order: one warp per point. Lane l
// takes a contiguous run of the point's mask words, counts its bits, and
// writes its cells after those of the lanes before it (warp prefix sum), so a
// point with hundreds of near cells does not run 256 words in one thread.
__global__ void near_fill_kernel(const unsigned* __restrict__ mask, int n_words, int n_pts,
                                 const long long* __restrict__ offs, int* __restrict__ pair_cell,
                                 int* __restrict__ pair_pt) {
    const int p = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (p >= n_pts) return;  // whole warps
    const long long o0 = offs[p];
    if (offs[p + 1] == o0) return;
    const int run = (n_words + 31) / 32, w0 = min(n_words, lane * run), w1 = min(n_words, w0 + run);
    int cnt = 0;
    for (int w = w0; w < w1; w++) cnt += __popc(mask[(size_t)w * n_pts + p]);
    int incl = cnt;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += t;
    }
    long long o = o0 + (incl - cnt);
    for (int w = w0; w < w1; w++) {
        unsigned b = mask[(size_t)w * n_pts + p];
        while (b) {
            const int bit = __ffs(b) - 1;
            b &= b - 1;
            pair_cell[o] = w * 32 + bit;
            pair_pt[o] = p;
            o++;
        }
    }
}

// Near pair: the J-independent parts of K_RotRot_Near_Smooth and R_Rot_Smooth
// (near_pair_moments, ops.cuh), one pair per group of G lanes.
template <int G>
__global__ void near_pair_kernel(const double* __restrict__ pts, const double* __restrict__ verts, int nv,
                                 const int* __restrict__ pair_cell, const int* __restrict__ pair_pt, long long n_pairs,
                                 cplx k, DNP np, cplx* __restrict__ out) {
    const Lanes<G> g = Lanes<G>::make();
    const long long q = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G;
    if (q >= n_pairs) return;  // whole groups
    int c = pair_cell[q], p = pair_pt[q];
    DCell cl;
    cl.nv = nv;
    for (int v = 0; v < nv; v++)
        for (int h = 0; h < 3; h++) cl.v[v][h] = verts[((size_t)c * nv + v) * 3 + h];
    double x[3] = {pts[3 * (size_t)p], pts[3 * (size_t)p + 1], pts[3 * (size_t)p + 2]};
    near_pair_moments<G>(g, x, cl, k, np, out + q * 13);
}

// Near pairs of a point contracted with one RHS: one warp per (point, RHS).
// Lane l takes the point's pairs l, l + 32, ... (cell order) and sums them in
// order; the 32 lane sums are combined by a fixed xor butterfly. The order depends
// only on the point's own pair list, and a point with hundreds of near cells (small
// cells near a pole) does not hold up a whole point tile in one thread. (The pairs'
// moments themselves are summed by 1, 8 or 32 lanes by the call's number of near
// pairs: near_lanes.) near[s][12][p] = E, H (re, im), already / 4pi.
__global__ void near_sum_kernel(const long long* __restrict__ offs, const int* __restrict__ pair_cell,
                                const cplx* __restrict__ moments, const cplx* __restrict__ J, int n_pts, int n_cells,
                                double* __restrict__ near) {
    const int p = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    const int s = blockIdx.y;
    if (p >= n_pts) return;  // whole warps
    const long long q0 = offs[p], q1 = offs[p + 1];
    if (q0 == q1) return;
    double v[12];
#pragma unroll
    for (int i = 0; i < 12; i++) v[i] = 0.;
    for (long long q = q0 + lane; q < q1; q += 32) {
        const int c = pair_cell[q];
        const cplx* o = moments + q * 13;
        const cplx* j = J + ((size_t)s * n_cells + c) * 3;
#pragma unroll
        for (int g = 0; g < 3; g++) {
            const cplx kv = o[0] * j[g] + o[1 + 3 * g] * j[0] + o[2 + 3 * g] * j[1] + o[3 + 3 * g] * j[2];
            v[2 * g] += kv.re;
            v[2 * g + 1] += kv.im;
        }
        cplx h[3];
        ccross_cc(o + 10, j, h);
#pragma unroll
        for (int g = 0; g < 3; g++) {
            v[6 + 2 * g] += h[g].re;
            v[7 + 2 * g] += h[g].im;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int i = 0; i < 12; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i], off);
    if (lane < 12) {
        double x = v[0];
#pragma unroll
        for (int i = 1; i < 12; i++)
            if (lane == i) x = v[i];
        near[((size_t)s * 12 + lane) * n_pts + p] = x;
    }
}

struct FinalArgs {
    const double* pts;
    int n_pts, n_rhs, n_cells, splits;
    const double* partial;
    const long long* offs;  // near-pair offsets per point, or null without near pairs
    const double* near;     // near_sum_kernel's sums
    cplx mult;
    double kvec[3], e0[3], h_scale;
    int add_E, add_H;
    double* E;
    double* H;
    unsigned long long* nonfinite;
};

// Per (point, RHS): far partials over the splits (in split order), near sum, mult,
// incident field. A CTA takes 32 points: warp q sums component q (12 of them) of its
// lanes' points, eight splits' loads in flight at a time, then warp 0 finishes E
// and warp 1 H. With one thread per point all 12 components' loads of a split had to
// return before the next split's were issued: 100 points x 10 splits 27 us, 3001 x 4
// right-hand sides 75 us; with a warp per point and lanes over the splits every
// 8-byte load fetched a sector of its own.
constexpr int kFinalThreads = 12 * 32;
__global__ void __launch_bounds__(kFinalThreads) finalize_kernel(const __grid_constant__ FinalArgs a) {
    __shared__ double s_v[12][32];
    __shared__ int s_bad[32];
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5, s = blockIdx.y;
    const int p = blockIdx.x * 32 + lane;
    const size_t P = a.n_pts;
    if (p < a.n_pts) {
        const double* src = a.partial + ((size_t)s * 12 + q) * P + p;
        const size_t step = (size_t)a.n_rhs * 12 * P;
        double v = 0.;
#pragma unroll 8
        for (int sp = 0; sp < a.splits; sp++) v += src[sp * step];
        s_v[q][lane] = v;
    }
    __syncthreads();
    bool bad = false;
    if (q < 2 && p < a.n_pts) {  // warp 0: E, warp 1: H
        cplx F[3];
        for (int g = 0; g < 3; g++) F[g] = mk(s_v[6 * q + 2 * g][lane], s_v[6 * q + 2 * g + 1][lane]) * kInvFourPi;
        if (a.offs && a.offs[p + 1] > a.offs[p]) {
            const double* nv = a.near + ((size_t)s * 12 + 6 * q) * P + p;
            for (int g = 0; g < 3; g++) F[g] += mk(nv[(size_t)(2 * g) * P], nv[(size_t)(2 * g + 1) * P]);
        }
        if (q == 0)
            for (int g = 0; g < 3; g++) F[g] = F[g] * a.mult;
        if (q == 0 ? a.add_E : a.add_H) {
            const double* x = a.pts + 3 * (size_t)p;
            double sn, cs, f[3];
            sincos(a.kvec[0] * x[0] + a.kvec[1] * x[1] + a.kvec[2] * x[2], &sn, &cs);
            if (q == 0) {
                for (int g = 0; g < 3; g++) F[g] += mk(a.e0[g] * cs, a.e0[g] * sn);
            } else {
                cross3(a.kvec, a.e0, f);
                for (int g = 0; g < 3; g++) F[g] += mk(f[g] * cs * a.h_scale, f[g] * sn * a.h_scale);
            }
        }
        double* out = q == 0 ? a.E : a.H;
        if (out) {
            cplx* o = reinterpret_cast<cplx*>(out) + ((size_t)s * P + p) * 3;
            for (int g = 0; g < 3; g++) {
                o[g] = F[g];
                bad |= !isfinite(F[g].re) || !isfinite(F[g].im);
            }
        }
    }
    if (!a.nonfinite) return;
    if (q == 1) s_bad[lane] = bad;
    __syncthreads();
    if (q == 0 && (bad || s_bad[lane])) atomicAdd(a.nonfinite, 1ull);  // once per (point, RHS)
}

// ---------------------------------------------------------------- host launchers
static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }
static size_t mask_words(int n_cells) { return (size_t)(n_cells + 31) / 32; }
// Mask-word ranges per point of far_refine_sum_kernel (p_max > 3).
static int refine_parts(const FieldLaunch& f) {
    return (int)std::min<size_t>(8, std::max<size_t>(1, mask_words(f.mesh->n_cells)));
}
// Partial-sum slots [slot][S][12][P]: one per cell split; with p_max = 3 as
// many again for the third pass of the pairs that fail the convergence test;
// with p_max > 3 one per mask-word range of the pairs that take the whole
// refinement loop.
static int partial_slots(const FieldLaunch& f, int splits) {
    return splits + (far_third_pass(f.np) ? splits : (far_adaptive(f.np) ? refine_parts(f) : 0));
}
// Resident CTAs (whole GPU) of the far-kernel variant a launch starts with:
// NRHS 4 / 2 / 1 (the first RHS chunk), real / complex k, FP64 / mixed.
static int far_slots(int n_rhs, bool ck, bool mixed) {
    static std::atomic<int> cache[2][3][2];
    const int ri = n_rhs >= 4 ? 0 : (n_rhs >= 2 ? 1 : 2);
    std::atomic<int>& c = cache[ck][ri][mixed];
    int v = c.load(std::memory_order_relaxed);
    if (v) return v;
    int dev = 0, sms = 148, per = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const void* fn;
#define BIELCC_FK(R, C, M) (const void*)far_kernel<R, C, M>
    if (ri == 0) fn = ck ? (mixed ? BIELCC_FK(4, true, true) : BIELCC_FK(4, true, false))
                              : (mixed ? BIELCC_FK(4, false, true) : BIELCC_FK(4, false, false));
    else if (ri == 1) fn = ck ? (mixed ? BIELCC_FK(2, true, true) : BIELCC_FK(2, true, false))
                              : (mixed ? BIELCC_FK(2, false, true) : BIELCC_FK(2, false, false));
    else fn = ck ? (mixed ? BIELCC_FK(1, true, true) : BIELCC_FK(1, true, false))
                 : (mixed ? BIELCC_FK(1, false, true) : BIELCC_FK(1, false, false));
#undef BIELCC_FK
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, kFarThreads, 0);
    v = std::max(1, sms * std::max(1, per));
    c.store(v, std::memory_order_relaxed);
    return v;
}

// Cells per split of the far kernel: whole 32-cell mask words, or 16 or 8 cells
// (bytes of a word) when the splits outnumber the words.
static int far_cells_per_split(int n_cells, int splits) {
    if (splits > (n_cells + 31) / 32) return (n_cells + 15) / 16 == splits ? 16 : 8;
    return round_cells_per_split(n_cells, splits);
}

// The far kernel's grid. 128-point tiles with whole-warp cell sweeps when they
// fill the GPU at one mask word (32 cells) per split, the finest a sweep can be
// cut; below that a resident CTA slot would stay empty, so 32-point tiles whose
// warps share the cells, and if that is still short 16 or 8 cells per split (the
// decision kernel of p_max >= 3 keeps whole words).
struct FarGrid {
    int tiles, splits, ways;
};
static FarGrid far_grid(const FieldLaunch& f, int max_splits) {
    const int N = f.mesh->n_cells, slots = far_slots(f.n_rhs, f.k.im != 0.0, f.precision == 1);
    FarGrid g;
    g.tiles = (f.n_pts + kFarThreads - 1) / kFarThreads;
    g.ways = (size_t)g.tiles * std::min((N + 31) / 32, max_splits) < (size_t)slots ? kFarWays : 1;
    if (g.ways > 1) g.tiles = (f.n_pts + 31) / 32;
    g.splits = choose_cell_splits(g.tiles, N, slots, max_splits);
    if (g.ways > 1 && !far_adaptive(f.np))
        for (int cps = 16; cps >= 8 && g.splits >= N / 32 && (size_t)g.tiles * g.splits < (size_t)slots; cps -= 8) {
            const int fine = (N + cps - 1) / cps;
            if (fine > max_splits) break;
            if (fine > (N + 31) / 32) g.splits = fine;
        }
    return g;
}

size_t field_ws_base_bytes(const FieldLaunch& f, int* splits_out, size_t partial_cap) {
    const int N = f.mesh->n_cells;
    const size_t P = f.n_pts;
    const size_t per_split = (size_t)f.n_rhs * 12 * P * sizeof(double);
    const int max_splits = (int)std::max<size_t>(1, partial_cap / std::max<size_t>(1, per_split));
    int splits = far_grid(f, max_splits).splits;
    if (far_third_pass(f.np)) {
        // p_max = 3: the third pass's work sits on the points whose integrals
        // failed the test (near-field points, a few tiles), so a grid balanced
        // for the plain far kernel leaves most SMs idle. Cells split as finely
        // as the near mask allows (32 per split), within partial_cap for both
        // slot sets: 2000 x 8192 cells, FP64 94.6 -> 78.0 ms, mixed 61.8 -> 53.7 ms.
        const int want = (int)std::min<size_t>((N + 31) / 32, partial_cap / std::max<size_t>(1, 2 * per_split));
        if (want > splits) {
            const int cps = round_cells_per_split(N, want);
            splits = (N + cps - 1) / cps;
        }
    }
    *splits_out = splits;
    return align256((size_t)partial_slots(f, splits) * per_split) + 2 * align256((P + 1) * sizeof(long long)) +
           align256(sizeof(long long)) + align256(mask_words(N) * P * sizeof(unsigned)) +
           align256((size_t)f.n_rhs * 12 * P * sizeof(double)) +
           (far_adaptive(f.np) ? align256((size_t)(1 + f.n_rhs) * mask_words(N) * P * sizeof(unsigned)) : 0);
}

template <int NRHS, bool CK, bool MIXED>
static void launch_far_t(const FarArgs& a, int tiles, int splits, cudaStream_t s) {
    far_kernel<NRHS, CK, MIXED><<<dim3(tiles, splits), kFarThreads, 0, s>>>(a);
}

// p_max >= 3: one RHS per launch of the marks-reading variant.
template <bool CK, bool MIXED>
static int launch_far_marks(FarArgsMarks a, int tiles, int splits, cudaStream_t s) {
    for (int r = 0; r < a.n_rhs; r++) {
        a.rhs0 = r;
        far_kernel<1, CK, MIXED, true><<<dim3(tiles, splits), kFarThreads, 0, s>>>(a);
    }
    return a.n_rhs;
}

template <bool CK, bool MIXED>
static int launch_far_rhs(FarArgs a, int tiles, int splits, cudaStream_t s) {
    int n = 0;
    for (int r0 = 0; r0 < a.n_rhs; n++) {
        a.rhs0 = r0;
        int left = a.n_rhs - r0;
        if (left >= 4) { launch_far_t<4, CK, MIXED>(a, tiles, splits, s); r0 += 4; }
        else if (left >= 2) { launch_far_t<2, CK, MIXED>(a, tiles, splits, s); r0 += 2; }
        else { launch_far_t<1, CK, MIXED>(a, tiles, splits, s); r0 += 1; }
    }
    return n;
}

cudaError_t field_stage1(const FieldLaunch& f, void* ws, int splits, long long* d_total, cudaStream_t s,
                         int* launches, cudaEvent_t far_begin, cudaEvent_t far_end, int* far_launches) {
    const MeshDev& m = *f.mesh;
    const size_t P = f.n_pts;
    char* w = (char*)ws;
    double* partial = (double*)w;
    w += align256((size_t)partial_slots(f, splits) * f.n_rhs * 12 * P * sizeof(double));
    long long* counts = (long long*)w;
    w += align256((P + 1) * sizeof(long long));
    long long* offs = (long long*)w;
    w += align256((P + 1) * sizeof(long long)) + align256(sizeof(long long));
    unsigned* mask = (unsigned*)w;
    const int n_words = (int)mask_words(m.n_cells);
    w += align256(mask_words(m.n_cells) * P * sizeof(unsigned)) + align256((size_t)f.n_rhs * 12 * P * sizeof(double));
    // p_max >= 3, after the near sums: the marks of grad F, then of F . J per RHS
    unsigned* markG = far_adaptive(f.np) ? (unsigned*)w : nullptr;
    unsigned* markK = markG ? markG + mask_words(m.n_cells) * P : nullptr;

    FarArgs a;
    a.pts = f.pts;
    a.n_pts = f.n_pts;
    a.geo = m.geo;
    a.n_cells = m.n_cells;
    a.nodes64 = m.nodes64;
    a.nodes32 = m.nodes32;
    a.rho32 = m.rho32;
    // the decision kernel of p_max >= 3 reads FP64 rows in the mixed form too
    a.rules = rules_read(m.rules, f.precision != 1 || far_adaptive(f.np));
    a.nn = far_split_n(f.np) * far_split_n(f.np);
    a.J = reinterpret_cast<const cplx*>(f.J);
    a.n_rhs = f.n_rhs;
    a.rhs0 = 0;
    a.k = f.k;
    a.analytic_calc = f.np.analytic_calc;
    a.cells_per_split = far_cells_per_split(m.n_cells, splits);
    a.partial = partial;
    a.nearmask = mask;
    const int tiles128 = (f.n_pts + kFarThreads - 1) / kFarThreads;  // one point per thread
    // the split count is the caller's; fewer 128-point CTAs than slots: shared cells
    a.ways = (size_t)tiles128 * std::min(n_words, splits) < (size_t)far_slots(f.n_rhs, f.k.im != 0.0, f.precision == 1) ? kFarWays : 1;
    const int tiles = a.ways > 1 ? (f.n_pts + 31) / 32 : tiles128;
    bool ck = f.k.im != 0.0;
    bool mixed = f.precision == 1;
    int nl = 0;
    if (tiles > 0 && m.table_n != far_split_n(f.np))
        return cudaErrorInvalidValue;  // node tables of another split: the caller builds far_split_n's
    if (tiles > 0 && far_adaptive(f.np) && (m.table_lo_n != f.np.n_start || !m.nodes64_lo))
        return cudaErrorInvalidValue;  // no n_start table for the convergence test
    if (tiles > 0 && far_third_pass(f.np) && (m.table_hi_n != 4 * f.np.n_start || !m.nodes64_hi))
        return cudaErrorInvalidValue;  // no 4 n_start tables for the third pass
    if (far_begin) cudaEventRecord(far_begin, s);
    if (tiles > 0 && far_adaptive(f.np)) {
        // the convergence test of every far pair's integrals; the failing ones
        // are marked, the passing ones added to the split sums (slots [0, splits))
        cudaError_t e = cudaMemsetAsync(markK, 0, (size_t)f.n_rhs * n_words * P * sizeof(unsigned), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(partial, 0, (size_t)splits * f.n_rhs * 12 * P * sizeof(double), s);
        if (e != cudaSuccess) return e;
        const int nn_lo = f.np.n_start * f.np.n_start;
        far_refine_decide_kernel<<<dim3(tiles128, splits), kFarThreads, 0, s>>>(
            a, rules_read(m.rules_lo, true), m.nodes64_lo, nn_lo, f.np.eps * f.np.eps, markG, markK);
        nl++;
    }
    FarArgsMarks am;
    static_cast<FarArgs&>(am) = a;
    am.markG = markG;
    am.markK = markK;
    if (tiles > 0 && !markG) {
        if (mixed) nl += ck ? launch_far_rhs<true, true>(a, tiles, splits, s) : launch_far_rhs<false, true>(a, tiles, splits, s);
        else nl += ck ? launch_far_rhs<true, false>(a, tiles, splits, s) : launch_far_rhs<false, false>(a, tiles, splits, s);
    }
    if (tiles > 0 && far_third_pass(f.np)) {
        // p_max = 3: the marked pairs return the third pass, at 4 n_start, into
        // their own partial slots
        FarArgsMarks a3 = am;
        a3.nodes64 = m.nodes64_hi;
        a3.nodes32 = m.nodes32_hi;
        a3.rho32 = m.rho32_hi;
        a3.rules = rules_read(m.rules_hi, !mixed);
        a3.nn = 16 * f.np.n_start * f.np.n_start;
        a3.partial = partial + (size_t)splits * f.n_rhs * 12 * P;
        a3.take_marked = 1;
        if (mixed) nl += ck ? launch_far_marks<true, true>(a3, tiles, splits, s) : launch_far_marks<false, true>(a3, tiles, splits, s);
        else nl += ck ? launch_far_marks<true, false>(a3, tiles, splits, s) : launch_far_marks<false, false>(a3, tiles, splits, s);
    } else if (tiles > 0 && f.n_rhs > 0 && far_adaptive(f.np)) {
        DNP np{f.np.eps, f.np.rs, f.np.rs_seg, f.np.analytic_calc, f.np.n_start, f.np.n_start_seg, f.np.p_max,
               f.np.p_max_seg};
        far_refine_sum_kernel<<<dim3((f.n_pts + 7) / 8, f.n_rhs, refine_parts(f)), 256, 0, s>>>(
            a, markG, markK, m.verts, m.nv, np, partial + (size_t)splits * f.n_rhs * 12 * P);
        nl++;
    }
    if (far_end) cudaEventRecord(far_end, s);
    if (tiles > 0) near_count_kernel<<<tiles128, kFarThreads, 0, s>>>(mask, n_words, f.n_pts, counts);
    *far_launches = nl;
    *launches = nl + (tiles > 0 ? 1 : 0) + 1;
    scan_kernel<<<1, 1024, 0, s>>>(counts, f.n_pts, offs, d_total);
    return cudaGetLastError();
}

cudaError_t field_stage2(const FieldLaunch& f, void* ws, int splits, long long n_near, void* pair_ws,
                         unsigned long long* d_nonfinite, cudaStream_t s, int* launches) {
    *launches = 0;
    const MeshDev& m = *f.mesh;
    const size_t P = f.n_pts;
    char* w = (char*)ws;
    double* partial = (double*)w;
    w += align256((size_t)partial_slots(f, splits) * f.n_rhs * 12 * P * sizeof(double));
    w += align256((P + 1) * sizeof(long long));
    long long* offs = (long long*)w;
    w += align256((P + 1) * sizeof(long long)) + align256(sizeof(long long));
    const unsigned* mask = (const unsigned*)w;
    const int n_words = (int)mask_words(m.n_cells);
    w += align256(mask_words(m.n_cells) * P * sizeof(unsigned));
    double* near = (double*)w;

    int* pair_cell = nullptr;
    int* pair_pt = nullptr;
    cplx* moments = nullptr;
    int tiles = (f.n_pts + kFarThreads - 1) / kFarThreads;
    if (n_near > 0) {
        char* pw = (char*)pair_ws;
        moments = (cplx*)pw;
        pw += align256((size_t)n_near * 13 * sizeof(cplx));
        pair_cell = (int*)pw;
        pw += align256((size_t)n_near * sizeof(int));
        pair_pt = (int*)pw;
        near_fill_kernel<<<(f.n_pts + 7) / 8, 256, 0, s>>>(mask, n_words, f.n_pts, offs, pair_cell, pair_pt);
        DNP np{f.np.eps, f.np.rs, f.np.rs_seg, f.np.analytic_calc, f.np.n_start, f.np.n_start_seg, f.np.p_max,
               f.np.p_max_seg};
        const int lanes = near_lanes(n_near, np), blocks = (int)((n_near * lanes + 127) / 128);
        const auto near_pairs = lanes == 1 ? near_pair_kernel<1> : (lanes == 8 ? near_pair_kernel<8> : near_pair_kernel<32>);
        near_pairs<<<blocks, 128, 0, s>>>(f.pts, m.verts, m.nv, pair_cell, pair_pt, n_near, f.k, np, moments);
        near_sum_kernel<<<dim3((f.n_pts + 7) / 8, f.n_rhs), 256, 0, s>>>(
            offs, pair_cell, moments, reinterpret_cast<const cplx*>(f.J), f.n_pts, m.n_cells, near);
        *launches += 3;
    }
    FinalArgs fa;
    fa.pts = f.pts;
    fa.n_pts = f.n_pts;
    fa.n_rhs = f.n_rhs;
    fa.n_cells = m.n_cells;
    fa.splits = partial_slots(f, splits);
    fa.partial = partial;
    fa.offs = n_near > 0 ? offs : nullptr;
    fa.near = near;
    fa.mult = f.mult;
    for (int g = 0; g < 3; g++) {
        fa.kvec[g] = f.kvec[g];
        fa.e0[g] = f.e0[g];
    }
    fa.h_scale = f.h_scale;
    fa.add_E = f.add_E;
    fa.add_H = f.add_H;
    fa.E = f.E;
    fa.H = f.H;
    fa.nonfinite = d_nonfinite;
    if (tiles > 0 && f.n_rhs > 0) {
        finalize_kernel<<<dim3((f.n_pts + 31) / 32, f.n_rhs), kFinalThreads, 0, s>>>(fa);
        *launches += 1;
    }
    return cudaGetLastError();
}

// Bytes of the stage-2 pair workspace for n_near pairs (matches the carving).
size_t field_pair_ws_bytes(long long n_near) {
    return align256((size_t)n_near * 13 * sizeof(cplx)) + 2 * align256((size_t)n_near * sizeof(int));
}

}  // namespace bielcc_gpu
