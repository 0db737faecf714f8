// Fast-diagonalisation (FD) preconditioner of the WQ elasticity operator:
// the reference's fast_diagonalization_3d (src/yeti_iga/iga_wq_mf/fsrc/
// tensor_algebra.f90:1107-1161) with its eigen_decomposition (:992-1105),
// find_parametric_diag_3d (:1452-1482) and scaling_FastDiag (:1598-1625), as
// used by wq_mf_cg_3d (mf_wq_solver.f90:803-953), generalised from the
// scalar problem to the three displacement components.
//
// For component c the preconditioner inverts the separable operator
//     P_c = a[c][u] K_u (x) M_v (x) M_w + a[c][v] M_u (x) K_v (x) M_w
//         + a[c][w] M_u (x) M_v (x) K_w
// on the component's free box (the dofs off its clamped faces).  K_d / M_d
// are the 1-D WQ stiffness and mass matrices W11 B1^T and W00 B0^T
// (eigen_decomposition's KK and MM).  With K_d U_d = M_d U_d Lambda_d and
// U_d^T M_d U_d = I,
//     P_c^{-1} = (U_w (x) U_v (x) U_u) diag(1 / Lambda_c) (U_w (x) U_v (x) U_u)^T,
//     Lambda_c(i,j,k) = a[c][u] lu_i + a[c][v] lv_j + a[c][w] lw_k.
// a[c][d] is 1 (the reference's method 'C') or the mean over the WQ points
// of the coefficient S[(c,d),(c,d)] (the elastic counterpart of the
// Jacobian-mean lengths of jacobien_mean_3d, tensor_algebra.f90:1384-1448:
// method 'JM').  The scaled form ('JMS') applies z = s (P^{-1} (s r)) with
// s = sqrt(diag(P) / diag(K)).
//
// Device work per application: six passes of dense 1-D products along u, v,
// w (forward with U^T, the eigenvalue division fused into the w pass, then
// backward with U).  Each pass is a small-K GEMM over the lines of the box,
// its operands staged whole in shared memory; the vectors (a few MB) stay in
// L2 between passes.  FP64 runs on the FP64 matrix instructions, FP32 on
// packed FMAs over 4x8 register tiles (struct FdGemm).
#include <algorithm>
#include <cmath>
#include <deque>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "fd_stage.cuh"
#include "reduce.cuh"
#include "wq.cuh"

namespace yeti {

constexpr int kFdThreads = 256;
constexpr int kFdTL = 256;     // max lines per CTA
constexpr int kFdMaxM = 512;   // largest 1-D free size accepted
constexpr size_t kFdSmem = 200 * 1024;   // staged G and line tiles per CTA

// ------------------------------------------------------------------ host
// Symmetric eigenpairs of A (n x n, row-major, destroyed) by cyclic Jacobi
// rotations (Golub & Van Loan, Matrix Computations, sec. 8.5): A = V diag(w)
// V^T, V's columns the eigenvectors.  Returns false if it did not converge.
static bool sym_eig_jacobi(int n, std::vector<double> &A, std::vector<double> &w,
                           std::vector<double> &V) {
    V.assign((size_t)n * n, 0.0);
    for (int i = 0; i < n; i++) V[(size_t)i * n + i] = 1.0;
    auto at = [&](int i, int j) -> double & { return A[(size_t)i * n + j]; };
    double fro = 0.0;
    for (double v : A) fro += v * v;
    fro = std::sqrt(fro);
    bool ok = false;
    for (int sweep = 0; sweep < 60; sweep++) {
        double off = 0.0;
        for (int i = 0; i < n; i++)
            for (int j = i + 1; j < n; j++) off += at(i, j) * at(i, j);
        if (std::sqrt(2.0 * off) <= 1e-15 * fro) {
            ok = true;
            break;
        }
        for (int p = 0; p < n - 1; p++)
            for (int q = p + 1; q < n; q++) {
                const double apq = at(p, q);
                if (std::fabs(apq) <= 1e-300) continue;
                const double theta = (at(q, q) - at(p, p)) / (2.0 * apq);
                const double t = (theta >= 0 ? 1.0 : -1.0) /
                                 (std::fabs(theta) + std::sqrt(1.0 + theta * theta));
                const double cs = 1.0 / std::sqrt(1.0 + t * t), sn = t * cs;
                // A <- J^T A J with J the rotation in the (p, q) plane
                for (int k = 0; k < n; k++) {
                    const double akp = at(k, p), akq = at(k, q);
                    at(k, p) = cs * akp - sn * akq;
                    at(k, q) = sn * akp + cs * akq;
                }
                for (int k = 0; k < n; k++) {
                    const double apk = at(p, k), aqk = at(q, k);
                    at(p, k) = cs * apk - sn * aqk;
                    at(q, k) = sn * apk + cs * aqk;
                }
                at(p, q) = at(q, p) = 0.0;
                for (int k = 0; k < n; k++) {
                    double *vr = &V[(size_t)k * n];
                    const double vkp = vr[p], vkq = vr[q];
                    vr[p] = cs * vkp - sn * vkq;
                    vr[q] = sn * vkp + cs * vkq;
                }
            }
    }
    w.resize(n);
    for (int i = 0; i < n; i++) w[i] = at(i, i);
    return ok;
}

// Generalised symmetric-definite pencil K U = M U diag(lam), U^T M U = I,
// through M = L L^T and the standard form L^{-1} K L^{-T}.
static bool gen_eig(int n, const std::vector<double> &K, const std::vector<double> &M,
                    std::vector<double> &lam, std::vector<double> &U) {
    std::vector<double> L((size_t)n * n, 0.0);
    for (int j = 0; j < n; j++) {
        double d = M[(size_t)j * n + j];
        for (int k = 0; k < j; k++) d -= L[(size_t)j * n + k] * L[(size_t)j * n + k];
        if (!(d > 0.0)) return false;
        const double ljj = std::sqrt(d);
        L[(size_t)j * n + j] = ljj;
        for (int i = j + 1; i < n; i++) {
            double v = M[(size_t)i * n + j];
            for (int k = 0; k < j; k++) v -= L[(size_t)i * n + k] * L[(size_t)j * n + k];
            L[(size_t)i * n + j] = v / ljj;
        }
    }
    // Y = L^{-1} K (forward substitution per column), C = L^{-1} Y^T
    std::vector<double> Y((size_t)n * n), C((size_t)n * n);
    for (int col = 0; col < n; col++)
        for (int i = 0; i < n; i++) {
            double v = K[(size_t)i * n + col];
            for (int k = 0; k < i; k++) v -= L[(size_t)i * n + k] * Y[(size_t)k * n + col];
            Y[(size_t)i * n + col] = v / L[(size_t)i * n + i];
        }
    for (int col = 0; col < n; col++)
        for (int i = 0; i < n; i++) {
            double v = Y[(size_t)col * n + i];   // (Y^T)[i][col]
            for (int k = 0; k < i; k++) v -= L[(size_t)i * n + k] * C[(size_t)k * n + col];
            C[(size_t)i * n + col] = v / L[(size_t)i * n + i];
        }
    for (int i = 0; i < n; i++)
        for (int j = i + 1; j < n; j++) {
            const double s = 0.5 * (C[(size_t)i * n + j] + C[(size_t)j * n + i]);
            C[(size_t)i * n + j] = C[(size_t)j * n + i] = s;
        }
    std::vector<double> Q;
    if (!sym_eig_jacobi(n, C, lam, Q)) return false;
    // U = L^{-T} Q (back substitution per column)
    U.assign((size_t)n * n, 0.0);
    for (int col = 0; col < n; col++)
        for (int i = n - 1; i >= 0; i--) {
            double v = Q[(size_t)i * n + col];
            for (int k = i + 1; k < n; k++) v -= L[(size_t)k * n + i] * U[(size_t)k * n + col];
            U[(size_t)i * n + col] = v / L[(size_t)i * n + i];
        }
    return true;
}

// 1-D WQ matrices of one direction restricted to functions [lo, hi),
// symmetrised: M = W00 B0^T, K = W11 B1^T (eigen_decomposition's MM, KK).
static void wq_1d_matrices(const WQRule1D &R, int lo, int hi, std::vector<double> &K,
                           std::vector<double> &M) {
    const int m = hi - lo, nq = R.nqp;
    K.assign((size_t)m * m, 0.0);
    M.assign((size_t)m * m, 0.0);
    for (int i = 0; i < m; i++)
        for (int j = 0; j < m; j++) {
            const double *w0 = &R.W00[(size_t)(lo + i) * nq], *b0 = &R.B0[(size_t)(lo + j) * nq];
            const double *w1 = &R.W11[(size_t)(lo + i) * nq], *b1 = &R.B1[(size_t)(lo + j) * nq];
            double sm = 0.0, sk = 0.0;
            for (int q = 0; q < nq; q++) {
                sm += w0[q] * b0[q];
                sk += w1[q] * b1[q];
            }
            M[(size_t)i * m + j] = sm;
            K[(size_t)i * m + j] = sk;
        }
    for (int i = 0; i < m; i++)
        for (int j = i + 1; j < m; j++) {
            const double a = 0.5 * (M[(size_t)i * m + j] + M[(size_t)j * m + i]);
            const double b = 0.5 * (K[(size_t)i * m + j] + K[(size_t)j * m + i]);
            M[(size_t)i * m + j] = M[(size_t)j * m + i] = a;
            K[(size_t)i * m + j] = K[(size_t)j * m + i] = b;
        }
}

// ---------------------------------------------------------------- device
template <class T>
struct FdArgs {
    const T *in;
    T *out;
    const T *g;        // G for this pass: out_row = sum_k G[k][row] in_k
    const T *dsc;      // a[c][d] * lambda_d
    const T *s;        // scaling (nullptr: none)
    const T *r;        // residual (reduction modes)
    T *p;              // FD_START: p = z
    const int *done;
    CGScal *cg;
    double *parts;
    int red, vec;      // vec: lines can be copied in 16-byte pieces
    int n[3];
    int64_t ncp;
    int lo[3][3], m[3][3];
    int64_t goff[3];   // per component, for this pass
    int64_t goff2[3];  // fused w pass: the backward matrix
    int64_t doff[3][3];
    int nA[3], nL[3], ntA[3], cta_end[3];
};

// The product of a pass on staged operands: out[a][l] = sum_k G[k][a] x(k, l)
// for the CTA's rows a < kRow nA and lines l < kLine nL, G at Gs[k ldg + a] and x at
// Xs[k ldx + l] (LK = false) or Xs[l ldx + k] (LK = true); K, rows and lines
// beyond the data are zero in shared memory.  run() gives the calling
// thread's outputs to visit, eight at a time, after all have been formed:
// visit(a, l, v) with the rows, lines and values of the eight (FP32: two
// groups of four consecutive lines, LK: rows).  `between` runs first (a
// barrier, when visit overwrites an operand).
template <class T> struct FdGemm;

// FP32: a thread per 4 rows (4 ag ..) x 8 lines (LK: lg + nL j; else 4 lg .. and
// 4 (nL + lg) ..); consecutive threads take consecutive outputs in memory:
// lines, LK: rows.  The 32 FMAs of a warp take 8 cycles of the SM, the 16-byte
// loads that feed them 12 wavefronts (4x4 tiles: 8 for 4).  8x8 tiles balance
// the two (16 and 16), but leave 64^3 elements five warps per SM, which the
// latency of a step then bounds: 26 us for the plane pass against 22 us.
template <>
struct FdGemm<float> {
    static constexpr int kRow = 4, kLine = 8;   // rows / lines per unit of nA / nL
    __host__ __device__ static int threads(int nA, int nL) { return (nA * nL + 31) / 32 * 32; }
    __host__ __device__ static int ldg(int nA) { return 4 * nA; }
    __host__ __device__ static int ldx(int m, int nL, bool lk) {
        // LK: a multiple of 4 floats, odd in units of 4 (bank groups of 8 lanes)
        return lk ? ((m + 3) / 4 | 1) * 4 : 8 * nL;
    }

    template <bool LK, class B, class V>
    static __device__ __forceinline__ void run(const float *Gs, int ldg, const float *Xs, int ldx,
                                               int m4, int nA, int nL, B between, V visit) {
        const int t0 = LK ? nA : nL, fast = threadIdx.x % t0, slow = threadIdx.x / t0;
        const int lg = LK ? slow : fast, ag = LK ? fast : slow;
        const bool act = slow < (LK ? nL : nA);
        // LK: rows in pairs, acc[line][row / 2]; else lines in pairs,
        // acc[line / 2 + 4 (row / 2)][row % 2]
        float2 acc[8][2];
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
        auto ld = [](const float *p) { return *reinterpret_cast<const float4 *>(p); };
        if (act && LK) {
            const float *g0 = Gs + 4 * ag, *xp = Xs + lg * ldx;
            const int js = nL * ldx;
            for (int k = 0; k < m4; k += 4) {
                float4 x4[8], g[4];
#pragma unroll
                for (int j = 0; j < 8; j++) x4[j] = ld(xp + j * js + k);
#pragma unroll
                for (int kk = 0; kk < 4; kk++) g[kk] = ld(g0 + (k + kk) * ldg);
#pragma unroll
                for (int kk = 0; kk < 4; kk++)
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float x = kk == 0 ? x4[j].x : kk == 1 ? x4[j].y : kk == 2 ? x4[j].z : x4[j].w;
                        acc[j][0] = __ffma2_rn(make_float2(g[kk].x, g[kk].y), make_float2(x, x), acc[j][0]);
                        acc[j][1] = __ffma2_rn(make_float2(g[kk].z, g[kk].w), make_float2(x, x), acc[j][1]);
                    }
            }
        }
        if (act && !LK) {
            const float *g0 = Gs + 4 * ag, *x0 = Xs + 4 * lg, *x1 = x0 + 4 * nL;
#pragma unroll 4
            for (int k = 0; k < m4; k++) {
                const float4 g = ld(g0 + k * ldg), xa = ld(x0 + k * ldx), xb = ld(x1 + k * ldx);
                const float2 x[4] = {{xa.x, xa.y}, {xa.z, xa.w}, {xb.x, xb.y}, {xb.z, xb.w}};
                const float gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        acc[j + 4 * (i / 2)][i % 2] =
                            __ffma2_rn(make_float2(gv[i], gv[i]), x[j], acc[j + 4 * (i / 2)][i % 2]);
            }
        }
        between();
        if (!act) return;
#pragma unroll
        for (int o = 0; o < 4; o++) {
            int a[8], l[8];
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; e++) {
                // LK: lines 2 o, 2 o + 1 with four rows each; else row o with its lines
                const int i = LK ? e % 4 : o, j = LK ? 2 * o + e / 4 : e;
                a[e] = 4 * ag + i;
                l[e] = LK ? lg + nL * j : (j < 4 ? 4 * lg : 4 * (nL + lg) - 4) + j;
                const float2 p = LK ? acc[j][i / 2] : acc[j / 2 + 4 * (i / 2)][i % 2];
                v[e] = (LK ? i : j) & 1 ? p.y : p.x;
            }
            visit(a, l, v);
        }
    }
};

// d += a b on the FP64 matrix instruction (8x4 times 4x8): lane holds
// a[lane / 4][lane % 4], b[lane % 4][lane / 4] and d[lane / 4][2 (lane % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// FP64: a warp per block of 16 rows x 16 lines, blocks dealt out in turn
// (at most kBlocks per warp).  Bound by the FP64 pipe: the four matrix
// instructions of four k take 16 cycles of the SM, their eight wavefronts of
// operands 8; a 4x4 register tile on scalar FMAs took 16 wavefronts for 8
// cycles of FMAs.  Leading dimensions are 4 or 12 modulo 16 doubles, so that the
// 4 x 4 doubles a half warp reads lie on distinct banks.  Measured on B200
// (u + v + w + v + u of one application): 64^3 p=3 177 -> 80 us, 21x17x25 p=3 (two
// plane passes and w) 42 -> 18 us; FP32 128x128x32 p=4 218 -> 138 us.
template <>
struct FdGemm<double> {
    static constexpr int kRow = 16, kLine = 16, kBlocks = 4;
    __host__ __device__ static int threads(int nA, int nL) {
        const int w = nA * nL;
        return 32 * (w <= 8 ? w : 8);
    }
    __host__ __device__ static int ldg(int nA) { return 16 * nA + 4; }
    __host__ __device__ static int ldx(int m, int nL, bool lk) {
        const int m4 = (m + 3) / 4 * 4;
        return !lk ? 16 * nL + 4 : m4 % 8 ? m4 : m4 + 4;
    }

    template <bool LK, class B, class V>
    static __device__ __forceinline__ void run(const double *Gs, int ldg, const double *Xs, int ldx,
                                               int m4, int nA, int nL, B between, V visit) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
        const int r = lane >> 2, q = lane & 3;
        double acc[kBlocks][2][2][2];
#pragma unroll
        for (int b = 0; b < kBlocks; b++) {
            const int blk = warp + b * nwarp;
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) acc[b][i][j][0] = acc[b][i][j][1] = 0.0;
            if (blk >= nA * nL) continue;
            const int ab = blk / nL, lb = blk - ab * nL;
            const double *g = Gs + q * ldg + 16 * ab + r;
            const double *x = LK ? Xs + (16 * lb + r) * ldx + q : Xs + q * ldx + 16 * lb + r;
            const int xj = LK ? 8 * ldx : 8, xk = LK ? 1 : ldx;
#pragma unroll 4
            for (int k = 0; k < m4; k += 4) {
                const double a0 = g[k * ldg], a1 = g[k * ldg + 8];
                const double b0 = x[k * xk], b1 = x[k * xk + xj];
                dmma(acc[b][0][0], a0, b0);
                dmma(acc[b][0][1], a0, b1);
                dmma(acc[b][1][0], a1, b0);
                dmma(acc[b][1][1], a1, b1);
            }
        }
        between();
#pragma unroll
        for (int b = 0; b < kBlocks; b++) {
            const int blk = warp + b * nwarp;
            if (blk >= nA * nL) continue;
            const int ab = blk / nL, lb = blk - ab * nL;
            int a[8], l[8];
            double v[8];
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const int i = e >> 2, j = e >> 1 & 1;
                a[e] = 16 * ab + 8 * i + r;
                l[e] = 16 * lb + 8 * j + 2 * q + (e & 1);
                v[e] = acc[b][i][j][e & 1];
            }
            visit(a, l, v);
        }
    }
};
// Largest number of units nA nL of a CTA.
template <class T>
constexpr int kFdUnits = sizeof(T) == 4 ? kFdThreads : 8 * FdGemm<double>::kBlocks;

// Least threads of a CTA.  FP64 CTAs of small patches have a few blocks only:
// the other warps help to stage the operands (21x17x25 p=3: plane pass 5.9 ->
// 5.3 us, w pass 7.4 -> 6.6 us); in FP32 they cost the 64^3 plane pass 1 us.
template <class T>
constexpr int kFdLeast = sizeof(T) == 4 ? 32 : kFdThreads;

// Leading dimension of the 1-D matrices in global memory: that of a staged
// matrix with all its rows in one tile, so that it is copied as one run.
template <class T>
__host__ __device__ inline int fd_ldm(int m) {
    return FdGemm<T>::ldg((m + FdGemm<T>::kRow - 1) / FdGemm<T>::kRow);
}
// Elements of such a matrix (zero rows up to fd_m4(m)).
template <class T>
__host__ __device__ inline int64_t fd_matrix(int m) {
    return (int64_t)fd_m4(m) * fd_ldm<T>(m);
}

// Tiles of one pass for one component: nA units of rows (ntA row tiles) and
// nL units of lines per CTA, the whole contraction staged in shared memory.
// The fused w pass (two G matrices) needs one row tile.  Of the tilings
// that fit, the one whose busiest SM has the least work (units, in whole
// warps) is taken, counting the CTAs that share an SM; ties go to the larger
// tile, which reads G less often.
template <class T>
static FdTile fd_tile(int m, int64_t nlines, bool lk, bool fused) {
    using Gm = FdGemm<T>;
    const int m4 = fd_m4(m), units = (m + Gm::kRow - 1) / Gm::kRow;
    FdTile best;
    best.ctas = -1;
    double best_cost = 0.0;
    for (int ntA = 1; ntA <= (fused ? 1 : units); ntA++) {
        const int nA = (units + ntA - 1) / ntA;
        for (int nL = 1; nL * Gm::kLine <= kFdTL && nA * nL <= kFdUnits<T>; nL++) {
            FdTile t;
            t.ntA = ntA;
            t.nA = nA;
            t.nL = nL;
            const size_t g = (size_t)m4 * Gm::ldg(nA) * (fused ? 2 : 1);
            const int ldx = Gm::ldx(m, nL, lk);
            const size_t x = lk ? (size_t)nL * Gm::kLine * ldx
                                : (size_t)(fused ? std::max(m4, nA * Gm::kRow) : m4) * ldx;
            t.smem = (g + x) * sizeof(T);
            if (t.smem > kFdSmem) continue;
            t.threads = Gm::threads(nA, nL);
            t.ctas = ntA * (int)((nlines + nL * Gm::kLine - 1) / (nL * Gm::kLine));
            // three components share the SMs
            const double per_sm = std::ceil(3.0 * t.ctas / 148.0);
            const double resident = std::max(1.0, std::min(std::floor(227.0 * 1024 / (t.smem + 8192)),
                                                           std::floor(512.0 / t.threads)));
            const double work = sizeof(T) == 4 ? t.threads / 32 : nA * nL;
            // units on the busiest SM (four schedulers take them in
            // fours); a round of CTAs also pays its loads
            const double rounds = std::ceil(per_sm / resident);
            const double cost = std::ceil(per_sm * work / 4.0) * 4.0 + rounds * 2.0;
            if (best.ctas < 0 || cost < best_cost - 1e-9 ||
                (cost < best_cost + 1e-9 && nA * nL > best.nA * best.nL)) {
                best = t;
                best_cost = cost;
            }
        }
        if (best.ctas > 0 && ntA >= 4) break;
    }
    return best;   // ctas -1: not possible
}

// Asynchronous global -> shared copy of one element (cp.async, sm_80+);
// valid == false writes zero and reads nothing.
template <class T>
__device__ __forceinline__ void cp_elem(T *sdst, const T *gsrc, bool valid) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(saddr), "l"(gsrc),
                 "n"((int)sizeof(T)), "r"(valid ? (int)sizeof(T) : 0)
                 : "memory");
}
// 16 bytes (both addresses 16-byte aligned), of which the first n elements
// (0 <= n <= 16 / sizeof(T): fd_piece) are read and the rest written as zero.
template <class T>
__device__ __forceinline__ void cp_vec(T *sdst, const T *gsrc, int n) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(saddr), "l"(gsrc),
                 "r"(n * (int)sizeof(T))
                 : "memory");
}
// Four consecutive values; aligned: one 16-byte store.
__device__ __forceinline__ void store4(float *o, const float *v, bool aligned) {
    if (aligned) *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
    else
#pragma unroll
        for (int e = 0; e < 4; e++) o[e] = v[e];
}
__device__ __forceinline__ void store4(double *o, const double *v, bool) {
#pragma unroll
    for (int e = 0; e < 4; e++) o[e] = v[e];
}

// The last step of a pass for eight outputs of a thread at idx (-1: none):
// EPI 2 scales, adds to r.z and sets p.  Loads first: the stores that follow
// would each be waited for.  Four consecutive outputs (FP32) go out as one
// store where they are aligned.
template <class T, int EPI>
__device__ __forceinline__ void fd_write(const FdArgs<T> &a, const int64_t (&idx)[8], T (&v)[8],
                                         double &rz) {
    if (EPI == 2) {
        T sv[8], rv[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            sv[e] = a.s && idx[e] >= 0 ? __ldg(a.s + idx[e]) : T(1);
            rv[e] = a.red != FD_NONE && idx[e] >= 0 ? __ldg(a.r + idx[e]) : T(0);
        }
#pragma unroll
        for (int e = 0; e < 8; e++) {
            if (a.s) v[e] *= sv[e];
            if (a.red != FD_NONE && idx[e] >= 0) rz += (double)rv[e] * (double)v[e];
        }
    }
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
        const bool run = sizeof(T) == 4 && idx[h] >= 0 && idx[h + 3] == idx[h] + 3 && idx[h + 1] == idx[h] + 1;
        if (run) {
            store4(a.out + idx[h], v + h, (reinterpret_cast<uintptr_t>(a.out + idx[h]) & 15) == 0);
            if (EPI == 2 && a.red == FD_START)
                store4(a.p + idx[h], v + h, (reinterpret_cast<uintptr_t>(a.p + idx[h]) & 15) == 0);
        } else {
#pragma unroll
            for (int e = h; e < h + 4; e++) {
                if (idx[e] < 0) continue;
                a.out[idx[e]] = v[e];
                if (EPI == 2 && a.red == FD_START) a.p[idx[e]] = v[e];
            }
        }
    }
}

// Columns a0 .. a0 + n of a 1-D matrix into Gs[k ldg + a], k < fd_m4(m); zero
// beyond the data, in 16-byte pieces, consecutive threads on consecutive
// ones (the whole matrix as one run).
template <class T>
__device__ __forceinline__ void stage_matrix(T *Gs, int ldg, const T *G, int m, int a0, int n) {
    constexpr int VEC = 16 / sizeof(T);
    const int ldm = fd_ldm<T>(m);
    if (a0 == 0 && ldg == ldm) {
        const int tot = fd_m4(m) * ldm;
        for (int t = threadIdx.x * VEC; t < tot; t += blockDim.x * VEC) cp_vec(Gs + t, G + t, VEC);
        return;
    }
    const int nv = n / VEC, tot = fd_m4(m) * nv;
    for (int t = threadIdx.x; t < tot; t += blockDim.x) {
        const int k = t / nv, a = (t - k * nv) * VEC;
        const bool in = a0 + a < ldm;
        cp_vec(Gs + k * ldg + a, in ? G + (int64_t)k * ldm + a0 + a : G, in ? VEC : 0);
    }
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// End of the last pass of a CG application: the r.z partials of the block,
// then (last block) the CG scalars of the reduction mode.
template <class T>
__device__ __forceinline__ void fd_finish_rz(const FdArgs<T> &a, double rz, double *sh) {
    rz = block_sum(rz, sh);
    if (threadIdx.x == 0) __stcg(&a.parts[blockIdx.x], rz);
    if (!last_block(&a.cg->ticket)) return;
    double srz = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) srz += __ldcg(&a.parts[i]);
    srz = block_sum(srz, sh);
    if (threadIdx.x == 0) {
        CGScal *s = a.cg;
        s->ticket = 0;
        if (a.red == FD_ITER) {
            const double old = s->rz;
            s->beta = srz / old;
            if (!isfinite(srz) || !(old != 0.0)) {
                s->breakdown = 1;
                s->done = 1;
            }
        }
        s->rz = srz;
    }
}

// One pass along axis AX: out_row(line) = sum_k G[k][row] in_k(line).
// EPI 1: divide by Lambda; EPI 2: multiply by s, r.z partials and the
// reduction mode; EPI 3 (AX == 2, one row tile): forward product, division
// by Lambda and backward product in one CTA, the intermediate kept in shared
// memory.  The G columns and the lines are staged by cp.async (all copies in
// flight at once): lines along u as they lie in memory (LK), the others with
// the lines consecutive.
template <class T, int AX, int EPI>
__global__ void __launch_bounds__(kFdThreads, sizeof(T) == 4 ? 3 : 2) k_fd_pass(FdArgs<T> a) {
    using Gm = FdGemm<T>;
    constexpr bool LK = AX == 0;
    extern __shared__ __align__(16) unsigned char fd_smem[];
    __shared__ int64_t lb[kFdTL];
    __shared__ T ll12[kFdTL];    // EPI 1, 3: the line's part of Lambda
    __shared__ double sh[32];
    if (a.done && *a.done) return;
    int b = blockIdx.x, c = 0;
    while (c < 2 && b >= a.cta_end[c]) c++;
    if (c > 0) b -= a.cta_end[c - 1];
    constexpr int D1 = AX == 0 ? 1 : 0, D2 = AX == 2 ? 1 : 2;
    const int nA = a.nA[c], nL = a.nL[c], ntA = a.ntA[c];
    const int m = a.m[c][AX], m1 = a.m[c][D1], m2 = a.m[c][D2], m4 = fd_m4(m);
    const int nlines = m1 * m2;
    const int TA = Gm::kRow * nA, TL = Gm::kLine * nL, ldg = Gm::ldg(nA), ldx = Gm::ldx(m, nL, LK);
    T *Gs = reinterpret_cast<T *>(fd_smem);
    T *G2 = Gs + (size_t)m4 * ldg;                     // EPI 3
    T *Xs = EPI == 3 ? G2 + (size_t)m4 * ldg : G2;
    const int a0 = (b % ntA) * TA;
    const int l0 = (b / ntA) * TL;
    const int64_t st[3] = {1, (int64_t)a.n[0], (int64_t)a.n[0] * a.n[1]};
    const int64_t sk = st[AX];
    const int tid = threadIdx.x, nthr = blockDim.x;
    stage_matrix(Gs, ldg, a.g + a.goff[c], m, a0, TA);
    if (EPI == 3) stage_matrix(G2, ldg, a.g + a.goff2[c], m, 0, TA);
    for (int ll = tid; ll < TL; ll += nthr) {
        const int l = l0 + ll;
        int64_t base = -1;
        int i1 = 0, i2 = 0;
        if (l < nlines) {
            i2 = l / m1;
            i1 = l - i2 * m1;
            base = c * a.ncp + (int64_t)a.lo[c][AX] * sk + (int64_t)(a.lo[c][D1] + i1) * st[D1] +
                   (int64_t)(a.lo[c][D2] + i2) * st[D2];
        }
        lb[ll] = base;
        if (EPI == 1 || EPI == 3)
            ll12[ll] = base >= 0 ? a.dsc[a.doff[c][D1] + i1] + a.dsc[a.doff[c][D2] + i2] : T(1);
    }
    __syncthreads();   // lb
    constexpr int VEC = 16 / sizeof(T);
    if (LK) {
        // lines are contiguous: a warp per line, in 16-byte pieces when every
        // line begins on one
        for (int ll = tid >> 5; ll < TL; ll += nthr >> 5) {
            const int64_t base = lb[ll];
            const T *src = base >= 0 ? a.in + base : a.in;
            if (a.vec)
                for (int k = (tid & 31) * VEC; k < m4; k += 32 * VEC) {
                    const int n = base >= 0 ? fd_piece(m, k, VEC) : 0;
                    cp_vec(Xs + ll * ldx + k, n ? src + k : a.in, n);
                }
            else
                for (int k = tid & 31; k < m4; k += 32)
                    cp_elem(Xs + ll * ldx + k, k < m ? src + k : src, base >= 0 && k < m);
        }
    } else if (a.vec) {
        // row k of the tile is contiguous along the lines of a run, and the
        // runs are whole 16-byte pieces
        const int nv = TL / VEC;
        for (int t = tid; t < nv * m4; t += nthr) {
            const int k = t / nv, ll = (t - k * nv) * VEC;
            const int64_t base = lb[ll];
            const bool in = base >= 0 && k < m;
            cp_vec(Xs + k * ldx + ll, in ? a.in + base + (int64_t)k * sk : a.in, in ? VEC : 0);
        }
    } else {
        for (int t = tid; t < TL * m4; t += nthr) {
            const int k = t / TL, ll = t - k * TL;
            const int64_t base = lb[ll];
            const bool in = base >= 0 && k < m;
            cp_elem(Xs + k * ldx + ll, in ? a.in + base + (int64_t)k * sk : a.in, in);
        }
    }
    cp_wait_all();
    __syncthreads();
    double rz = 0.0;
    // Lambda of (row e, line ll); AX == 2: (lambda_u + lambda_v) + lambda_w
    static_assert(AX == 2 || (EPI != 1 && EPI != 3), "the division belongs to the w pass");
    auto lambda = [&](int e, int ll) { return ll12[ll] + __ldg(a.dsc + a.doff[c][2] + e); };
    auto write = [&](const int (&row)[8], const int (&ll)[8], T (&v)[8]) {
        int64_t idx[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const int64_t base = lb[ll[e]];
            idx[e] = a0 + row[e] < m && base >= 0 ? base + (int64_t)(a0 + row[e]) * sk : -1;
            if (EPI == 1 && idx[e] >= 0) v[e] = v[e] / lambda(a0 + row[e], ll[e]);
        }
        fd_write<T, EPI>(a, idx, v, rz);
    };
    auto nothing = [] {};
    if constexpr (EPI == 3) {
        // divide by Lambda, park the eigen-space values in Xs, contract back
        Gm::template run<false>(
            Gs, ldg, Xs, ldx, m4, nA, nL, [] { __syncthreads(); },
            [&](const int (&row)[8], const int (&ll)[8], T (&v)[8]) {
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    if (row[e] >= m4) continue;
                    const bool in = row[e] < m && lb[ll[e]] >= 0;
                    Xs[row[e] * ldx + ll[e]] = in ? v[e] / lambda(row[e], ll[e]) : T(0);
                }
            });
        __syncthreads();
        Gm::template run<false>(G2, ldg, Xs, ldx, m4, nA, nL, nothing, write);
    } else {
        Gm::template run<LK>(Gs, ldg, Xs, ldx, m4, nA, nL, nothing, write);
    }
    if (EPI != 2 || a.red == FD_NONE) return;
    fd_finish_rz(a, rz, sh);
}

// The u and v products of one w plane in one CTA: with X the plane's values
// (rows v, columns u of the component's free box),
//     T[v][a] = sum_i X[v][i] Gu[i][a],   Y[b][a] = sum_j Gv[j][b] T[j][a],
// forward (Gu = U_u, Gv = U_v; in positions, out eigen indices) or backward
// (Gu = U_u^T, Gv = U_v^T).  The plane (rows as they lie in memory), Gu's
// columns of the CTA's column split, Gv and T stay in shared memory.  goff:
// Gu, goff2: Gv; ntA: column splits, nA: units of columns per split, nL: units
// of rows.  EPI 2 as k_fd_pass.
template <class T, int EPI>
__global__ void __launch_bounds__(kFdThreads, sizeof(T) == 4 ? 3 : 2) k_fd_plane(FdArgs<T> a) {
    using Gm = FdGemm<T>;
    extern __shared__ __align__(16) unsigned char fd_smem[];
    __shared__ double sh[32];
    if (a.done && *a.done) return;
    int b = blockIdx.x, c = 0;
    while (c < 2 && b >= a.cta_end[c]) c++;
    if (c > 0) b -= a.cta_end[c - 1];
    const int mu = a.m[c][0], mv = a.m[c][1], mu4 = fd_m4(mu), mv4 = fd_m4(mv);
    const int nsplit = a.ntA[c], nA = a.nA[c], nL = a.nL[c];
    const int sp = b % nsplit, kw = b / nsplit;
    const int TA = Gm::kRow * nA, TB = Gm::kLine * nL, a0 = sp * TA;
    const int ldx = Gm::ldx(mu, nL, true), ldu = Gm::ldg(nA), ldv = Gm::ldg(TB / Gm::kRow),
              ldt = Gm::ldx(mv, TA / Gm::kLine, false);
    T *Xs = reinterpret_cast<T *>(fd_smem);       // [TB][ldx]: X[v][i]
    T *Gu = Xs + (size_t)TB * ldx;                // [mu4][ldu]
    T *Gv = Gu + (size_t)mu4 * ldu;               // [mv4][ldv]
    T *Tm = Gv + (size_t)mv4 * ldv;               // [TB][ldt]: T[v][a]
    const int64_t nu = a.n[0], nv = a.n[1];
    const int64_t plane = c * a.ncp + (int64_t)(a.lo[c][2] + kw) * nu * nv +
                          (int64_t)a.lo[c][1] * nu + a.lo[c][0];
    const int tid = threadIdx.x, nthr = blockDim.x;
    // the plane, a warp per row v (contiguous along u); rows mv .. TB zero
    constexpr int VEC = 16 / sizeof(T);
    for (int v = tid >> 5; v < TB; v += nthr >> 5) {
        const T *src = v < mv ? a.in + plane + v * nu : a.in;
        if (a.vec)
            for (int i = (tid & 31) * VEC; i < mu4; i += 32 * VEC) {
                const int n = v < mv ? fd_piece(mu, i, VEC) : 0;
                cp_vec(Xs + v * ldx + i, n ? src + i : a.in, n);
            }
        else
            for (int i = tid & 31; i < mu4; i += 32)
                cp_elem(Xs + v * ldx + i, i < mu ? src + i : src, v < mv && i < mu);
    }
    stage_matrix(Gu, ldu, a.g + a.goff[c], mu, a0, TA);
    stage_matrix(Gv, ldv, a.g + a.goff2[c], mv, 0, TB);
    cp_wait_all();
    __syncthreads();
    Gm::template run<true>(Gu, ldu, Xs, ldx, mu4, nA, nL, [] {},
                           [&](const int (&col)[8], const int (&v)[8], T (&t)[8]) {
#pragma unroll
                               for (int e = 0; e < 8; e++) Tm[v[e] * ldt + col[e]] = t[e];
                           });
    __syncthreads();
    double rz = 0.0;
    Gm::template run<false>(Gv, ldv, Tm, ldt, mv4, TB / Gm::kRow, TA / Gm::kLine, [] {},
                            [&](const int (&row)[8], const int (&col)[8], T (&v)[8]) {
                                int64_t idx[8];
#pragma unroll
                                for (int e = 0; e < 8; e++)
                                    idx[e] = row[e] < mv && a0 + col[e] < mu
                                                 ? plane + (int64_t)row[e] * nu + a0 + col[e]
                                                 : -1;
                                fd_write<T, EPI>(a, idx, v, rz);
                            });
    if (EPI != 2 || a.red == FD_NONE) return;
    fd_finish_rz(a, rz, sh);
}

// out = s in (elementwise; s is zero off the free boxes)
template <class T>
__global__ void k_fd_scale_in(const T *in, const T *sv, T *out, int64_t n, const int *done) {
    if (done && *done) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = in[i] * sv[i];
}

// s = sqrt(diag(P) / diag(K)) on every component's free box, 0 elsewhere;
// diag(P) from the 1-D diagonals (find_parametric_diag_3d).
__global__ void k_fd_scaling(const double *diagK, const double *kdmd, double *s64, float *s32, int3 n, int64_t ncp, int lo0, int lo1,
                             int lo2, int m0, int m1, int m2, int c, int64_t off_u,
                             int64_t off_v, int64_t off_w, double au, double av, double aw) {
    const int64_t tot = (int64_t)m0 * m1 * m2;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < tot;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(t % m0), j = (int)((t / m0) % m1), k = (int)(t / ((int64_t)m0 * m1));
        const double ku = kdmd[off_u + i], mu = kdmd[off_u + m0 + i];
        const double kv = kdmd[off_v + j], mv = kdmd[off_v + m1 + j];
        const double kw = kdmd[off_w + k], mw = kdmd[off_w + m2 + k];
        const double dp = au * ku * mv * mw + av * mu * kv * mw + aw * mu * mv * kw;
        const int64_t idx = c * ncp + (int64_t)(lo0 + i) + (int64_t)n.x * ((lo1 + j) + (int64_t)n.y * (lo2 + k));
        const double v = sqrt(dp / diagK[idx]);
        if (s64) s64[idx] = v;
        if (s32) s32[idx] = (float)v;
    }
}

// ------------------------------------------------------------------ plan
// Tiling of the fused plane pass for one component: column splits of the
// u products (each CTA recomputes nothing, it reads the whole plane), with
// the staged plane, Gu columns, Gv and T within kFdSmem, and splits added while
// the pass (three components) has fewer CTAs than SMs.  ctas = -1: does not
// fit (the line passes run instead).
template <class T>
static FdPlane fd_plane_tile(int mu, int mv, int mw) {
    using Gm = FdGemm<T>;
    // rows and lines change roles between the products: whole units of both
    constexpr int per = std::max(1, Gm::kLine / Gm::kRow);
    const int units = (mu + Gm::kRow - 1) / Gm::kRow;
    FdPlane t, best;
    best.ctas = -1;
    t.nL = (mv + Gm::kLine - 1) / Gm::kLine;
    const int TB = Gm::kLine * t.nL;
    for (t.nsplit = 1; t.nsplit <= units; t.nsplit++) {
        t.nA = ((units + t.nsplit - 1) / t.nsplit + per - 1) / per * per;
        t.smem = ((size_t)TB * Gm::ldx(mu, t.nL, true) + (size_t)fd_m4(mu) * Gm::ldg(t.nA) +
                  (size_t)fd_m4(mv) * Gm::ldg(TB / Gm::kRow) +
                  (size_t)TB * Gm::ldx(mv, t.nA * Gm::kRow / Gm::kLine, false)) * sizeof(T);
        if (t.nA * t.nL > kFdUnits<T> || t.smem > kFdSmem) continue;
        t.ctas = mw * t.nsplit;
        t.threads = std::max(Gm::threads(t.nA, t.nL), kFdLeast<T>);
        best = t;
        if (3 * t.ctas >= 148) break;
    }
    return best;
}

template <class T>
static int fd_set_attrs() {
    const int b = (int)kFdSmem;
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    YETI_CUDA(cudaFuncSetAttribute(k_fd_pass<T, 0, 0>, a, b));
    YETI_CUDA(cudaFuncSetAttribute(k_fd_pass<T, 1, 0>, a, b));
    YETI_CUDA(cudaFuncSetAttribute(k_fd_pass<T, 2, 0>, a, b));
    YETI_CUDA(cudaFuncSetAttribute(k_fd_pass<T, 2, 1>, a, b));
    YETI_CUDA(cudaFuncSetAttribute(k_fd_pass<T, 2, 3>, a, b));
    YETI_CUDA(cudaFuncSetAttribute(k_fd_pass<T, 0, 2>, a, b));
    YETI_CUDA(cudaFuncSetAttribute(k_fd_plane<T, 0>, a, b));
    YETI_CUDA(cudaFuncSetAttribute(k_fd_plane<T, 2>, a, b));
    return YETI_OK;
}

// 1-D matrices with per-point weights (eigen_decomposition's 'TD' branch,
// tensor_algebra.f90:1045-1071): M = W00 (B0 diag(mw))^T and K = W11 (B1
// diag(kw))^T on the rows lo..hi-1, made symmetric by averaging with the
// transpose, as the unweighted matrices are.  (The reference hands the
// non-symmetric products to dsygvd, which reads their upper triangle; with
// the point-to-point variation of a rough coefficient field that triangle
// is indefinite, its eigenvalue sums negative, while the symmetric part
// stays definite.)
static void wq_1d_matrices_weighted(const WQRule1D &R, int lo, int hi, const double *mw,
                                    const double *kw, std::vector<double> &K,
                                    std::vector<double> &M) {
    const int m = hi - lo, nq = R.nqp;
    K.assign((size_t)m * m, 0.0);
    M.assign((size_t)m * m, 0.0);
    for (int i = 0; i < m; i++)
        for (int j = 0; j < m; j++) {
            const double *w0 = &R.W00[(size_t)(lo + i) * nq], *b0 = &R.B0[(size_t)(lo + j) * nq];
            const double *w1 = &R.W11[(size_t)(lo + i) * nq], *b1 = &R.B1[(size_t)(lo + j) * nq];
            double sm = 0.0, sk = 0.0;
            for (int q = 0; q < nq; q++) {
                sm += w0[q] * (b0[q] * mw[q]);
                sk += w1[q] * (b1[q] * kw[q]);
            }
            M[(size_t)i * m + j] = sm;
            K[(size_t)i * m + j] = sk;
        }
    for (int i = 0; i < m; i++)
        for (int j = i + 1; j < m; j++) {
            const double a = 0.5 * (M[(size_t)i * m + j] + M[(size_t)j * m + i]);
            const double b = 0.5 * (K[(size_t)i * m + j] + K[(size_t)j * m + i]);
            M[(size_t)i * m + j] = M[(size_t)j * m + i] = a;
            K[(size_t)i * m + j] = K[(size_t)j * m + i] = b;
        }
}

// One sweep of tensor_decomposition_3d (tensor_algebra.f90:1256-1382) for
// one displacement component: cc[k] the diagonal coefficient S[(c,k),(c,k)]
// at every WQ point (u fastest), M[d] / K[d] the per-point 1-D weights of
// direction d, updated in place.  Stiffness weights first: K_k(i) =
// sqrt(min V max V) over the slice i of direction k, V = cc_k M_k /
// (M_u M_v M_w); then mass weights: M_k(i) = sqrt(min N max W) over the
// slice, from cc_k M_k M_l / (M_u M_v M_w K_k), l != k.  (The reference
// bounds its direction-3 slice loops by the v count; the w count is used
// here, which agrees whenever the two are equal.)
static void td_sweep(const int nq[3], const double *const cc[3], std::vector<double> M[3],
                     std::vector<double> K[3]) {
    const int64_t n = (int64_t)nq[0] * nq[1] * nq[2];
    for (int k = 0; k < 3; k++) {
        std::vector<double> vmin(nq[k], INFINITY), vmax(nq[k], -INFINITY);
        int64_t g = 0;
        for (int i2 = 0; i2 < nq[2]; i2++)
            for (int i1 = 0; i1 < nq[1]; i1++)
                for (int i0 = 0; i0 < nq[0]; i0++, g++) {
                    const int i[3] = {i0, i1, i2};
                    const double uu[3] = {M[0][i0], M[1][i1], M[2][i2]};
                    const double v = cc[k][g] * uu[k] / (uu[0] * uu[1] * uu[2]);
                    vmin[i[k]] = std::min(vmin[i[k]], v);
                    vmax[i[k]] = std::max(vmax[i[k]], v);
                }
        for (int a = 0; a < nq[k]; a++) K[k][a] = std::sqrt(vmin[a] * vmax[a]);
    }
    for (int k = 0; k < 3; k++) {
        std::vector<double> nmin(nq[k], INFINITY), mmax(nq[k], -INFINITY);
        int64_t g = 0;
        for (int i2 = 0; i2 < nq[2]; i2++)
            for (int i1 = 0; i1 < nq[1]; i1++)
                for (int i0 = 0; i0 < nq[0]; i0++, g++) {
                    const int i[3] = {i0, i1, i2};
                    const double uu[3] = {M[0][i0], M[1][i1], M[2][i2]};
                    const double ww[3] = {K[0][i0], K[1][i1], K[2][i2]};
                    double lo = INFINITY, hi = -INFINITY;
                    for (int l = 0; l < 3; l++) {
                        if (l == k) continue;
                        const double w = cc[k][g] * uu[k] * uu[l] / (uu[0] * uu[1] * uu[2] * ww[k]);
                        lo = std::min(lo, w);
                        hi = std::max(hi, w);
                    }
                    nmin[i[k]] = std::min(nmin[i[k]], lo);
                    mmax[i[k]] = std::max(mmax[i[k]], hi);
                }
        for (int a = 0; a < nq[k]; a++) M[k][a] = std::sqrt(nmin[a] * mmax[a]);
    }
    (void)n;
}

// The diagonal coefficients S[(c,k),(c,k)] of every WQ point, in point
// order (u fastest), gathered from the streaming FP64 layout: out[(3c+k) n + g].
__global__ void k_fd_diag_coef(const double *coef, const int64_t *tile_off, const int *pstride,
                               const int *tq0u, const int *tnqu, const int *tq0v,
                               const int *tnqv, int ntu, int nqu, int nqv, int nqw,
                               double *out) {
    const int64_t n = (int64_t)nqu * nqv * nqw;
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n;
         g += (int64_t)gridDim.x * blockDim.x) {
        const int qu = (int)(g % nqu), qv = (int)((g / nqu) % nqv);
        const int qw = (int)(g / ((int64_t)nqu * nqv));
        int tu = 0, tv = 0;
        while (tq0u[tu] + tnqu[tu] <= qu) tu++;
        while (tq0v[tv] + tnqv[tv] <= qv) tv++;
        const int t = tu + ntu * tv;
        const int npts = tnqu[tu] * tnqv[tv];
        const int pt = (qv - tq0v[tv]) * tnqu[tu] + (qu - tq0u[tu]);
        const double *blk = coef + tile_off[t] + (int64_t)qw * pstride[t] + pt;
        for (int c = 0; c < 3; c++)
            for (int k = 0; k < 3; k++)
                out[(int64_t)(3 * c + k) * n + g] = blk[(int64_t)sym9(3 * c + k, 3 * c + k) * npts];
    }
}

// The same gather from the element-block layout of the setup kernels
// (operators of mixed degrees or degree > 5): point (qu, qv, qw) of block b
// at coef[qoff[b] 45 + e nq_b + (lw nv_b + lv) nu_b + lu].
__global__ void k_fd_diag_coef_blk(const double *coef, const int64_t *qoff,
                                   const int *const *blk1, const int *const *loc1,
                                   const int *const *nq1, int nbu, int nbv, int nqu, int nqv,
                                   int nqw, double *out) {
    const int64_t n = (int64_t)nqu * nqv * nqw;
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n;
         g += (int64_t)gridDim.x * blockDim.x) {
        const int qu = (int)(g % nqu), qv = (int)((g / nqu) % nqv);
        const int qw = (int)(g / ((int64_t)nqu * nqv));
        const int bu = blk1[0][qu], bv = blk1[1][qv], bw = blk1[2][qw];
        const int64_t b = bu + (int64_t)nbu * (bv + (int64_t)nbv * bw);
        const int nu1 = nq1[0][bu], nv1 = nq1[1][bv], nw1 = nq1[2][bw];
        const int64_t nqb = (int64_t)nu1 * nv1 * nw1;
        const double *base = coef + qoff[b] * kWQCoef +
                             (loc1[2][qw] * (int64_t)nv1 + loc1[1][qv]) * nu1 + loc1[0][qu];
        for (int c = 0; c < 3; c++)
            for (int k = 0; k < 3; k++)
                out[(int64_t)(3 * c + k) * n + g] = base[(int64_t)sym9(3 * c + k, 3 * c + k) * nqb];
    }
}

// U, then U^T (m x m, row-major), appended to g in the layout of the passes.
template <class T>
static void add_matrices(const std::vector<double> &U, int m, std::vector<T> &g, int64_t &off) {
    const int ldm = fd_ldm<T>(m);
    off = (int64_t)g.size();
    g.resize(g.size() + 2 * fd_matrix<T>(m), T(0));
    T *u = &g[off], *ut = u + fd_matrix<T>(m);
    for (int i = 0; i < m; i++)
        for (int j = 0; j < m; j++)
            u[(size_t)i * ldm + j] = ut[(size_t)j * ldm + i] = (T)U[(size_t)i * m + j];
}

// The tilings of every pass; returns the most CTAs of a pass (partials of its
// reduction).
template <class T>
static int fd_plan_tiles(WQFdPlan &F) {
    const int w = sizeof(T) == 4;
    int most = 0;
    for (int ps = 0; ps < 4; ps++) {   // u, v, w, fused w
        const int ax = std::min(ps, 2);
        int tot = 0;
        for (int c = 0; c < 3; c++) {
            F.tile[w][ps][c] = fd_tile<T>(F.m[c][ax], (int64_t)F.m[c][ax == 0 ? 1 : 0] *
                                                          F.m[c][ax == 2 ? 1 : 2], ax == 0, ps == 3);
            tot += std::max(0, F.tile[w][ps][c].ctas);
        }
        most = std::max(most, tot);
    }
    int tot = 0;
    for (int c = 0; c < 3; c++) {
        F.plane[w][c] = fd_plane_tile<T>(F.m[c][0], F.m[c][1], F.m[c][2]);
        tot += std::max(0, F.plane[w][c].ctas);
    }
    return std::max(most, tot);
}

int wq_fd_prepare(yeti_wq_op *op, int variant, bool f32) {
    WQFdPlan &F = op->fd;
    variant &= (YETI_PCG_FD | YETI_PCG_FD_SCALED | YETI_PCG_FD_UNIT | YETI_PCG_FD_TD);
    if (F.variant == variant && (!f32 || F.g32.ptr)) return YETI_OK;
    const bool td = (variant & YETI_PCG_FD_TD) != 0;
    YETI_CHECK(!td || op->coef64.ptr, YETI_EUNSUPPORTED,
               "fast diagonalisation 'TD': needs the operator's FP64 data");
    // the passes stage up to kFdSmem bytes: opt in once per device (the
    // attribute is always this maximum, so concurrent callers agree)
    YETI_TRY(fd_set_attrs<double>());
    YETI_TRY(fd_set_attrs<float>());
    yeti_ctx *ctx = op->ctx;
    cudaStream_t s = ctx->stream;
    const bool unit = (variant & YETI_PCG_FD_UNIT) != 0;
    const bool scaled = (variant & YETI_PCG_FD_SCALED) != 0;
    // free boxes
    for (int c = 0; c < 3; c++) {
        YETI_CHECK(op->cmask[c] != 0, YETI_EINVAL,
                   "fast diagonalisation: component %d has no clamped face (singular)", c);
        for (int d = 0; d < 3; d++) {
            const int lo = (op->cmask[c] >> (2 * d)) & 1;
            const int hi = op->n[d] - ((op->cmask[c] >> (2 * d + 1)) & 1);
            F.lo[c][d] = lo;
            F.m[c][d] = hi - lo;
            YETI_CHECK(F.m[c][d] >= 1 && F.m[c][d] <= kFdMaxM, YETI_EINVAL,
                       "fast diagonalisation: %d free functions along direction %d "
                       "(1..%d supported)", F.m[c][d], d, kFdMaxM);
        }
    }
    // coefficients a[c][d] ('TD': 1, the weights carry the coefficients)
    double acoef[3][3];
    if (unit || td) {
        for (int c = 0; c < 3; c++)
            for (int d = 0; d < 3; d++) acoef[c][d] = 1.0;
    } else {
        std::vector<double> sd((size_t)op->nblocks * 9);
        YETI_CUDA(cudaMemcpyAsync(sd.data(), op->sdiag.ptr, sd.size() * sizeof(double),
                                  cudaMemcpyDeviceToHost, s));
        YETI_CUDA(cudaStreamSynchronize(s));
        double sum[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int64_t b = 0; b < op->nblocks; b++)
            for (int k = 0; k < 9; k++) sum[k] += sd[(size_t)b * 9 + k];
        for (int c = 0; c < 3; c++)
            for (int d = 0; d < 3; d++) {
                acoef[c][d] = sum[3 * c + d] / (double)op->nqp_total;
                YETI_CHECK(acoef[c][d] > 0.0 && std::isfinite(acoef[c][d]), YETI_ENUMERIC,
                           "fast diagonalisation: mean coefficient %g", acoef[c][d]);
            }
    }
    // eigenpairs per distinct (p, nel, lo, hi)
    WQRule1D R[3];
    for (int d = 0; d < 3; d++)
        YETI_CHECK(wq_rule_1d(op->p[d], op->nel[d], R[d]) == 0, YETI_EINVAL,
                   "fast diagonalisation: WQ rule failed");
    // 'TD': per component, two sweeps of the tensor decomposition of the
    // diagonal coefficients give per-point 1-D weights (wq_mf_cg_3d,
    // mf_wq_solver.f90:809-826, per displacement component)
    std::vector<double> tdM[3][3], tdK[3][3];
    if (td) {
        const int nq[3] = {op->nqp[0], op->nqp[1], op->nqp[2]};
        const int64_t n = (int64_t)nq[0] * nq[1] * nq[2];
        DevBuf dcc;
        YETI_TRY(dcc.alloc(ctx, (size_t)9 * n * sizeof(double)));
        WQStreamPlan &st = op->st;
        DevBuf blk[3], loc[3], nqb[3], ptrs;   // block-layout maps (freed on return)
        if (st.active) {
            k_fd_diag_coef<<<592, 256, 0, s>>>(op->coef64.as<double>(), st.tile_off.as<int64_t>(),
                                               st.tile_pstride.as<int>(), st.tq0[0].as<int>(),
                                               st.tnq[0].as<int>(), st.tq0[1].as<int>(),
                                               st.tnq[1].as<int>(), st.ntile[0], nq[0], nq[1],
                                               nq[2], dcc.as<double>());
        } else {
            const int *hp[9];
            for (int d = 0; d < 3; d++) {
                std::vector<int> b(nq[d]), l(nq[d]), m(op->blk[d].size());
                for (size_t k = 0; k < op->blk[d].size(); k++) {
                    const BlkInfo &B = op->blk[d][k];
                    m[k] = B.nq;
                    for (int q = 0; q < B.nq; q++) {
                        b[B.q0 + q] = (int)k;
                        l[B.q0 + q] = q;
                    }
                }
                YETI_TRY(upload(ctx, blk[d], b.data(), b.size()));
                YETI_TRY(upload(ctx, loc[d], l.data(), l.size()));
                YETI_TRY(upload(ctx, nqb[d], m.data(), m.size()));
                hp[d] = blk[d].as<int>();
                hp[3 + d] = loc[d].as<int>();
                hp[6 + d] = nqb[d].as<int>();
            }
            YETI_TRY(upload(ctx, ptrs, hp, 9));
            const int *const *dp = ptrs.as<const int *>();
            k_fd_diag_coef_blk<<<592, 256, 0, s>>>(op->coef64.as<double>(), op->qoff.as<int64_t>(),
                                                   dp, dp + 3, dp + 6, (int)op->blk[0].size(),
                                                   (int)op->blk[1].size(), nq[0], nq[1], nq[2],
                                                   dcc.as<double>());
        }
        count_launches(1);
        YETI_CUDA(cudaGetLastError());
        std::vector<double> cc((size_t)9 * n);
        YETI_CUDA(cudaMemcpyAsync(cc.data(), dcc.ptr, cc.size() * sizeof(double),
                                  cudaMemcpyDeviceToHost, s));
        YETI_CUDA(cudaStreamSynchronize(s));
        for (int c = 0; c < 3; c++) {
            std::vector<double> Mw[3], Kw[3];
            for (int d = 0; d < 3; d++) {
                Mw[d].assign(nq[d], 1.0);
                Kw[d].assign(nq[d], 1.0);
            }
            const double *ccp[3] = {&cc[(size_t)(3 * c) * n], &cc[(size_t)(3 * c + 1) * n],
                                    &cc[(size_t)(3 * c + 2) * n]};
            for (int sweep = 0; sweep < 2; sweep++) td_sweep(nq, ccp, Mw, Kw);
            for (int d = 0; d < 3; d++) {
                for (int q = 0; q < nq[d]; q++)
                    YETI_CHECK(Mw[d][q] > 0.0 && Kw[d][q] > 0.0 && std::isfinite(Mw[d][q]) &&
                                   std::isfinite(Kw[d][q]),
                               YETI_ENUMERIC, "fast diagonalisation 'TD': weight %g / %g",
                               Mw[d][q], Kw[d][q]);
                tdM[c][d] = Mw[d];
                tdK[c][d] = Kw[d];
            }
        }
    }
    struct Eig {
        std::vector<double> lam, U, kd, md;
    };
    // unweighted eigenpairs depend on (p, nel, lo, hi) only: operators set
    // up back to back (the serving loop's) share them through a bounded
    // process-wide cache; 'TD' ones are the operator's own
    static std::mutex g_eig_mtx;
    static std::map<std::tuple<int, int, int, int>, Eig> g_eig;
    static std::deque<std::tuple<int, int, int, int>> g_eig_order;
    constexpr size_t kEigCacheEntries = 512;
    std::map<std::tuple<int, int, int, int, int>, Eig> cache;
    Eig *E[3][3];
    for (int c = 0; c < 3; c++)
        for (int d = 0; d < 3; d++) {
            const int lo = F.lo[c][d], hi = lo + F.m[c][d];
            // 'TD' weights differ per component: no sharing between components
            auto key = std::make_tuple(op->p[d], op->nel[d], lo, hi, td ? 3 * c + d : -1);
            auto it = cache.find(key);
            if (it == cache.end() && !td) {
                std::lock_guard<std::mutex> lock(g_eig_mtx);
                auto g = g_eig.find(std::make_tuple(op->p[d], op->nel[d], lo, hi));
                if (g != g_eig.end()) it = cache.emplace(key, g->second).first;
            }
            if (it == cache.end()) {
                Eig e;
                std::vector<double> K, M;
                if (td)
                    wq_1d_matrices_weighted(R[d], lo, hi, tdM[c][d].data(), tdK[c][d].data(), K, M);
                else
                    wq_1d_matrices(R[d], lo, hi, K, M);
                const int m = hi - lo;
                e.kd.resize(m);
                e.md.resize(m);
                for (int i = 0; i < m; i++) {
                    e.kd[i] = K[(size_t)i * m + i];
                    e.md[i] = M[(size_t)i * m + i];
                }
                YETI_CHECK(gen_eig(m, K, M, e.lam, e.U), YETI_ENUMERIC,
                           "fast diagonalisation: eigen decomposition failed (direction %d)", d);
                if (!td) {
                    std::lock_guard<std::mutex> lock(g_eig_mtx);
                    const auto gk = std::make_tuple(op->p[d], op->nel[d], lo, hi);
                    if (g_eig.emplace(gk, e).second) {
                        g_eig_order.push_back(gk);
                        if (g_eig_order.size() > kEigCacheEntries) {
                            g_eig.erase(g_eig_order.front());
                            g_eig_order.pop_front();
                        }
                    }
                }
                it = cache.emplace(key, std::move(e)).first;
            }
            E[c][d] = &it->second;
        }
    // Lambda_c > 0 needs at least one direction without a zero eigenvalue
    for (int c = 0; c < 3; c++) {
        double lmin = 0.0;
        for (int d = 0; d < 3; d++)
            lmin += acoef[c][d] * *std::min_element(E[c][d]->lam.begin(), E[c][d]->lam.end());
        YETI_CHECK(lmin > 0.0, YETI_ENUMERIC,
                   "fast diagonalisation: separable operator of component %d is singular", c);
    }
    // device tables: G (U then U^T) per (c, d); a * lambda; 1-D diagonals
    std::vector<double> g64, dsc, kdmd;
    std::vector<float> g32;
    for (int c = 0; c < 3; c++)
        for (int d = 0; d < 3; d++) {
            const int m = F.m[c][d];
            const Eig &e = *E[c][d];
            add_matrices<double>(e.U, m, g64, F.goff[0][c][d]);
            if (f32) add_matrices<float>(e.U, m, g32, F.goff[1][c][d]);
            F.doff[c][d] = (int64_t)dsc.size();
            for (int i = 0; i < m; i++) dsc.push_back(acoef[c][d] * e.lam[i]);
            for (int i = 0; i < m; i++) kdmd.push_back(e.kd[i]);
            for (int i = 0; i < m; i++) kdmd.push_back(e.md[i]);
        }
    YETI_TRY(upload(ctx, F.g64, g64.data(), g64.size()));
    YETI_TRY(upload(ctx, F.d64, dsc.data(), dsc.size()));
    F.g32.release();
    F.d32.release();
    if (f32) {
        std::vector<float> df(dsc.begin(), dsc.end());
        YETI_TRY(upload(ctx, F.g32, g32.data(), g32.size()));
        YETI_TRY(upload(ctx, F.d32, df.data(), df.size()));
    }
    // scaling vector
    F.scaled = scaled;
    F.s64.release();
    F.s32.release();
    if (scaled) {
        DevBuf dk;
        YETI_TRY(upload(ctx, dk, kdmd.data(), kdmd.size()));
        YETI_TRY(F.s64.alloc(ctx, op->ndof * sizeof(double)));
        YETI_CUDA(cudaMemsetAsync(F.s64.ptr, 0, op->ndof * sizeof(double), s));
        if (f32) {
            YETI_TRY(F.s32.alloc(ctx, op->ndof * sizeof(float)));
            YETI_CUDA(cudaMemsetAsync(F.s32.ptr, 0, op->ndof * sizeof(float), s));
        }
        for (int c = 0; c < 3; c++) {
            // kdmd offsets: twice the dsc offsets (kd then md per block)
            k_fd_scaling<<<592, 256, 0, s>>>(
                op->diag.as<double>(), dk.as<double>(), F.s64.as<double>(),
                f32 ? F.s32.as<float>() : nullptr, make_int3(op->n[0], op->n[1], op->n[2]),
                op->ncp, F.lo[c][0], F.lo[c][1], F.lo[c][2], F.m[c][0], F.m[c][1], F.m[c][2], c,
                2 * F.doff[c][0], 2 * F.doff[c][1], 2 * F.doff[c][2], acoef[c][0], acoef[c][1],
                acoef[c][2]);
            count_launches(1);
        }
        YETI_CUDA(cudaGetLastError());
        YETI_CUDA(cudaStreamSynchronize(s));   // dk is freed on return
    }
    // intermediates and reduction partials
    YETI_TRY(F.t64.alloc(ctx, 2 * op->ndof * sizeof(double)));
    F.t32.release();
    if (f32) YETI_TRY(F.t32.alloc(ctx, 2 * op->ndof * sizeof(float)));
    F.max_grid = std::max(fd_plan_tiles<double>(F), fd_plan_tiles<float>(F));
    YETI_TRY(F.parts.alloc(ctx, (size_t)F.max_grid * sizeof(double)));
    // the tables were uploaded (and, on a stream-ordered context,
    // allocated) on the context's stream; solves may run on other streams
    YETI_CUDA(cudaStreamSynchronize(s));
    F.variant = variant;
    return YETI_OK;
}

template <class T> struct FdBufs;
template <> struct FdBufs<double> {
    static const double *g(const WQFdPlan &F) { return F.g64.as<double>(); }
    static const double *d(const WQFdPlan &F) { return F.d64.as<double>(); }
    static const double *s(const WQFdPlan &F) { return F.s64.as<double>(); }
    static double *t(const WQFdPlan &F) { return F.t64.as<double>(); }
};
template <> struct FdBufs<float> {
    static const float *g(const WQFdPlan &F) { return F.g32.as<float>(); }
    static const float *d(const WQFdPlan &F) { return F.d32.as<float>(); }
    static const float *s(const WQFdPlan &F) { return F.s32.as<float>(); }
    static float *t(const WQFdPlan &F) { return F.t32.as<float>(); }
};

template <class T, int AX, int EPI>
static int fd_pass(yeti_wq_op *op, FdArgs<T> a, bool bwd, cudaStream_t s) {
    const WQFdPlan &F = op->fd;
    int tot = 0, threads = 32;
    size_t smem = 0;
    // 16-byte copies of the lines: rows begin on 16 bytes, and where lines are
    // consecutive their runs along u are whole pieces
    constexpr int VEC = 16 / sizeof(T);
    bool vec = (reinterpret_cast<uintptr_t>(a.in) & 15) == 0 && op->n[0] % VEC == 0;
    for (int c = 0; c < 3; c++) {
        const int m = F.m[c][AX];
        const FdTile &t = F.tile[sizeof(T) == 4][EPI == 3 ? 3 : AX][c];
        YETI_CHECK(t.ctas > 0, YETI_EINVAL, "fast diagonalisation: no tiling for m=%d", m);
        a.nA[c] = t.nA;
        a.nL[c] = t.nL;
        a.ntA[c] = t.ntA;
        tot += t.ctas;
        a.cta_end[c] = tot;
        const int64_t off = F.goff[sizeof(T) == 4][c][AX];
        a.goff[c] = off + (bwd ? fd_matrix<T>(m) : 0);
        a.goff2[c] = off + fd_matrix<T>(m);
        smem = std::max(smem, t.smem);
        threads = std::max(std::max(threads, t.threads), kFdLeast<T>);
        vec = vec && (AX == 0 || F.m[c][0] % VEC == 0) && F.lo[c][0] % VEC == 0;
    }
    a.vec = vec;
    // every component's units fit `threads`.  The shared-memory opt-in (the
    // 48 KB default covers static plus dynamic memory) is set by
    // wq_fd_prepare on this device, outside any capture
    k_fd_pass<T, AX, EPI><<<tot, threads, smem, s>>>(a);
    count_launches(1);
    return YETI_OK;
}

// The fused u and v products of every w plane (forward or backward).
template <class T, int EPI>
static int fd_plane(yeti_wq_op *op, FdArgs<T> a, bool bwd, cudaStream_t s) {
    const WQFdPlan &F = op->fd;
    int tot = 0, threads = 32;
    size_t smem = 0;
    constexpr int VEC = 16 / sizeof(T);
    bool vec = (reinterpret_cast<uintptr_t>(a.in) & 15) == 0 && op->n[0] % VEC == 0;
    for (int c = 0; c < 3; c++) {
        const int mu = F.m[c][0], mv = F.m[c][1];
        const FdPlane &t = F.plane[sizeof(T) == 4][c];
        YETI_CHECK(t.ctas > 0, YETI_EINVAL, "fast diagonalisation: plane %dx%d does not fit", mu, mv);
        a.ntA[c] = t.nsplit;
        a.nA[c] = t.nA;
        a.nL[c] = t.nL;
        tot += t.ctas;
        a.cta_end[c] = tot;
        const int64_t *off = F.goff[sizeof(T) == 4][c];
        a.goff[c] = off[0] + (bwd ? fd_matrix<T>(mu) : 0);
        a.goff2[c] = off[1] + (bwd ? fd_matrix<T>(mv) : 0);
        smem = std::max(smem, t.smem);
        threads = std::max(threads, t.threads);
        vec = vec && F.lo[c][0] % VEC == 0;
    }
    a.vec = vec;
    k_fd_plane<T, EPI><<<tot, threads, smem, s>>>(a);
    count_launches(1);
    return YETI_OK;
}

// The fused plane pass pays off when its tile leaves room for two CTAs per
// SM (64^3: FP32, 79 KB, 22 us against two line passes of 13 us or more each;
// FP64, 158 KB, one CTA per SM, takes the line passes, 12.4 us each).
constexpr size_t kFdPlaneSmem = 100 * 1024;
template <class T>
static bool fd_planes_fit(const WQFdPlan &F) {
    for (int c = 0; c < 3; c++) {
        const FdPlane &t = F.plane[sizeof(T) == 4][c];
        if (t.ctas <= 0 || t.smem > kFdPlaneSmem) return false;
    }
    return true;
}

// The w pass can run fused (forward, division, backward in one CTA) when
// every component's w tile is a single row tile that fits.
template <class T>
static bool fd_w_fused(const WQFdPlan &F) {
    for (int c = 0; c < 3; c++)
        if (F.tile[sizeof(T) == 4][3][c].ctas <= 0) return false;
    return true;
}

template <class T>
int wq_fd_apply(yeti_wq_op *op, const T *in, T *out, const int *done, int red, T *p,
                CGScal *cg, cudaStream_t s, T *tmp, double *parts) {
    const WQFdPlan &F = op->fd;
    FdArgs<T> a;
    a.g = FdBufs<T>::g(F);
    a.dsc = FdBufs<T>::d(F);
    a.s = F.scaled ? FdBufs<T>::s(F) : nullptr;
    a.r = in;
    a.p = p;
    a.done = done;
    a.cg = cg;
    a.parts = parts ? parts : F.parts.as<double>();
    a.red = red;
    for (int d = 0; d < 3; d++) a.n[d] = op->n[d];
    a.ncp = op->ncp;
    for (int c = 0; c < 3; c++)
        for (int d = 0; d < 3; d++) {
            a.lo[c][d] = F.lo[c][d];
            a.m[c][d] = F.m[c][d];
            a.doff[c][d] = F.doff[c][d];
        }
    T *t0 = tmp ? tmp : FdBufs<T>::t(F), *t1 = t0 + op->ndof;
    a.in = in;
    if (F.scaled) {
        // t1 = s r on the free boxes (the first pass reads the boxes only)
        k_fd_scale_in<T><<<592, 256, 0, s>>>(in, a.s, t1, op->ndof, done);
        count_launches(1);
        a.in = t1;
    }
    if (fd_planes_fit<T>(F) && fd_w_fused<T>(F)) {
        // three launches: u and v forward per plane, w, u and v backward
        a.out = t0;
        YETI_TRY((fd_plane<T, 0>(op, a, false, s)));
        a.in = t0;
        a.out = t1;
        YETI_TRY((fd_pass<T, 2, 3>(op, a, false, s)));
        a.in = t1;
        a.out = out;
        YETI_TRY((fd_plane<T, 2>(op, a, true, s)));
        YETI_CUDA(cudaGetLastError());
        return YETI_OK;
    }
    a.out = t0;
    YETI_TRY((fd_pass<T, 0, 0>(op, a, false, s)));
    a.in = t0;
    a.out = t1;
    YETI_TRY((fd_pass<T, 1, 0>(op, a, false, s)));
    a.in = t1;
    a.out = t0;
    if (fd_w_fused<T>(F)) {
        YETI_TRY((fd_pass<T, 2, 3>(op, a, false, s)));
    } else {
        YETI_TRY((fd_pass<T, 2, 1>(op, a, false, s)));
        a.in = t0;
        a.out = t1;
        YETI_TRY((fd_pass<T, 2, 0>(op, a, true, s)));
        std::swap(t0, t1);
    }
    a.in = t0;
    a.out = t1;
    YETI_TRY((fd_pass<T, 1, 0>(op, a, true, s)));
    a.in = t1;
    a.out = out;
    YETI_TRY((fd_pass<T, 0, 2>(op, a, true, s)));
    YETI_CUDA(cudaGetLastError());
    return YETI_OK;
}

template int wq_fd_apply<double>(yeti_wq_op *, const double *, double *, const int *, int,
                                 double *, CGScal *, cudaStream_t, double *, double *);
template int wq_fd_apply<float>(yeti_wq_op *, const float *, float *, const int *, int, float *,
                                CGScal *, cudaStream_t, float *, double *);

int wq_fd_parts(const yeti_wq_op *op) { return op->fd.max_grid; }

}  // namespace yeti

using namespace yeti;

YETI_API int yeti_wq_fd_apply(yeti_wq_op *op, const void *r, void *z, int prec, int variant,
                              int mem) {
    YETI_CHECK(op && r && z, YETI_EINVAL, "yeti_wq_fd_apply: NULL argument");
    YETI_CHECK(prec == YETI_PREC_F64 || prec == YETI_PREC_F32, YETI_EINVAL,
               "yeti_wq_fd_apply: prec %d", prec);
    YETI_CHECK((variant & YETI_PCG_FD) && !(variant & ~(YETI_PCG_FD | YETI_PCG_FD_SCALED |
                                                       YETI_PCG_FD_UNIT | YETI_PCG_FD_TD)) &&
                   !((variant & YETI_PCG_FD_UNIT) && (variant & YETI_PCG_FD_TD)),
               YETI_EINVAL, "yeti_wq_fd_apply: variant %d", variant);
    DeviceGuard guard(op->ctx->device);
    const bool f32 = prec == YETI_PREC_F32;
    YETI_TRY(wq_fd_prepare(op, variant, f32));
    cudaStream_t s = op->ctx->stream;
    const size_t es = f32 ? sizeof(float) : sizeof(double);
    const size_t bytes = (size_t)op->ndof * es;
    DevBuf dr, dz;
    const void *rin = r;
    void *zout = z;
    if (mem == YETI_MEM_HOST) {
        YETI_TRY(dr.alloc(op->ctx, bytes));
        YETI_TRY(dz.alloc(op->ctx, bytes));
        YETI_CUDA(cudaMemcpyAsync(dr.ptr, r, bytes, cudaMemcpyHostToDevice, s));
        rin = dr.ptr;
        zout = dz.ptr;
    }
    YETI_CUDA(cudaMemsetAsync(zout, 0, bytes, s));
    if (f32)
        YETI_TRY(wq_fd_apply<float>(op, (const float *)rin, (float *)zout, nullptr, FD_NONE,
                                    nullptr, nullptr, s));
    else
        YETI_TRY(wq_fd_apply<double>(op, (const double *)rin, (double *)zout, nullptr, FD_NONE,
                                     nullptr, nullptr, s));
    if (mem == YETI_MEM_HOST)
        YETI_CUDA(cudaMemcpyAsync(z, zout, bytes, cudaMemcpyDeviceToHost, s));
    YETI_CUDA(cudaStreamSynchronize(s));
    return YETI_OK;
}
