// Sum-factorised U1 element stiffness: the same COO slots and values as the
// point-by-pair kernel of assemble_u1.cu (stiffmatrix.F90:130-225,
// UELMAT.f90:109-171), with the B^T D B contraction done direction by
// direction over the 1-D basis tables instead of pair by pair.  The sums run
// in another order, so the values agree with the reference to rounding
// (relative 1e-14 on the test meshes), not bit for bit.
//
// Factorisation
// -------------
// With N_a = N1_{i1}(q1) N2_{i2}(q2) N3_{i3}(q3) the B-spline product of
// local node a, W = sum_a w_a N_a and W_d = sum_a w_a dN_a/dxi_d, the
// physical gradient of the rational function R_a = w_a N_a / W is
//
//     dR_a/dx_r = w_a sum_kappa Phi^kappa_a(q) c^kappa_r(q),
//
// over the four kinds kappa = value, d/du, d/dv, d/dw of the tensor product
// (Phi^value = N_a, Phi^u = N1' N2 N3, ...) with the point coefficients
// c^{d}_r = Jinv[d][r] / W and c^{value}_r = -sum_d W_d Jinv[d][r] / W^2.
// For the isotropic D of stiffmatrix.F90:167-216 the 3x3 block of a node
// pair is
//
//     K_kl(a, b) = lam G_kl + mu G_lk + [k = l] mu (G_00 + G_11 + G_22),
//     G_rs(a, b) = sum_q dv(q) dR_a/dx_r dR_b/dx_s,
//
// so the nine integrals G_rs carry the element matrix; they are contracted
// along w, then v, then u.  After the w contraction the value and d/dw kinds
// share their factors in u and v (class 0), d/du is class 1 and d/dv class
// 2; after v only the kind along u (value or derivative) remains.  Each
// contraction runs one side (the row node a) and then the other (b).  For
// one pair (i3, j3) of w indices the steps cost about 81 g^3,
// 30 n2 g^3 + 27 n2^2 g^2 and 36 n1 n2^2 g + 18 n1^2 n2^2 g multiply-adds
// (n = p+1 functions, g Gauss points per direction); only the pairs
// i3 <= j3 are needed, the slots hold the upper triangle.
//
// One CTA per element.  Shared memory holds the point coefficients (13 per
// point), T1 = G_rs per class pair and (q1, q2), and T2, the 36 values of
// (rs, u-kind pair) together per (i2, j2, q1).
//
// What bounds it: the shared-memory reads beside the multiply-adds (the data
// path of shared memory is busy 75 % of the time where a thread has three
// column nodes), then the latency of short passes on few warps.  So the u
// contraction, the longest, gives a thread all nine G_rs of up to JT column
// nodes: 18 16-byte reads of T2 per q1 serve 36 + 18 JT multiply-adds, and the
// 3x3 blocks are formed where their sums are, nine slots in a row.  The w
// contraction of the next pair of layers shares its pass (two barriers per
// pair), a thread per row class reads a point's 13 coefficients once for the
// three column classes, and the rows and columns go out in whole lines by the
// warps that have no 1-D table to fill.  With a lane per r (blocks gathered by
// shuffles, three barriers, rows and columns beside the values in 4-byte
// stores) p=4 took 407,000 warp instructions per element, of which 66,000 are
// the multiply-adds.  Measured on B200: 12^3 elements of p=4 1470 -> 833 us (the 1.95 GB
// of the matrix take 0.3 ms), 16^3 of p=3 1471 -> 590 us, of p=2 348 -> 159 us, 6^3 of
// p=5 794 -> 456 us.
#include "nurbs.cuh"
#include "u1_model.cuh"

namespace yeti {

constexpr int kSfMaxG = 8;   // Gauss points per direction (template instances)

struct SfArgs {
    int n[3];        // functions per direction (p+1)
    int p[3];
    int nn;          // nodes
    int spaced;      // of the layout (sf_plan)
    const double *U[3];
    const double *gauss;   // 4 * g^3: weight, t1, t2, t3 (t3 fastest)
    const double *coords;
    const int32_t *ien;
    const double *w;
    const int32_t *span;
    const int64_t *slot;
    double lam, mu;
    double *kdata;
    int32_t *krow, *kcol;
};

// Shared memory of one CTA, in doubles: the 1-D tables, T2, T1, the point
// coefficients, weights, dofs.  The control-point coordinates (3 nn) are needed
// only by the per-point pass and share their space with T2/T1.  The blocks of
// 36 g values per (i2, j2) are spaced so that the (i2, j2) of a warp (i2 in
// steps of two doubles, j2 of eight) fall on different banks; spaced: 0 where
// that would not fit.
struct SfPlan {
    int sj, si;            // strides of j2 and i2 in T2
    int T2, T1, cq, we;    // offsets
    int total;
};
__host__ __device__ inline SfPlan sf_plan(const int n[3], int g, int spaced) {
    SfPlan P;
    const int nn = n[0] * n[1] * n[2];
    P.sj = 36 * g;
    if (spaced) P.sj += (8 - P.sj % 16 + 16) % 16;
    P.si = n[1] * P.sj;
    if (spaced) P.si += (2 - P.si % 16 + 16) % 16;
    P.T2 = 2 * g * (n[0] + n[1] + n[2]);
    P.T1 = P.T2 + n[1] * P.si;
    const int work = n[1] * P.si + 81 * g * g;
    P.cq = P.T2 + (work > 3 * nn ? work : 3 * nn);
    P.we = P.cq + 13 * g * g * g;
    P.total = P.we + nn + (nn + 1) / 2;
    return P;
}

// Threads of a CTA (the passes have 3 g^2, 9 n2 g and n1^2 n2^2 / JT tasks, n = g
// as a rule), CTAs on an SM that the registers must leave room for, and column
// nodes of a thread in the u contraction.  Few threads with all column nodes
// read the least up to five points; beyond, 9 JT sums leave no registers.  Tried
// (threads / CTAs / JT, us): p=2 96/6/2 192, 96/6/3 194, 64/8/3 176, 32/16/3 168,
// 32/12/3 162; p=3 160/4/2 617, 64/6/4 643, 96/5/4 594; p=4 256/2/3 1010,
// 128/3/3 953, 96/4/5 975, 128/3/5 838; p=5 256/2/6 590, 192/2/6 511, 256/2/3 457,
// 224/2/3 451.
template <int G>
struct SfShape {
    static constexpr int threads = G == 2 ? 64 : G == 3 ? 32 : G == 4 ? 96 : G == 5 ? 128 : 224;
    static constexpr int ctas = G == 2 ? 8 : G == 3 ? 12 : G == 4 ? 5 : G == 5 ? 3 : 2;
    static constexpr int JT = G == 2 ? 2 : G <= 5 ? G : 3;
    // lanes that share a point in the per-point pass
    static constexpr int lanes = 4 * G * G * G <= threads ? 4 : 2 * G * G * G <= threads ? 2 : 1;
};

// The nine values of a block, by 16-byte stores.
__device__ __forceinline__ void store9(double *o, const double (&v)[9]) {
    const int odd = (reinterpret_cast<uintptr_t>(o) & 15) != 0;
    if (odd) {
        o[0] = v[0];
#pragma unroll
        for (int i = 1; i < 9; i += 2) *reinterpret_cast<double2 *>(o + i) = make_double2(v[i], v[i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; i += 2) *reinterpret_cast<double2 *>(o + i) = make_double2(v[i], v[i + 1]);
        o[8] = v[8];
    }
}

__device__ __forceinline__ double det3(const double J[3][3]) {
    return J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) -
           J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
           J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
}

template <int G>
__global__ void __launch_bounds__(SfShape<G>::threads, SfShape<G>::ctas) k_u1_stiffness_sf(SfArgs a) {
    extern __shared__ __align__(16) double smem[];
    constexpr int g = G, gg = G * G, nq = G * G * G, JT = SfShape<G>::JT, NT = SfShape<G>::threads;
    const int n1 = a.n[0], n2 = a.n[1], n3 = a.n[2], nn = a.nn;
    const int n12 = n1 * n2;
    const SfPlan S = sf_plan(a.n, G, a.spaced);
    // (value, derivative) of function i at point q, [i][q]
    double2 *A1 = reinterpret_cast<double2 *>(smem), *A2 = A1 + n1 * g, *A3 = A2 + n2 * g;
    double *T2 = smem + S.T2;                 // [i2][j2][q1][rs][be][al]
    double *T1 = smem + S.T1;                 // [rs][ck ce][q1 q2]
    double *cq = smem + S.cq;                 // 13 nq: c[kind][r], dv
    double *we = smem + S.we;                 // nn
    int *dof = reinterpret_cast<int *>(we + nn);   // nn, first dof of each node
    double *xe = T2;                          // 3 nn, per-point pass only
    __shared__ double su1[3], su2[3];
    __shared__ int sni[3];
    const int e = blockIdx.x, tid = threadIdx.x;
    const int32_t *ien = a.ien + (size_t)e * nn;
    for (int i = tid; i < nn; i += NT) {
        const int cp = ien[i];
        dof[i] = 3 * cp;
        xe[3 * i] = a.coords[3 * cp];
        xe[3 * i + 1] = a.coords[3 * cp + 1];
        xe[3 * i + 2] = a.coords[3 * cp + 2];
        we[i] = a.w[(size_t)e * nn + i];
    }
    if (tid < 3) {
        const int ni = a.span[3 * e + tid];
        sni[tid] = ni;
        su1[tid] = a.U[tid][ni - 1];
        su2[tid] = a.U[tid][ni];
    }
    __syncthreads();
    // ---- 1-D tables: local index i uses the span's function p - i
    // (descending local node order of the reference's IEN)
    if (tid < 3 * g) {
        const int d = tid / g, q = tid - d * g;
        const int qq = d == 0 ? q * gg : (d == 1 ? q * g : q);
        const double t = a.gauss[4 * qq + 1 + d];
        const double xi = ((su2[d] - su1[d]) * t + (su2[d] + su1[d])) * 0.5;
        double N[kMaxDeg1], dN[kMaxDeg1];
        bspline_ders(sni[d], a.p[d], xi, a.U[d], N, dN);
        double2 *A = d == 0 ? A1 : (d == 1 ? A2 : A3);
        for (int i = 0; i < a.n[d]; i++) A[i * g + q] = make_double2(N[a.p[d] - i], dN[a.p[d] - i]);
    }
    // rows and columns of the slots, by the warps that have no table to fill
    const int64_t base_slot = a.slot[e];
    {
        constexpr int busy = NT > 32;
        if (tid >= 32 * busy)
            for_slots(nn, base_slot, (tid >> 5) - busy, NT / 32 - busy, [&](int64_t o, int i, int j, int kk, int ll) {
                a.krow[o] = dof[i] + kk;
                a.kcol[o] = dof[j] + ll;
            });
    }
    __syncthreads();
    // ---- per point: W, dW, x sums -> Jacobian, its inverse, dv, c; the four
    // kinds are shared out over L lanes, each sum keeps the order of the nodes
    constexpr int L = SfShape<G>::lanes, KN = 4 / L;
    for (int t = tid; t < (L * nq + 31) / 32 * 32; t += NT) {
        const int q = min(t / L, nq - 1), k0 = t % L * KN;
        const int q1 = q / gg, q2 = (q / g) % g, q3 = q % g;
        double s[KN][4];   // of kind k0 + k: sum of w Phi, of w Phi x_r
#pragma unroll
        for (int k = 0; k < KN; k++)
#pragma unroll
            for (int r = 0; r < 4; r++) s[k][r] = 0.0;
        int n = 0;
        for (int i3 = 0; i3 < n3; i3++) {
            const double2 c = A3[i3 * g + q3];
            for (int i2 = 0; i2 < n2; i2++) {
                const double2 b = A2[i2 * g + q2];
                double v23[KN];
#pragma unroll
                for (int k = 0; k < KN; k++) v23[k] = (k0 + k == 2 ? b.y : b.x) * (k0 + k == 3 ? c.y : c.x);
                for (int i1 = 0; i1 < n1; i1++, n++) {
                    const double2 d = A1[i1 * g + q1];
                    const double wn = we[n], x0 = xe[3 * n], x1 = xe[3 * n + 1], x2 = xe[3 * n + 2];
#pragma unroll
                    for (int k = 0; k < KN; k++) {
                        const double ph = (k0 + k == 1 ? d.y : d.x) * v23[k] * wn;
                        s[k][0] += ph;
                        s[k][1] += x0 * ph;
                        s[k][2] += x1 * ph;
                        s[k][3] += x2 * ph;
                    }
                }
            }
        }
        double W, Wd[3], P[4][3];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            double v[4];
#pragma unroll
            for (int r = 0; r < 4; r++)
                v[r] = L == 1 ? s[k % KN][r] : __shfl_sync(0xffffffffu, s[k % KN][r], k / KN, L);
            if (k == 0) W = v[0];
            else Wd[k - 1] = v[0];
#pragma unroll
            for (int r = 0; r < 3; r++) P[k][r] = v[r + 1];
        }
        if (t >= L * nq || t % L) continue;
        const double iW = 1.0 / W;
        double J[3][3], Ji[3][3];
        for (int r = 0; r < 3; r++)
            for (int d = 0; d < 3; d++) J[r][d] = (P[d + 1][r] - P[0][r] * Wd[d] * iW) * iW;
        const double det = det3(J), idet = 1.0 / det;
        Ji[0][0] = (J[1][1] * J[2][2] - J[1][2] * J[2][1]) * idet;
        Ji[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) * idet;
        Ji[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) * idet;
        Ji[1][0] = (J[1][2] * J[2][0] - J[1][0] * J[2][2]) * idet;
        Ji[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * idet;
        Ji[1][2] = (J[0][2] * J[1][0] - J[0][0] * J[1][2]) * idet;
        Ji[2][0] = (J[1][0] * J[2][1] - J[1][1] * J[2][0]) * idet;
        Ji[2][1] = (J[0][1] * J[2][0] - J[0][0] * J[2][1]) * idet;
        Ji[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * idet;
        // dv = w_q |det(J diag(h/2))| (shap.f90:155-178)
        const double hs = 0.125 * (su2[0] - su1[0]) * (su2[1] - su1[1]) * (su2[2] - su1[2]);
        double *c = cq + 13 * q;
        for (int r = 0; r < 3; r++) {
            c[r] = -(Wd[0] * Ji[0][r] + Wd[1] * Ji[1][r] + Wd[2] * Ji[2][r]) * iW * iW;
            for (int d = 0; d < 3; d++) c[3 * (d + 1) + r] = Ji[d][r] * iW;
        }
        c[12] = a.gauss[4 * q] * fabs(det * hs);
    }
    const double lam = a.lam, mu = a.mu;
    // ---- step 1 (w): T1[rs][ck ce][q1 q2] = sum_q3 dv Pa_r Pb_s, with
    // P^{class}_r(i3, q) = sum_{kinds of the class} A3[kind along w][i3][q3] c_r
    const auto w_sums = [&](int i3, int j3) {
        for (int t = tid; t < 3 * gg; t += NT) {
            const int ck = t / gg, q12 = t - ck * gg;
            double acc[3][9];
#pragma unroll
            for (int ce = 0; ce < 3; ce++)
#pragma unroll
                for (int k = 0; k < 9; k++) acc[ce][k] = 0.0;
#pragma unroll 1
            for (int q3 = 0; q3 < G; q3++) {
                const double *c = cq + 13 * (q12 * g + q3);
                const double2 ai = A3[i3 * g + q3], bj = A3[j3 * g + q3];
                const double dv = c[12];
                double v[4][3], pd[3];
#pragma unroll
                for (int k = 0; k < 4; k++)
#pragma unroll
                    for (int r = 0; r < 3; r++) v[k][r] = c[3 * k + r];
#pragma unroll
                for (int r = 0; r < 3; r++)
                    pd[r] = dv * (ck == 0 ? ai.x * v[0][r] + ai.y * v[3][r] : ai.x * (ck == 1 ? v[1][r] : v[2][r]));
#pragma unroll
                for (int ce = 0; ce < 3; ce++)
#pragma unroll
                    for (int s = 0; s < 3; s++) {
                        const double pb = ce == 0 ? bj.x * v[0][s] + bj.y * v[3][s] : bj.x * v[ce][s];
#pragma unroll
                        for (int r = 0; r < 3; r++) acc[ce][3 * r + s] += pd[r] * pb;
                    }
            }
#pragma unroll
            for (int rs = 0; rs < 9; rs++)
#pragma unroll
                for (int ce = 0; ce < 3; ce++) T1[(rs * 9 + 3 * ck + ce) * gg + q12] = acc[ce][rs];
        }
    };
    __syncthreads();
    w_sums(0, 0);
    for (int i3 = 0; i3 < n3; i3++)
        for (int j3 = i3; j3 < n3; j3++) {
            __syncthreads();
            // ---- step 2 (v): T2[i2][j2][q1][rs][be][al]; along u the classes
            // 0 and 2 carry the value kind, class 1 the derivative.  One task
            // per (rs, i2, q1) for both u-kinds al, so each A2 read serves six
            // multiply-adds.
            for (int t = tid; t < 9 * n2 * g; t += NT) {
                int r = t;
                const int q1 = r % g; r /= g;
                const int i2 = r % n2;
                const int rs = r / n2;
                const double *t1 = T1 + rs * 9 * gg + q1 * g;
                double V[2][3][G];   // V[al][ce][q2] = sum_{ck of u-kind al} A2 T1
#pragma unroll
                for (int q2 = 0; q2 < G; q2++) {
                    const double2 b = A2[i2 * g + q2];
#pragma unroll
                    for (int ce = 0; ce < 3; ce++) {
                        V[0][ce][q2] = b.x * t1[(0 * 3 + ce) * gg + q2] + b.y * t1[(2 * 3 + ce) * gg + q2];
                        V[1][ce][q2] = b.x * t1[(1 * 3 + ce) * gg + q2];
                    }
                }
                double *t2 = T2 + i2 * S.si + 36 * q1 + 4 * rs;
                // the pairs below the diagonal of equal layers are not used
                for (int j2 = i3 == j3 ? i2 : 0; j2 < n2; j2++) {
                    double s00 = 0.0, s01 = 0.0, s10 = 0.0, s11 = 0.0;   // s[al][be]
#pragma unroll
                    for (int q2 = 0; q2 < G; q2++) {
                        const double2 c = A2[j2 * g + q2];
                        s00 += c.x * V[0][0][q2];
                        s01 += c.x * V[0][1][q2];
                        s10 += c.x * V[1][0][q2];
                        s11 += c.x * V[1][1][q2];
                        s00 += c.y * V[0][2][q2];
                        s10 += c.y * V[1][2][q2];
                    }
                    double2 *o = reinterpret_cast<double2 *>(t2 + j2 * S.sj);
                    o[0] = make_double2(s00, s10);
                    o[1] = make_double2(s01, s11);
                }
            }
            __syncthreads();
            // the next pair's step 1 shares this pass: T1 is used up
            if (j3 + 1 < n3) w_sums(i3, j3 + 1);
            else if (i3 + 1 < n3) w_sums(i3 + 1, i3 + 1);
            // ---- steps 3 (u) and 4 (the COO slots): a thread per (i1, i2), j2
            // and up to JT j1; lanes run along the row nodes, whose blocks of
            // one column node are contiguous
            const int nch = (n1 + JT - 1) / JT, jt = (n1 + nch - 1) / nch;
            for (int t = tid; t < n12 * n2 * nch; t += NT) {
                const int a12 = t % n12;
                int r = t / n12;
                const int j2 = r % n2, jb = r / n2 * jt;
                const int i2 = a12 / n1, i1 = a12 - i2 * n1;
                if (i3 == j3 && j2 < i2) continue;   // below the diagonal
                double acc[JT][9];
#pragma unroll
                for (int j = 0; j < JT; j++)
#pragma unroll
                    for (int k = 0; k < 9; k++) acc[j][k] = 0.0;
                const double2 *t2 = reinterpret_cast<const double2 *>(T2 + i2 * S.si + j2 * S.sj);
#pragma unroll 1
                for (int q1 = 0; q1 < G; q1++, t2 += 18) {
                    const double2 ai = A1[i1 * g + q1];
                    double2 c[JT];
#pragma unroll
                    for (int j = 0; j < JT; j++) c[j] = A1[min(jb + j, n1 - 1) * g + q1];
#pragma unroll
                    for (int k = 0; k < 9; k++) {
                        const double2 x = t2[2 * k], y = t2[2 * k + 1];
                        const double u0 = ai.x * x.x + ai.y * x.y, u1 = ai.x * y.x + ai.y * y.y;
#pragma unroll
                        for (int j = 0; j < JT; j++) acc[j][k] += c[j].x * u0;
#pragma unroll
                        for (int j = 0; j < JT; j++) acc[j][k] += c[j].y * u1;
                    }
                }
                // K_kl = lam G_kl + mu G_lk + [k = l] mu (G_00 + G_11 + G_22)
                const int ia = a12 + n12 * i3;
                const double wa = we[ia];
#pragma unroll
                for (int j = 0; j < JT; j++) {
                    const int ib = jb + j + n1 * j2 + n12 * j3;
                    if (j >= jt || jb + j >= n1 || ia > ib) continue;
                    const double wab = wa * we[ib];
                    double K[9];   // [l][k]
#pragma unroll
                    for (int k = 0; k < 9; k++) acc[j][k] *= wab;
                    const double tr = mu * (acc[j][0] + acc[j][4] + acc[j][8]);
#pragma unroll
                    for (int l = 0; l < 3; l++)
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            K[3 * l + k] = lam * acc[j][3 * k + l] + mu * acc[j][3 * l + k];
                            if (k == l) K[3 * l + k] += tr;
                        }
                    double *o = a.kdata + base_slot + slot_col(ib) + 9LL * ia;
                    if (ia < ib) store9(o, K);
                    else {
#pragma unroll
                        for (int l = 0; l < 3; l++)
#pragma unroll
                            for (int k = 0; k <= l; k++) o[l * (l + 1) / 2 + k] = k == l ? K[4 * l] * 0.5 : K[3 * l + k];
                    }
                }
            }
        }
}

int launch_u1_stiffness_sf(yeti_ctx *ctx, const U1Patch &P, const double *coords,
                           double lam, double mu, double *kdata, int32_t *krow,
                           int32_t *kcol, size_t smem_cap) {
    YETI_CHECK(P.nq == P.ng * P.ng * P.ng && P.ng >= 2 && P.ng <= kSfMaxG, YETI_EUNSUPPORTED,
               "sum-factorised stiffness: needs a full tensor Gauss rule of at "
               "least 2 and at most %d points per direction (NBINT %d)", kSfMaxG, P.nq);
    SfArgs a;
    for (int d = 0; d < 3; d++) {
        a.p[d] = P.p[d];
        a.n[d] = P.p[d] + 1;
    }
    a.nn = P.nn;
    a.spaced = sf_plan(a.n, P.ng, 1).total * sizeof(double) <= smem_cap;
    const size_t smem = sf_plan(a.n, P.ng, a.spaced).total * sizeof(double);
    YETI_CHECK(smem <= smem_cap, YETI_EUNSUPPORTED,
               "sum-factorised stiffness: an element of degrees (%d,%d,%d) "
               "with %d Gauss points per direction does not fit shared memory",
               P.p[0], P.p[1], P.p[2], P.ng);
    a.U[0] = P.knots.as<double>();
    a.U[1] = a.U[0] + P.nkv[0];
    a.U[2] = a.U[1] + P.nkv[1];
    a.gauss = P.gauss.as<double>();
    a.coords = coords;
    a.ien = P.ien.as<int32_t>();
    a.w = P.w.as<double>();
    a.span = P.span.as<int32_t>();
    a.slot = P.slotd.as<int64_t>();
    a.lam = lam;
    a.mu = mu;
    a.kdata = kdata;
    a.krow = krow;
    a.kcol = kcol;
    void (*kern)(SfArgs) = nullptr;
    int threads = 0;
    switch (P.ng) {
#define YETI_CASE(GG)                     \
    case GG:                              \
        kern = k_u1_stiffness_sf<GG>;     \
        threads = SfShape<GG>::threads;   \
        break;
        YETI_CASE(2)
        YETI_CASE(3)
        YETI_CASE(4)
        YETI_CASE(5)
        YETI_CASE(6)
        YETI_CASE(7)
        YETI_CASE(8)
#undef YETI_CASE
        default: break;
    }
    YETI_CHECK(kern, YETI_EUNSUPPORTED, "sum-factorised stiffness: %d Gauss points per direction", P.ng);
    YETI_TRY(set_smem_optin((const void *)kern, ctx->device, smem, "sum-factorised stiffness element"));
    int64_t left = P.nactive, off = 0;
    while (left > 0) {   // grid.x limit
        const int64_t n = std::min<int64_t>(left, 1 << 30);
        SfArgs b = a;
        b.ien += off * P.nn;
        b.w += off * P.nn;
        b.span += off * 3;
        b.slot += off;
        kern<<<(unsigned)n, threads, smem, ctx->stream>>>(b);
        count_launches(1);
        YETI_CUDA(cudaGetLastError());
        left -= n;
        off += n;
    }
    return YETI_OK;
}

}  // namespace yeti
