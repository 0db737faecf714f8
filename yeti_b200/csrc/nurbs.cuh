// NURBS helpers shared by the Gauss-quadrature kernels (assembly, gradient).
#pragma once
#include <cmath>

#include "common.cuh"

namespace yeti {

constexpr int kMaxDeg = 8;            // maximum degree per direction
constexpr int kMaxDeg1 = kMaxDeg + 1;

// B-spline values N[0..p] and first derivatives dN[0..p] of the p+1
// functions nonzero on knot span `ni` (1-based, the reference's Nijk
// convention) at u: the Cox-de Boor triangle of The NURBS Book A2.3 with one
// derivative (the algorithm of dersbasisfuns.f90:30-131).
template <int MAXP>
__host__ __device__ __forceinline__ void bspline_ders_upto(int ni, int p, double u, const double *U,
                                                           double *N, double *dN) {
    double ndu[MAXP + 1][MAXP + 1];
    double left[MAXP + 2], right[MAXP + 2];
    ndu[0][0] = 1.0;
#pragma unroll
    for (int j = 1; j <= p; j++) {
        left[j] = u - U[ni - j];
        right[j] = U[ni + j - 1] - u;
        double saved = 0.0;
#pragma unroll
        for (int r = 0; r < j; r++) {
            ndu[j][r] = right[r + 1] + left[j - r];
            double temp = ndu[r][j - 1] / ndu[j][r];
            ndu[r][j] = saved + right[r + 1] * temp;
            saved = left[j - r] * temp;
        }
        ndu[j][j] = saved;
    }
#pragma unroll
    for (int j = 0; j <= p; j++) N[j] = ndu[j][p];
    // first derivatives in the reciprocal form of the reference's k-loop
    // (dersbasisfuns.f90:79-124 with nders = 1)
#pragma unroll
    for (int r = 0; r <= p; r++) {
        double d = 0.0;
        if (p >= 1) {
            if (r >= 1) {
                double a = 1.0 / ndu[p][r - 1];
                d = a * ndu[r - 1][p - 1];
            }
            if (r <= p - 1) {
                double a = -1.0 / ndu[p][r];
                d = d + a * ndu[r][p - 1];
            }
        }
        dN[r] = d * (double)p;
    }
}
__host__ __device__ inline void bspline_ders(int ni, int p, double u, const double *U, double *N,
                                             double *dN) {
    bspline_ders_upto<kMaxDeg>(ni, p, u, U, N, dN);
}
// The same, the triangle of degrees 1..4 in registers.
__device__ inline void bspline_ders_fast(int ni, int p, double u, const double *U, double *N,
                                         double *dN) {
    switch (p) {
        case 1: bspline_ders_upto<1>(ni, 1, u, U, N, dN); break;
        case 2: bspline_ders_upto<2>(ni, 2, u, U, N, dN); break;
        case 3: bspline_ders_upto<3>(ni, 3, u, U, N, dN); break;
        case 4: bspline_ders_upto<4>(ni, 4, u, U, N, dN); break;
        default: bspline_ders(ni, p, u, U, N, dN);
    }
}

// Rational basis R[nn] and its parametric derivatives dR[3 a + i] of one
// element at xi: the tensor product with reversed 1-D indices (the
// descending local node order of the reference's IEN), times the element's
// weights, then divided by their sum (evalnurbs,
// src/yeti_iga/main/evaluatenurbsfcts.f:94-209, in its operation order).
__device__ inline void nurbs_eval_elem(int p0, int p1, int p2, const double *U0,
                                       const double *U1, const double *U2, int nn,
                                       const int *ni, const double *xi, const double *we,
                                       double *R, double *dR) {
    double FN[kMaxDeg1], dFN[kMaxDeg1], FM[kMaxDeg1], dFM[kMaxDeg1], FL[kMaxDeg1],
        dFL[kMaxDeg1];
    bspline_ders(ni[0], p0, xi[0], U0, FN, dFN);
    bspline_ders(ni[1], p1, xi[1], U1, FM, dFM);
    bspline_ders(ni[2], p2, xi[2], U2, FL, dFL);
    int n = 0;
    double S = 0.0, sx0 = 0.0, sx1 = 0.0, sx2 = 0.0;
    for (int k = 0; k <= p2; k++)
        for (int j = 0; j <= p1; j++)
            for (int i = 0; i <= p0; i++, n++) {
                R[n] = FN[p0 - i] * FM[p1 - j] * FL[p2 - k] * we[n];
                S = S + R[n];
                dR[3 * n] = dFN[p0 - i] * FM[p1 - j] * FL[p2 - k] * we[n];
                sx0 = sx0 + dR[3 * n];
                dR[3 * n + 1] = FN[p0 - i] * dFM[p1 - j] * FL[p2 - k] * we[n];
                sx1 = sx1 + dR[3 * n + 1];
                dR[3 * n + 2] = FN[p0 - i] * FM[p1 - j] * dFL[p2 - k] * we[n];
                sx2 = sx2 + dR[3 * n + 2];
            }
    const double inv = 1.0 / S;
    const double sx[3] = {sx0, sx1, sx2};
    for (int q = 0; q < nn; q++) {
        R[q] = R[q] * inv;
        for (int i = 0; i < 3; i++) dR[3 * q + i] = (dR[3 * q + i] - R[q] * sx[i]) * inv;
    }
}

constexpr int kBasisQS = 13;              // scalars per point of basis_chunk

// 1-D rows of an element (doubles): values and derivatives of the p+1
// functions at the ng Gauss points of each direction.
__host__ __device__ inline int basis_rows_doubles(int ng) { return 6 * ng * kMaxDeg1; }

// The 1-D B-spline rows of an element (shap.f90:75-90): the Gauss points are
// a tensor grid (point q at (q / ng^2, q / ng % ng, q % ng)), so a row depends
// on a point's index along its direction only, and 3 ng evaluations serve
// all the points (one per point and direction took 3 ng^3).  Row g of
// direction d: values at rows + ((d ng + g) 2) kMaxDeg1, derivatives
// kMaxDeg1 further.  nodes[n] = i | j << 8 | k << 16 of local node n.
__device__ inline void basis_rows(const int pd[3], const double *const Ud[3], const int *sni,
                                  const double *su1, const double *su2, const double *gauss,
                                  int ng, int nn, double *rows, int *nodes) {
    for (int t = threadIdx.x; t < 3 * ng; t += blockDim.x) {
        const int d = t / ng, g = t - d * ng;
        const int q = d == 0 ? g * ng * ng : d == 1 ? g * ng : g;
        const double tq = gauss[4 * q + 1 + d];
        const double xi = ((su2[d] - su1[d]) * tq + (su2[d] + su1[d])) * 0.5;
        double *f = rows + (size_t)t * 2 * kMaxDeg1;
        bspline_ders_fast(sni[d], pd[d], xi, Ud[d], f, f + kMaxDeg1);
    }
    for (int n = threadIdx.x; n < nn; n += blockDim.x) {
        const int i = n % (pd[0] + 1), j = (n / (pd[0] + 1)) % (pd[1] + 1);
        nodes[n] = i | j << 8 | (n / ((pd[0] + 1) * (pd[1] + 1))) << 16;
    }
}

// Stage A of the Gauss kernels for a chunk of points q0..q0+nqc-1
// (shap.f90:75-178, evalnurbs, evaluatenurbsfcts.f:94-209): the rational
// numerators R0[ql rs + n] (R0 == nullptr: not kept) and dR/dxi at
// dR[ql ds + 3 n + c] of every (point, node), the per-point sums of the
// derivative numerators (qs[0..2]), 1/S (qs[3]) and dx/dxi
// (qs[4 + 3 r + c]), at a stride of qss >= kBasisQS per point (odd: no bank
// conflicts).  The products of every
// (point, node) are formed in parallel, a warp per point and its lanes over
// the nodes; each sum over the nodes stays one thread's loop in node order,
// so the values are those of the point-serial evaluation bit for bit.  The
// threads of a warp sum the same entry of consecutive points: ds should not
// be a multiple of 16 doubles (32 banks).  Barriers on entry (rows, nodes)
// and on return.
__device__ inline void basis_chunk(const int pd[3], const double *rows, const int *nodes, int ng,
                                   int q0, int nqc, int nn, const double *xe, const double *we,
                                   double *R0, int rs, double *dR, int ds, double *qs, int qss) {
    const int tid = threadIdx.x, nth = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, nwarp = nth >> 5;
    struct Rows {
        const double *u, *v, *w;
    };
    auto at = [&](int q) -> Rows {
        const int g2 = q / ng, g0 = g2 / ng;
        auto row = [&](int d, int g) { return rows + (d * ng + g) * 2 * kMaxDeg1 + pd[d]; };
        return {row(0, g0), row(1, g2 - g0 * ng), row(2, q - g2 * ng)};
    };
    // numerator of node n at rows f, as FN * FM * FL * w
    auto num = [&](const Rows &f, int n) {
        const int c = nodes[n];
        return f.u[-(c & 255)] * f.v[-(c >> 8 & 255)] * f.w[-(c >> 16)] * we[n];
    };
    __syncthreads();
    // A1: the numerator products of every (point, node)
    for (int ql = warp; ql < nqc; ql += nwarp) {
        const Rows f = at(q0 + ql);
        for (int n = lane; n < nn; n += 32) {
            const int c = nodes[n], i = -(c & 255), j = -(c >> 8 & 255), k = -(c >> 16);
            const double FN = f.u[i], dFN = f.u[kMaxDeg1 + i];
            const double FM = f.v[j], dFM = f.v[kMaxDeg1 + j];
            const double FL = f.w[k], dFL = f.w[kMaxDeg1 + k];
            const double wa = we[n];
            if (R0) R0[(size_t)ql * rs + n] = FN * FM * FL * wa;
            double *d = dR + (size_t)ql * ds + 3 * n;
            d[0] = dFN * FM * FL * wa;
            d[1] = FN * dFM * FL * wa;
            d[2] = FN * FM * dFL * wa;
        }
    }
    __syncthreads();
    // A2: the sums over the nodes (one thread per (sum, point), node order)
    for (int t = tid; t < 4 * nqc; t += nth) {
        const int c = t / nqc, ql = t - c * nqc;
        double acc = 0.0;
        if (c == 3) {
            const Rows f = at(q0 + ql);
#pragma unroll 4
            for (int n = 0; n < nn; n++) acc += num(f, n);
            qs[(size_t)ql * qss + 3] = 1.0 / acc;
        } else {
            const double *d = dR + (size_t)ql * ds + c;
#pragma unroll 8
            for (int n = 0; n < nn; n++) acc += d[3 * n];
            qs[(size_t)ql * qss + c] = acc;
        }
    }
    __syncthreads();
    // A3: rational derivatives dR/dxi of every (point, node)
    for (int ql = warp; ql < nqc; ql += nwarp) {
        const Rows f = at(q0 + ql);
        const double *sq = qs + (size_t)ql * qss;
        const double s0 = sq[0], s1 = sq[1], s2 = sq[2], inv = sq[3];
        for (int n = lane; n < nn; n += 32) {
            const double R = num(f, n) * inv;
            double *d = dR + (size_t)ql * ds + 3 * n;
            d[0] = (d[0] - R * s0) * inv;
            d[1] = (d[1] - R * s1) * inv;
            d[2] = (d[2] - R * s2) * inv;
        }
    }
    __syncthreads();
    // A4: dx/dxi, one thread per (entry, point), node order
    for (int t = tid; t < 9 * nqc; t += nth) {
        const int rc = t / nqc, ql = t - rc * nqc, r = rc / 3, c = rc - 3 * r;
        const double *d = dR + (size_t)ql * ds + c;
        double acc = 0.0;
#pragma unroll 8
        for (int n = 0; n < nn; n++) acc += xe[3 * n + r] * d[3 * n];
        qs[(size_t)ql * qss + 4 + rc] = acc;
    }
    __syncthreads();
}

// Gauss-Legendre nodes/weights of order n on [-1, 1] (ascending): roots of
// the Legendre polynomial P_n by Newton iteration on its recurrence.
void gauss_legendre_host(int n, double *x, double *w);

// Volume rule with the reference's ordering (GaussLegendre.f90:175-187):
// g[4q] = weight, g[4q+1..3] = parent coordinates, xi1 slowest.
void gauss_volume_host(int n, std::vector<double> &g);
// Face rule of face 1..6 (GaussLegendre.f90:217-270).
void gauss_face_host(int n, int face, std::vector<double> &g);

}  // namespace yeti
