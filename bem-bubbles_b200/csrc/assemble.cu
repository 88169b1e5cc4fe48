// Dense collocation assembly of G (single layer) and H (double layer) in FP64.
//
// Replaces ColocSim::assemble_matrices (Bem/Simulation/ColocSim.cpp:21-110) with the per-pair
// integrals of Integrator::integrate_Lin_coloc_local[_mir] (Bem/Integration/Integrator.cpp:237-283):
//   * regular pairs (vertex i not on triangle t): 7-point rule on the triangle
//     (integrate_disjoint_coloc[_mir], Integrator.hpp:471-513, kernel Integrator.hpp:116-119);
//   * singular pairs (i on t): polar rule with the analytic radial integral and 7-point Gauss in
//     the angle (integrate_identical_coloc[_mir], Integrator.cpp:13-89);
//   * the "4 pi rule" diagonal H(i,i) -= 4 pi + sum_j H(i,j) (ColocSim.cpp:85-97).
//
// Tiling (B200): a CTA owns one column group (cg vertices, i.e. cg columns of G and H) and a block
// of collocation rows, one row per thread.  It walks the triangles incident to its
// vertices in increasing index order (the reference's per-column summation order), with the
// triangle records staged in shared memory and read as broadcasts, and accumulates the cg columns
// of its rows in shared memory.  Column writes are coalesced (column-major, consecutive rows).
// No atomics: every entry is summed by exactly one thread in a fixed order, so the result is
// bit-reproducible run to run.  The same pass produces the per-group partial row sums of H and
// partial H*phi, so the 4 pi diagonal and the right-hand side need no second read of H.
#include <math.h>
#include <mutex>

#include "ctx.h"
#include "rsqrt.cuh"

namespace bemb {

// c[q][k] = w_q * basis_k(u_q, v_q) for the 7-point rule mapped to the 45-degree unit triangle
// (u, v) = (qx + qy, qy), basis (1-u, u-v, v) (ResultTypes.hpp:111-117); u_q, v_q; Gauss-7 angle data.
__constant__ double c_qc[7][3];
__constant__ double c_quv[7][2];
__constant__ double c_gcos[7], c_gsin[7], c_gw[7];
// The 7-point rule is symmetric: the centroid plus two orbits of three points whose barycentric
// weights are rotations of (alpha, beta, beta).  With S the orbit sum of kernel values and
// g_k the orbit point whose alpha sits on vertex k, sum_q w_q basis_k(q) K(q) =
//   C + dA * gA_k + dB * gB_k,   C = w0 b0 K(centroid) + cA*S_A + cB*S_B.
// c_orb = {w0*b0, cA, dA, cB, dB}.
__constant__ double c_orb[5];
// The same orbits for the patch kernel: beta and alpha - beta, and the weights of the centroid and the orbits.
__constant__ double c_pbeta[2], c_pdiff[2], c_pw[3];

// Reference tables (quadrature.hpp:30-38 gauss_7, :88-96 quadrature_7) in the forms the kernels use:
// per point the basis weights (1-u, u-v, v) * w of the triangle rule applied as (x+y, y) on the
// unit triangle, and cos, sin and weight of the Gauss angles on (0, pi/4).
void quad_tables(QuadTables& t) {
    const double Q[7][3] = {{0.33333333333333333, 0.33333333333333333, 0.22500000000000000 * 0.5},
                            {0.79742698535308720, 0.10128650732345633, 0.12593918054482717 * 0.5},
                            {0.10128650732345633, 0.79742698535308720, 0.12593918054482717 * 0.5},
                            {0.10128650732345633, 0.10128650732345633, 0.12593918054482717 * 0.5},
                            {0.05971587178976981, 0.47014206410511505, 0.13239415278850616 * 0.5},
                            {0.47014206410511505, 0.05971587178976981, 0.13239415278850616 * 0.5},
                            {0.47014206410511505, 0.47014206410511505, 0.13239415278850616 * 0.5}};
    const double GL[7][2] = {{0.5 * (1.0 + 0.0000000000000000), 0.5 * 0.4179591836734694},
                             {0.5 * (1.0 + 0.4058451513773972), 0.5 * 0.3818300505051189},
                             {0.5 * (1.0 - 0.4058451513773972), 0.5 * 0.3818300505051189},
                             {0.5 * (1.0 - 0.7415311855993945), 0.5 * 0.2797053914892766},
                             {0.5 * (1.0 + 0.7415311855993945), 0.5 * 0.2797053914892766},
                             {0.5 * (1.0 - 0.9491079123427585), 0.5 * 0.1294849661688697},
                             {0.5 * (1.0 + 0.9491079123427585), 0.5 * 0.1294849661688697}};
    for (int q = 0; q < 7; ++q) {
        double u = Q[q][0] + Q[q][1], v = Q[q][1], w = Q[q][2];
        t.quv[q][0] = u;
        t.quv[q][1] = v;
        t.w[q] = w;
        t.qc[q][0] = (1.0 - u) * w;
        t.qc[q][1] = (u - v) * w;
        t.qc[q][2] = v * w;
        double th = GL[q][0] * 0.78539816339744830962;
        t.gc[q] = cos(th);
        t.gs[q] = sin(th);
        t.gw[q] = GL[q][1];
    }
    // orbit form: point 0 is the centroid; points 3,1,2 carry alpha on vertex 0,1,2 (orbit A) and
    // points 6,4,5 (orbit B), with barycentric coordinates (1-u, u-v, v)
    const double w0 = Q[0][2], wA = Q[1][2], wB = Q[4][2];
    const double aA = 1.0 - (Q[3][0] + Q[3][1]), bA = Q[3][1];  // point 3: (alpha, beta, beta)
    const double aB = 1.0 - (Q[6][0] + Q[6][1]), bB = Q[6][1];  // point 6
    const double orb[5] = {w0 * (1.0 / 3.0), wA * bA, wA * (aA - bA), wB * bB, wB * (aB - bB)};
    for (int k = 0; k < 5; ++k) t.orb[k] = orb[k];
    // quadrature_19 (quadrature.hpp:126-146), the rule of compute_exterior_pot (LinLinSim.cpp:455)
    const double Q19[19][3] = {{0.33333333333333331, 0.33333333333333331, 9.71357962827961025e-2 * 0.5},
                               {2.06349616025259287e-2, 0.48968251919873701, 3.13347002271398278e-2 * 0.5},
                               {0.48968251919873701, 2.06349616025259287e-2, 3.13347002271398278e-2 * 0.5},
                               {0.48968251919873701, 0.48968251919873701, 3.13347002271398278e-2 * 0.5},
                               {0.12582081701412900, 0.43708959149293553, 7.78275410047754301e-2 * 0.5},
                               {0.43708959149293553, 0.12582081701412900, 7.78275410047754301e-2 * 0.5},
                               {0.43708959149293553, 0.43708959149293553, 7.78275410047754301e-2 * 0.5},
                               {0.62359292876193562, 0.18820353561903219, 7.96477389272090969e-2 * 0.5},
                               {0.18820353561903219, 0.62359292876193562, 7.96477389272090969e-2 * 0.5},
                               {0.18820353561903219, 0.18820353561903219, 7.96477389272090969e-2 * 0.5},
                               {0.91054097321109406, 4.47295133944529688e-2, 2.55776756586981006e-2 * 0.5},
                               {4.47295133944529688e-2, 0.91054097321109406, 2.55776756586981006e-2 * 0.5},
                               {4.47295133944529688e-2, 4.47295133944529688e-2, 2.55776756586981006e-2 * 0.5},
                               {0.74119859878449801, 3.68384120547362581e-2, 4.32835393772893970e-2 * 0.5},
                               {0.74119859878449801, 0.22196298916076573, 4.32835393772893970e-2 * 0.5},
                               {3.68384120547362581e-2, 0.74119859878449801, 4.32835393772893970e-2 * 0.5},
                               {3.68384120547362581e-2, 0.22196298916076573, 4.32835393772893970e-2 * 0.5},
                               {0.22196298916076573, 0.74119859878449801, 4.32835393772893970e-2 * 0.5},
                               {0.22196298916076573, 3.68384120547362581e-2, 4.32835393772893970e-2 * 0.5}};
    for (int q = 0; q < 19; ++q) {
        t.q19[q][0] = Q19[q][0] + Q19[q][1];
        t.q19[q][1] = Q19[q][1];
        t.q19[q][2] = Q19[q][2];
    }
}

static void upload_constants() {
    static std::atomic<uint64_t> done{0};
    once_per_device(done, [] {
        QuadTables t;
        quad_tables(t);
        double pbeta[2], pdiff[2];
        for (int o = 0; o < 2; ++o) {
            const double* uv = t.quv[o ? 6 : 3];  // alpha on vertex 0: (alpha, beta, beta)
            pbeta[o] = uv[1];
            pdiff[o] = (1.0 - uv[0]) - uv[1];
        }
        const double pw[3] = {t.w[0], t.w[3], t.w[6]};
        return cudaMemcpyToSymbol(c_pbeta, pbeta, sizeof(pbeta)) == cudaSuccess &&
               cudaMemcpyToSymbol(c_pdiff, pdiff, sizeof(pdiff)) == cudaSuccess &&
               cudaMemcpyToSymbol(c_pw, pw, sizeof(pw)) == cudaSuccess &&
               cudaMemcpyToSymbol(c_orb, t.orb, sizeof(t.orb)) == cudaSuccess &&
               cudaMemcpyToSymbol(c_qc, t.qc, sizeof(t.qc)) == cudaSuccess &&
               cudaMemcpyToSymbol(c_quv, t.quv, sizeof(t.quv)) == cudaSuccess &&
               cudaMemcpyToSymbol(c_gcos, t.gc, sizeof(t.gc)) == cudaSuccess &&
               cudaMemcpyToSymbol(c_gsin, t.gs, sizeof(t.gs)) == cudaSuccess &&
               cudaMemcpyToSymbol(c_gw, t.gw, sizeof(t.gw)) == cudaSuccess;
    });
}

// Per-triangle record: Interpolator (Interpolator.hpp:15-37) quantities and what the 7-point rule
// needs of the quadrature points y_q = a + w_q, w_q = u_q*ab + v_q*bc.  For a row x,
//   |y_q - x|^2 = |a - x|^2 + u_q (a - x).2ab + v_q (a - x).2bc + |w_q|^2,
// so a pair costs three dot products with a - x and then two FMAs and an add per point.  Layout:
// a (0-2), 2ab (3-5), 2bc (6-8), |w_q|^2 (9-15), y_q.x (16-22, for the wall image), unit normal
// (23-25), area (26), plane offset a.n (27).
__global__ void k_triangle_records(int M, const double* __restrict__ x, const int* __restrict__ tri,
                                   double* __restrict__ rec) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= M) return;
    int ia = tri[3 * t], ib = tri[3 * t + 1], ic = tri[3 * t + 2];
    double ax = x[3 * ia], ay = x[3 * ia + 1], az = x[3 * ia + 2];
    double abx = x[3 * ib] - ax, aby = x[3 * ib + 1] - ay, abz = x[3 * ib + 2] - az;
    double bcx = x[3 * ic] - x[3 * ib], bcy = x[3 * ic + 1] - x[3 * ib + 1], bcz = x[3 * ic + 2] - x[3 * ib + 2];
    double nx = aby * bcz - abz * bcy, ny = abz * bcx - abx * bcz, nz = abx * bcy - aby * bcx;
    double area = sqrt(nx * nx + ny * ny + nz * nz);
    double ia_ = 1.0 / area;
    double* r = rec + (size_t)t * REC;
    r[0] = ax;
    r[1] = ay;
    r[2] = az;
    r[3] = 2.0 * abx;
    r[4] = 2.0 * aby;
    r[5] = 2.0 * abz;
    r[6] = 2.0 * bcx;
    r[7] = 2.0 * bcy;
    r[8] = 2.0 * bcz;
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        const double u = c_quv[q][0], v = c_quv[q][1];
        const double wx = u * abx + v * bcx, wy = u * aby + v * bcy, wz = u * abz + v * bcz;
        r[9 + q] = wx * wx + wy * wy + wz * wz;
        r[16 + q] = ax + wx;
    }
    const double unx = nx * ia_, uny = ny * ia_, unz = nz * ia_;
    r[23] = unx;
    r[24] = uny;
    r[25] = unz;
    r[26] = area;
    // plane offset a.n: every quadrature point y_q satisfies y_q.n = a.n, so (y_q - x).n is one
    // number per (row, triangle) pair
    r[27] = ax * unx + ay * uny + az * unz;
}

// Orbit-form basis sums of the 7 kernel values k[0..6] (see c_orb): out_k = C + dA*kA_k + dB*kB_k.
__device__ __forceinline__ void orbit_sums(const double* k, double& o0, double& o1, double& o2) {
    const double SA = (k[1] + k[2]) + k[3], SB = (k[4] + k[5]) + k[6];
    const double C = fma(c_orb[0], k[0], fma(c_orb[1], SA, __dmul_rn(c_orb[3], SB)));
    o0 = fma(c_orb[2], k[3], fma(c_orb[4], k[6], C));
    o1 = fma(c_orb[2], k[1], fma(c_orb[4], k[4], C));
    o2 = fma(c_orb[2], k[2], fma(c_orb[4], k[5], C));
}

// Basis sums of one regular pair.  G_k = g_k * area; H_k = h_k * sh (+ m_k * sm with the wall image).
// The accumulation into the shared-memory sums is written with explicit fused multiply-adds, so every
// kernel that inlines this code produces the same bits (no contraction left to the compiler).
struct PairSums {
    double g[3], h[3], m[3];
    double area, sh, sm;
};

// Regular 7-point rule of one (row, triangle) pair.  All quadrature points lie in the triangle's
// plane, so (y_q - x).n = n.a - n.x is hoisted out of the quadrature loop (and likewise for the image
// triangle).
template <bool MIRROR>
__device__ __forceinline__ void regular_pair(const double* __restrict__ r, double xi0, double xi1, double xi2,
                                             PairSums& p) {
    const double nx = r[23], ny = r[24], nz = r[25], area = r[26], dt = r[27];
    const double xn_yz = fma(xi1, ny, __dmul_rn(xi2, nz));
    const double dn = dt - fma(xi0, nx, xn_yz);  // (y - x).n
    const double ax = r[0] - xi0, ay = r[1] - xi1, az = r[2] - xi2;
    const double A = fma(ax, ax, fma(ay, ay, __dmul_rn(az, az)));
    const double B = fma(ax, r[3], fma(ay, r[4], __dmul_rn(az, r[5])));
    const double C = fma(ax, r[6], fma(ay, r[7], __dmul_rn(az, r[8])));
    const double x4 = 4.0 * xi0;
    double kg[7], kh[7], km[7];
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        const double r2 = fma(B, c_quv[q][0], fma(C, c_quv[q][1], A + r[9 + q]));
        const double inv = rsqrt_fp64(r2);
        kg[q] = inv;
        kh[q] = __dmul_rn(__dmul_rn(inv, inv), inv);
        if (MIRROR) {
            // image point (-y.x, y.y, y.z), image normal (-n.x, n.y, n.z) (Integrator.hpp:211-229):
            // |y' - x|^2 = |y - x|^2 + 4 x.x y.x
            const double inv2 = rsqrt_fp64(fma(x4, r[16 + q], r2));
            kg[q] += inv2;
            km[q] = __dmul_rn(__dmul_rn(inv2, inv2), inv2);
        }
    }
    orbit_sums(kg, p.g[0], p.g[1], p.g[2]);
    orbit_sums(kh, p.h[0], p.h[1], p.h[2]);
    p.area = area;
    p.sh = -__dmul_rn(dn, area);
    if (MIRROR) {
        orbit_sums(km, p.m[0], p.m[1], p.m[2]);
        // (y' - x).n' = n.a - (-x.x n.x + x.y n.y + x.z n.z)
        p.sm = -__dmul_rn(dt - fma(-xi0, nx, xn_yz), area);
    } else {
        p.m[0] = p.m[1] = p.m[2] = 0.0;
        p.sm = 0.0;
    }
}

template <bool MIRROR>
__device__ __forceinline__ double add_h(const PairSums& p, int k, double acc) {
    if (!MIRROR) return fma(p.h[k], p.sh, acc);
    return __dadd_rn(acc, fma(p.m[k], p.sm, __dmul_rn(p.h[k], p.sh)));
}

// Singular pair: row i is vertex `shift` of triangle (ta, tb, tc).  gg[m], hh[m]: the G and H
// contributions to the column of the triangle's vertex at position (m + shift) % 3.
template <bool MIRROR>
__device__ __forceinline__ void singular_sums(const double* __restrict__ x, int ta, int tb, int tc, int shift,
                                              double gg[3], double hh[3]) {
    const int r0 = shift == 0 ? ta : (shift == 1 ? tb : tc);
    const int r1 = shift == 0 ? tb : (shift == 1 ? tc : ta);
    const int r2 = shift == 0 ? tc : (shift == 1 ? ta : tb);
    double ax = x[3 * r0], ay = x[3 * r0 + 1], az = x[3 * r0 + 2];
    double abx = x[3 * r1] - ax, aby = x[3 * r1 + 1] - ay, abz = x[3 * r1 + 2] - az;
    double bcx = x[3 * r2] - x[3 * r1], bcy = x[3 * r2 + 1] - x[3 * r1 + 1], bcz = x[3 * r2 + 2] - x[3 * r1 + 2];
    double nx = aby * bcz - abz * bcy, ny = abz * bcx - abx * bcz, nz = abx * bcy - aby * bcx;
    double area = sqrt(nx * nx + ny * ny + nz * nz);
    double jac = 0.5 * area * 0.78539816339744830962;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        double cx = c_gcos[q], sx = c_gsin[q];
        double dx = cx * abx + sx * bcx, dy = cx * aby + sx * bcy, dz = cx * abz + sx * bcz;
        double dist = sqrt(dx * dx + dy * dy + dz * dz);
        double of = jac * c_gw[q] / dist;
        double fac = 1.0 / (cx * cx);
        s0 += of * cx * fac;
        s1 += of * (cx - sx) * fac;
        s2 += of * sx * fac;
    }
    double rg0 = s0, rg1 = s1, rg2 = s2, rh0 = 0.0, rh1 = 0.0, rh2 = 0.0;
    if (MIRROR) {
        // regular rule over the mirrored own triangle, plain kernel, H sign flipped (Integrator.cpp:70-86)
        double bx = ax + abx, by = ay + aby, bz = az + abz;
        double cxp = bx + bcx, cyp = by + bcy, czp = bz + bcz;
        double max_ = -ax, mbx = -bx, mcx = -cxp;
        double mabx = mbx - max_, maby = by - ay, mabz = bz - az;
        double mbcx = mcx - mbx, mbcy = cyp - by, mbcz = czp - bz;
        double mnx = maby * mbcz - mabz * mbcy, mny = mabz * mbcx - mabx * mbcz, mnz = mabx * mbcy - maby * mbcx;
        double marea = sqrt(mnx * mnx + mny * mny + mnz * mnz);
        double mi = 1.0 / marea;
        mnx *= mi;
        mny *= mi;
        mnz *= mi;
        double a0 = 0, a1 = 0, a2 = 0, b0 = 0, b1 = 0, b2 = 0;
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            double u = c_quv[q][0], w = c_quv[q][1];
            double zx = (max_ + u * mabx) + w * mbcx - ax;
            double zy = (ay + u * maby) + w * mbcy - ay;
            double zz = (az + u * mabz) + w * mbcz - az;
            double inv = 1.0 / sqrt(zx * zx + zy * zy + zz * zz);
            double hq = -(zx * mnx + zy * mny + zz * mnz) * inv * inv * inv;
            a0 += c_qc[q][0] * inv;
            a1 += c_qc[q][1] * inv;
            a2 += c_qc[q][2] * inv;
            b0 += c_qc[q][0] * hq;
            b1 += c_qc[q][1] * hq;
            b2 += c_qc[q][2] * hq;
        }
        rg0 += a0 * marea;
        rg1 += a1 * marea;
        rg2 += a2 * marea;
        rh0 = -(b0 * marea);
        rh1 = -(b1 * marea);
        rh2 = -(b2 * marea);
    }
    gg[0] = rg0;
    gg[1] = rg1;
    gg[2] = rg2;
    hh[0] = rh0;
    hh[1] = rh1;
    hh[2] = rh2;
}

// Singular pairs of a row and the row's 4 pi rule, one warp per row (row i, il within its block of n
// vertices whose G/H block starts at element mbase and whose group partials are rowHp, bp).
//  * The lanes take the triangles around vertex i (the vertex-to-triangle lists are sorted), 32 at a
//    time, and evaluate their singular pairs in parallel: entries (lane, m) with column j and the G
//    and H contributions, staged in shared memory.
//  * The lane holding the first entry of each column j adds that column's entries to G(i, j) and
//    H(i, j) one by one in entry order (increasing triangle index), after the tile kernel has written
//    the regular part.  Entries of one column are never split between two lanes, so nothing races.
//  * The row's sums sum_j H(i, j) and sum_j H(i, j) phi_j are the group partials of the tiles (a fixed
//    butterfly order) plus the singular share (entry order); H(i, i) -= 4 pi + sum_j H(i, j) and
//    b_i = (H phi)_i follow (ColocSim.cpp:85-97).  Every sum has one fixed order, the same as with one
//    thread per row walking the triangles in order.
// A separate pass because inside the tile loop the rare singular branch cost a fifth of the tile
// kernel's time (divergent warps waiting at the staging barriers, and the call in the hot loop).
// GONLY (the G-only assembly of the step path, no H matrix): the partials bp are the regular pairs'
// share of sum_j H(i, j) (phi_j - phi_i) and rowHp is unused; the singular pairs add their H entries
// times (phi_j - phi_i), and b_i = that sum - 4 pi phi_i, which is the reference's
// sum_j H(i, j) phi_j after the 4 pi rule H(i, i) -= 4 pi + sum_j H(i, j) (ColocSim.cpp:85-97).
constexpr int SD_WARPS = 8;  // rows per CTA
template <bool MIRROR, bool GONLY = false>
__device__ __forceinline__ void singular_diag_row(int i, int il, int n, long long mbase, int vbase, int ngroups,
                                                  const double* __restrict__ rowHp, const double* __restrict__ bp,
                                                  const double* __restrict__ x, const int* __restrict__ tri,
                                                  const int* __restrict__ csr_off, const int* __restrict__ csr_idx,
                                                  const double* __restrict__ phi, double* __restrict__ G,
                                                  double* __restrict__ H, double* __restrict__ b,
                                                  const double* __restrict__ x0, const double* __restrict__ gp,
                                                  double* __restrict__ r0) {
    __shared__ int s_j[SD_WARPS][96];
    __shared__ double s_g[SD_WARPS][96], s_h[SD_WARPS][96];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double rs = 0.0, bsing = 0.0;  // (lane 0) the singular share of the H row sum and of H phi
    double gx = 0.0;               // (x0) this lane's share of (G x0)_i
    const int e0 = csr_off[i], e1 = csr_off[i + 1];
    for (int base = e0; base < e1; base += 32) {
        const int e = base + lane;
        int jj[3] = {-1, -1, -1};
        if (e < e1) {
            const int t = csr_idx[e];
            const int ta = tri[3 * t], tb = tri[3 * t + 1], tc = tri[3 * t + 2];
            const int shift = (i == ta) ? 0 : ((i == tb) ? 1 : 2);
            double gg[3], hh[3];
            singular_sums<MIRROR>(x, ta, tb, tc, shift, gg, hh);
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                jj[m] = tri[3 * t + (m + shift) % 3];
                s_g[w][3 * lane + m] = gg[m];
                s_h[w][3 * lane + m] = hh[m];
            }
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) s_j[w][3 * lane + m] = jj[m];
        __syncwarp();
        const int ne = 3 * min(32, e1 - base);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const int j = jj[m], me = 3 * lane + m;
            if (j < 0) continue;
            bool first = true;
            for (int q = 0; q < me; ++q)
                if (s_j[w][q] == j) {
                    first = false;
                    break;
                }
            if (!first) continue;
            const size_t o = (size_t)mbase + (size_t)(j - vbase) * n + il;
            double gv = G[o], hv = (MIRROR && !GONLY) ? H[o] : 0.0, gsing = 0.0;
            for (int q = me; q < ne; ++q)
                if (s_j[w][q] == j) {
                    gv += s_g[w][q];
                    hv += s_h[w][q];
                    gsing += s_g[w][q];
                }
            G[o] = gv;
            if (x0) gx = fma(gsing, x0[j], gx);
            if (MIRROR && !GONLY) H[o] = hv;  // without the wall image the singular double layer vanishes (flat triangle)
        }
        if (MIRROR && lane == 0) {
            const double phii = GONLY ? phi[i] : 0.0;
            for (int q = 0; q < ne; ++q)
                if (s_j[w][q] >= 0) {
                    rs += s_h[w][q];
                    bsing = fma(s_h[w][q], GONLY ? phi[s_j[w][q]] - phii : phi[s_j[w][q]], bsing);
                }
        }
        __syncwarp();
    }
    // 4 pi rule and right-hand side: lane l sums the partials of groups l, l+32, ... and the warp adds
    // the lane sums in a fixed butterfly order (deterministic)
    double val = 0.0, bs = 0.0;
    const size_t pr = (size_t)il * ngroups;  // the row's partials, contiguous
    for (int g = lane; g < ngroups; g += 32) {
        if (!GONLY) val -= rowHp[pr + g];
        bs += bp[pr + g];
    }
    if (x0)
        for (int g = lane; g < ngroups; g += 32) gx += gp[pr + g];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        val += __shfl_xor_sync(0xffffffffu, val, o);
        bs += __shfl_xor_sync(0xffffffffu, bs, o);
        gx += __shfl_xor_sync(0xffffffffu, gx, o);
    }
    if (lane) return;
    bs += bsing;
    double bi;
    if (GONLY) {
        bi = fma(-4.0 * 3.14159265358979323846, phi[i], bs);
    } else {
        val -= rs;
        const double d = -(4.0 * 3.14159265358979323846 - val);
        const size_t oii = (size_t)mbase + (size_t)il * n + il;
        H[oii] += d;  // after the warp's singular update of H(i, i) (ordered by the last __syncwarp)
        bi = fma(d, phi[i], bs);
    }
    if (b) b[i] = bi;
    if (x0) r0[i] = bi - gx;  // the first residual b - G x0 of the solve that follows
}

template <bool MIRROR, bool GONLY = false>
__global__ void __launch_bounds__(32 * SD_WARPS)
    k_singular_diag(int N, int ngroups, const double* __restrict__ rowHp, const double* __restrict__ bp,
                    const double* __restrict__ x, const int* __restrict__ tri, const int* __restrict__ csr_off,
                    const int* __restrict__ csr_idx, const double* __restrict__ phi, double* __restrict__ G,
                    double* __restrict__ H, double* __restrict__ b, const double* __restrict__ x0,
                    const double* __restrict__ gp, double* __restrict__ r0) {
    const int i = blockIdx.x * SD_WARPS + (threadIdx.x >> 5);
    if (i >= N) return;
    singular_diag_row<MIRROR, GONLY>(i, i, N, 0, 0, ngroups, rowHp, bp, x, tri, csr_off, csr_idx, phi, G, H, b, x0,
                                     gp, r0);
}

// The same per block of a batch (rows of block vblk[i], its own groups and G/H block).
template <bool MIRROR>
__global__ void __launch_bounds__(32 * SD_WARPS)
    k_singular_diag_batch(int N, const int* __restrict__ vblk, const BlockInfo* __restrict__ blk,
                          const double* __restrict__ rowHp, const double* __restrict__ bp,
                          const double* __restrict__ x, const int* __restrict__ tri, const int* __restrict__ csr_off,
                          const int* __restrict__ csr_idx, const double* __restrict__ phi, double* __restrict__ G,
                          double* __restrict__ H, double* __restrict__ b) {
    const int i = blockIdx.x * SD_WARPS + (threadIdx.x >> 5);
    if (i >= N) return;
    const BlockInfo B = blk[vblk[i]];
    singular_diag_row<MIRROR>(i, i - B.vbase, B.n, B.mbase, B.vbase, B.ngroups, rowHp + B.pbase, bp + B.pbase, x,
                              tri, csr_off, csr_idx, phi, G, H, b, nullptr, nullptr, nullptr);
}

// Column-group tile: the columns of group g (local index gl within its block) for rows
// [row0, row0 + ROWS) clipped at rowend, of the block whose vertices start at vbase (n of them) and
// whose G/H block starts at element mbase.  CGT: vertices (columns) per group, ROWS: rows per CTA
// (one per thread).  Accumulators are thread-private columns of shared memory; the triangle
// records of the group are staged in shared memory ASM_TC at a time.
template <bool MIRROR, int CGT, int ROWS>
__device__ __forceinline__ void assemble_tile(double* smem, const double* __restrict__ x, const int* __restrict__ tri,
                                              const double* __restrict__ rec, const int* __restrict__ grp_off,
                                              const int* __restrict__ grp_tri, const int* __restrict__ grp_slot,
                                              const int* __restrict__ grp_vert, const double* __restrict__ phi,
                                              double* __restrict__ G, double* __restrict__ H,
                                              double* __restrict__ rowHp, double* __restrict__ bp, int g, int gl,
                                              int row0, int rowend, int n, int vbase, long long mbase,
                                              long long pbase, int ngrp, const double* __restrict__ x0,
                                              double* __restrict__ gp) {
    double* accG = smem;                      // [CGT][ROWS]
    double* accH = accG + CGT * ROWS;         // [CGT][ROWS]
    double* srec = accH + CGT * ROWS;         // [ASM_TC][REC]
    int* sinfo = reinterpret_cast<int*>(srec + ASM_TC * REC);  // [ASM_TC][4]
    const int tid = threadIdx.x;
    const int i = row0 + tid;
#pragma unroll 4
    for (int s = 0; s < CGT; ++s) {
        accG[s * ROWS + tid] = 0.0;
        accH[s * ROWS + tid] = 0.0;
    }
    double xi0 = 0.0, xi1 = 0.0, xi2 = 0.0;
    if (i < rowend) {
        xi0 = x[3 * i];
        xi1 = x[3 * i + 1];
        xi2 = x[3 * i + 2];
    }
    const int tb = grp_off[g], te = grp_off[g + 1];
    for (int c0 = tb; c0 < te; c0 += ASM_TC) {
        const int cnt = min(ASM_TC, te - c0);
        __syncthreads();
        for (int e = tid; e < cnt * (REC / 2); e += ROWS) {
            int tt = e / (REC / 2), w = e - tt * (REC / 2);
            const double2* src = reinterpret_cast<const double2*>(rec + (size_t)grp_tri[c0 + tt] * REC);
            reinterpret_cast<double2*>(srec + tt * REC)[w] = src[w];
        }
        for (int e = tid; e < cnt; e += ROWS) {
            int t = grp_tri[c0 + e];
            sinfo[4 * e] = grp_slot[c0 + e];
            sinfo[4 * e + 1] = tri[3 * t];
            sinfo[4 * e + 2] = tri[3 * t + 1];
            sinfo[4 * e + 3] = tri[3 * t + 2];
        }
        __syncthreads();
        if (i < rowend) {
            for (int tt = 0; tt < cnt; ++tt) {
                const int4 info = reinterpret_cast<const int4*>(sinfo)[tt];
                const int code = info.x;
                if (i == info.y || i == info.z || i == info.w) continue;  // singular: k_singular_diag
                PairSums p;
                regular_pair<MIRROR>(srec + tt * REC, xi0, xi1, xi2, p);
                const int s0 = code & SLOT_NONE, s1 = (code >> SLOT_BITS) & SLOT_NONE,
                          s2 = (code >> (2 * SLOT_BITS)) & SLOT_NONE;
                if (s0 != SLOT_NONE) {
                    accG[s0 * ROWS + tid] = fma(p.g[0], p.area, accG[s0 * ROWS + tid]);
                    accH[s0 * ROWS + tid] = add_h<MIRROR>(p, 0, accH[s0 * ROWS + tid]);
                }
                if (s1 != SLOT_NONE) {
                    accG[s1 * ROWS + tid] = fma(p.g[1], p.area, accG[s1 * ROWS + tid]);
                    accH[s1 * ROWS + tid] = add_h<MIRROR>(p, 1, accH[s1 * ROWS + tid]);
                }
                if (s2 != SLOT_NONE) {
                    accG[s2 * ROWS + tid] = fma(p.g[2], p.area, accG[s2 * ROWS + tid]);
                    accH[s2 * ROWS + tid] = add_h<MIRROR>(p, 2, accH[s2 * ROWS + tid]);
                }
            }
        }
    }
    if (i < rowend) {
        const int il = i - vbase;
        double rs = 0.0, bs = 0.0, gs = 0.0;
        for (int s = 0; s < CGT; ++s) {
            int v = grp_vert[g * CGT + s];
            if (v < 0) continue;
            double gv = accG[s * ROWS + tid], hv = accH[s * ROWS + tid];
            const size_t o = (size_t)mbase + (size_t)(v - vbase) * n + il;
            G[o] = gv;
            H[o] = hv;
            rs += hv;
            bs = fma(hv, phi[v], bs);
            if (x0) gs = fma(gv, x0[v], gs);
        }
        // row-major partials (row il, group gl of ngrp): the reduction over groups then reads each
        // row's partials as one contiguous run
        const size_t po = (size_t)pbase + (size_t)il * ngrp + gl;
        rowHp[po] = rs;
        bp[po] = bs;
        if (x0) gp[po] = gs;
    }
}

// Single system: one CTA per (column group, row tile).
template <bool MIRROR, int CGT, int ROWS, int MINB>
__global__ void __launch_bounds__(ROWS, MINB) k_assemble(int N, const double* __restrict__ x, const int* __restrict__ tri,
                                                         const double* __restrict__ rec, const int* __restrict__ grp_off,
                                                         const int* __restrict__ grp_tri, const int* __restrict__ grp_slot,
                                                         const int* __restrict__ grp_vert, const double* __restrict__ phi,
                                                         double* __restrict__ G, double* __restrict__ H,
                                                         double* __restrict__ rowHp, double* __restrict__ bp,
                                                         const double* __restrict__ x0, double* __restrict__ gp) {
    extern __shared__ __align__(16) double smem[];
    assemble_tile<MIRROR, CGT, ROWS>(smem, x, tri, rec, grp_off, grp_tri, grp_slot, grp_vert, phi, G, H, rowHp, bp,
                                     blockIdx.x, blockIdx.x, blockIdx.y * ROWS, N, N, 0, 0, 0, gridDim.x, x0, gp);
}

// Block-diagonal batch: one persistent launch over the work list of every block's tiles
// {group, first row, block, local group}; CTAs take tiles from an atomic counter, which the CTA
// that draws the last ticket resets for the next launch.
template <bool MIRROR, int CGT, int ROWS, int MINB>
__global__ void __launch_bounds__(ROWS, MINB)
    k_assemble_batch(const int4* __restrict__ tiles, int ntiles, unsigned* __restrict__ ctr,
                     const BlockInfo* __restrict__ blk, const double* __restrict__ x, const int* __restrict__ tri,
                     const double* __restrict__ rec, const int* __restrict__ grp_off, const int* __restrict__ grp_tri,
                     const int* __restrict__ grp_slot, const int* __restrict__ grp_vert, const double* __restrict__ phi,
                     double* __restrict__ G, double* __restrict__ H, double* __restrict__ rowHp,
                     double* __restrict__ bp) {
    extern __shared__ __align__(16) double smem[];
    __shared__ unsigned s_t;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            s_t = atomicAdd(ctr, 1u);
            if (s_t == (unsigned)ntiles + gridDim.x - 1) *ctr = 0u;  // last ticket of this launch
        }
        __syncthreads();
        const unsigned t = s_t;
        if (t >= (unsigned)ntiles) break;
        const int4 td = tiles[t];
        const BlockInfo B = blk[td.z];
        assemble_tile<MIRROR, CGT, ROWS>(smem, x, tri, rec, grp_off, grp_tri, grp_slot, grp_vert, phi, G, H, rowHp,
                                         bp, td.x, td.w, td.y, B.vbase + B.n, B.n, B.vbase, B.mbase, B.pbase, B.ngroups,
                                         nullptr, nullptr);
    }
}

void launch_triangle_records(Ctx& c, const double* x, cudaStream_t s) {
    upload_constants();
    int M = (int)c.topo.M;
    KLAUNCH(), k_triangle_records<<<(M + 127) / 128, 128, 0, s>>>(M, x, c.topo.tri, c.rec);
}

template <bool MIRROR, int CGT, int ROWS, int MINB>
static void launch_tiles_t(Ctx& c, const double* x, const double* phi, double* G, double* H, cudaStream_t s,
                           const double* x0) {
    const int N = (int)c.topo.N;
    const size_t sm = sizeof(double) * (2 * CGT * ROWS + ASM_TC * REC) + sizeof(int) * 4 * ASM_TC;
    static std::atomic<uint64_t> attr{0};
    once_per_device(attr, [sm] {
        return cudaFuncSetAttribute(k_assemble<MIRROR, CGT, ROWS, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sm) == cudaSuccess;
    });
    dim3 grid(c.topo.ngroups, (N + ROWS - 1) / ROWS);
    KLAUNCH(), k_assemble<MIRROR, CGT, ROWS, MINB><<<grid, ROWS, sm, s>>>(N, x, c.topo.tri, c.rec, c.topo.grp_off,
                                                                          c.topo.grp_tri, c.topo.grp_slot,
                                                                          c.topo.grp_vert, phi, G, H, c.rowHp, c.bp, x0,
                                                                          c.gp);
}

template <int CGT, int ROWS>
constexpr size_t tile_smem() {
    return sizeof(double) * (2 * CGT * ROWS + ASM_TC * REC) + sizeof(int) * 4 * ASM_TC;
}

template <bool MIRROR, int CGT, int ROWS, int MINB>
static void prepare_batch_t(Ctx& c) {
    const size_t sm = tile_smem<CGT, ROWS>();
    auto kern = k_assemble_batch<MIRROR, CGT, ROWS, MINB>;
    static std::atomic<uint64_t> attr{0};
    once_per_device(attr, [kern, sm] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) == cudaSuccess;
    });
    if (c.asm_grid_cg != CGT) {  // persistent grid: every CTA slot the SMs can hold
        int per_sm = 0, sms = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, ROWS, sm);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
        c.asm_grid = std::max(1, std::min(c.ntiles, std::max(1, per_sm) * sms));
        c.asm_grid_cg = CGT;
    }
}

template <bool MIRROR, int CGT, int ROWS, int MINB>
static void launch_batch_t(Ctx& c, const double* x, const double* phi, double* G, double* H, cudaStream_t s) {
    const size_t sm = tile_smem<CGT, ROWS>();
    auto kern = k_assemble_batch<MIRROR, CGT, ROWS, MINB>;
    prepare_batch_t<MIRROR, CGT, ROWS, MINB>(c);
    KLAUNCH(), kern<<<c.asm_grid, ROWS, sm, s>>>(c.tiles, c.ntiles, c.tile_ctr, c.blk, x, c.topo.tri, c.rec,
                                                c.topo.grp_off, c.topo.grp_tri, c.topo.grp_slot, c.topo.grp_vert, phi,
                                                G, H, c.rowHp, c.bp);
}

// Tile shapes: 16 columns x 256 rows (24 warps/SM, more boundary triangles), 32 x 128 (12 warps/SM),
// 48 x 64 and 64 x 64 (fewer boundary triangles, 6 warps/SM); all at 3 CTAs per SM within the 228 KB
// of shared memory.
void prepare_assemble_g(Ctx& c);

void prepare_assemble(Ctx& c) {
    if (c.topo.npatch > 0) prepare_assemble_g(c);
    if (!c.batch) return;
    c.asm_grid_cg = 0;
    if (c.prm.mirror) {
        if (c.topo.cg == 16) prepare_batch_t<true, 16, 256, 3>(c);
        else if (c.topo.cg == 64) prepare_batch_t<true, 64, 64, 3>(c);
        else if (c.topo.cg == 48) prepare_batch_t<true, 48, 64, 3>(c);
        else prepare_batch_t<true, 32, 128, 3>(c);
    } else {
        if (c.topo.cg == 16) prepare_batch_t<false, 16, 256, 3>(c);
        else if (c.topo.cg == 64) prepare_batch_t<false, 64, 64, 3>(c);
        else if (c.topo.cg == 48) prepare_batch_t<false, 48, 64, 3>(c);
        else prepare_batch_t<false, 32, 128, 3>(c);
    }
}

template <bool MIRROR>
static void launch_tiles(Ctx& c, const double* x, const double* phi, double* G, double* H, cudaStream_t s,
                         const double* x0) {
    if (c.batch) {
        switch (c.topo.cg) {
            case 16:
                launch_batch_t<MIRROR, 16, 256, 3>(c, x, phi, G, H, s);
                break;
            case 64:
                launch_batch_t<MIRROR, 64, 64, 3>(c, x, phi, G, H, s);
                break;
            case 48:
                launch_batch_t<MIRROR, 48, 64, 3>(c, x, phi, G, H, s);
                break;
            default:
                launch_batch_t<MIRROR, 32, 128, 3>(c, x, phi, G, H, s);
        }
        return;
    }
    switch (c.topo.cg) {
        case 16:
            launch_tiles_t<MIRROR, 16, 256, 3>(c, x, phi, G, H, s, x0);
            break;
        case 64:
            launch_tiles_t<MIRROR, 64, 64, 3>(c, x, phi, G, H, s, x0);
            break;
        case 48:
            launch_tiles_t<MIRROR, 48, 64, 3>(c, x, phi, G, H, s, x0);
            break;
        default:
            launch_tiles_t<MIRROR, 32, 128, 3>(c, x, phi, G, H, s, x0);
    }
}

// x0, r0 (single systems, may be null): with x0 the assembly also returns r0 = b - G x0, the first
// residual of a solve started from x0, from the G columns while they are in shared memory (per-group
// partials of G x0 beside those of H phi).
void launch_assemble(Ctx& c, const double* x, const double* phi, double* G, double* H, double* b, cudaStream_t s,
                     const double* x0, double* r0) {
    const int N = (int)c.topo.N;
    if (c.batch || !r0) x0 = nullptr;
    launch_triangle_records(c, x, s);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (c.prof) {
        e0 = c.take_event();
        e1 = c.take_event();
        cudaEventRecord(e0, s);
    }
    if (c.prm.mirror)
        launch_tiles<true>(c, x, phi, G, H, s, x0);
    else
        launch_tiles<false>(c, x, phi, G, H, s, x0);
    // singular pairs and the 4 pi rule, one warp per row
    const Topology& T = c.topo;
    const int nbs = (N + SD_WARPS - 1) / SD_WARPS, nt = 32 * SD_WARPS;
    if (c.batch) {
        if (c.prm.mirror)
            KLAUNCH(), k_singular_diag_batch<true><<<nbs, nt, 0, s>>>(N, c.vblk, c.blk, c.rowHp, c.bp, x, T.tri, T.csr_off,
                                                                      T.csr_idx, phi, G, H, b);
        else
            KLAUNCH(), k_singular_diag_batch<false><<<nbs, nt, 0, s>>>(N, c.vblk, c.blk, c.rowHp, c.bp, x, T.tri,
                                                                       T.csr_off, T.csr_idx, phi, G, H, b);
    } else {
        if (c.prm.mirror)
            KLAUNCH(), k_singular_diag<true><<<nbs, nt, 0, s>>>(N, T.ngroups, c.rowHp, c.bp, x, T.tri, T.csr_off,
                                                                T.csr_idx, phi, G, H, b, x0, c.gp, r0);
        else
            KLAUNCH(), k_singular_diag<false><<<nbs, nt, 0, s>>>(N, T.ngroups, c.rowHp, c.bp, x, T.tri, T.csr_off,
                                                                 T.csr_idx, phi, G, H, b, x0, c.gp, r0);
    }
    if (c.prof) {  // the profile's assembly time: tiles, singular pairs and the 4 pi rule
        cudaEventRecord(e1, s);
        c.ev_asm.emplace_back(e0, e1);
    }
}


// ------------------------------------------------------------------------------------------------
// G-only assembly of the step path (triangle patches)
// ------------------------------------------------------------------------------------------------
// The RK4 step needs G and b = H phi (after the 4 pi rule), never H itself.  Each triangle belongs
// to exactly one patch (Topology::patch_*), so every regular (row, triangle) pair is evaluated once:
// a CTA owns one patch and ROWS rows, accumulates the patch's columns (at most PCOLS vertices) in
// shared memory and, per row, b's regular share sum_t sum_k H_k(i, t) (phi_k - phi_i) in a register.
// The patch's triangle records are contiguous (patch order) and arrive in shared memory by one bulk
// copy (cp.async.bulk, completion counted on an mbarrier) while the threads clear their accumulators.
// A column whose vertex has all its triangles in the patch is complete and goes straight to G; the
// columns of vertices shared with other patches go to halo columns.  For each shared vertex and row
// tile, the patch CTA that finishes last (a ticket counter) sums the halo slices in increasing patch
// order, while they are still in L2, and writes the G column.
// Without the wall image the singular pairs (3 per triangle, the polar rule of Integrator.cpp:13-41)
// are evaluated beside the records, one thread per (triangle, corner), and the tile loop adds them
// where the row is a vertex of the triangle; k_rhs_finish then sums each row's patch partials of b
// and adds the 4 pi term.  Per G entry the order is: the pairs of each patch, regular and singular,
// in increasing triangle order (for a column inside one patch, the reference's per-column order),
// then the patches in increasing order.  With the wall image the singular pairs carry an H part too;
// k_singular_diag<true, true> adds them after the tiles, with the 4 pi term.  No atomics on values,
// so results are bit-reproducible.

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// An mbarrier counting one arrival, initialised before any thread uses it.
__device__ __forceinline__ void copy_bar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One 1-D bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned) from global to
// shared memory, its completion counted on `bar` (the arrival that also announces the bytes).
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"((unsigned long long)__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// Bounded wait for phase `parity` of `bar`: false after `limit` polls.
__device__ __forceinline__ bool copy_bar_wait(uint64_t* bar, uint32_t parity, int limit) {
    const uint32_t a = smem_addr(bar);
    for (int it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
constexpr int COPY_WAIT_POLLS = 1 << 22;  // each poll may suspend the thread for a while: seconds in all

// Patch-order triangle records (PREC doubles), for row distances from the corners: with
// A = |a - x|^2, B = |b - x|^2 - A = (a - x).2ab + |ab|^2 and C the same for ac, a point y with barycentric
// weights (l0, l1, l2) lies at |y - x|^2 = A + l1 B + l2 C - W, W = l0 l1 |ab|^2 + l0 l2 |ac|^2 + l1 l2 |bc|^2,
// so the points of an orbit (weights alpha, beta, beta in turn) share A + beta (B + C).  Layout: the three
// vertices' columns as byte offsets into the tile's accumulators, three ints (0-1); a (2-4), 2ab (5-7), 2ac (8-10), |ab|^2,
// |ac|^2 (11, 12), -area n (13-15), area (16), -W (17-23) and w phi (24-30) of the points.  The points are the
// centroid, then the orbits' points by the vertex that has alpha.  Without the wall image 31-39 hold the
// triangle's singular pairs: for row = vertex k of the triangle, the G entry of the column of vertex v at
// PR_SING + 3 k + v; with it y.x of the points (31-37).
constexpr int PR_W = 17, PR_PHI = 24, PR_SING = 31, PR_YX = 31;
static_assert(PR_SING + 9 <= PREC, "the record holds the singular pairs");
// the 7-point rule's index (c_quv) of the points in this order
__constant__ int c_porder[7] = {0, 3, 1, 2, 6, 4, 5};

// A CTA takes PR_TRI triangles: without the wall image one warp their records and three the singular pairs, one
// (triangle, corner) per thread (Integrator.cpp:13-41); with it each thread a record.  The records are put together
// in shared memory and written as one run: as 8-byte stores 320 bytes apart they took 186 us for the 618 thousand
// triangles of a sweep, now 74 (the singular pairs' divisions and roots).
template <bool MIRROR>
constexpr int PR_TRI = MIRROR ? 128 : 32;
template <bool MIRROR>
__global__ void __launch_bounds__(128) k_patch_records(int M, const double* __restrict__ x, const double* __restrict__ phi,
                                                       const int* __restrict__ tri, const int* __restrict__ ptri,
                                                       const int* __restrict__ pslot, double* __restrict__ prec) {
    constexpr int TRI = PR_TRI<MIRROR>, LD = PREC + 1;  // odd: no bank conflicts across triangles
    extern __shared__ double srecs[];                   // [TRI][LD]
    const int p0 = blockIdx.x * TRI, l = threadIdx.x % TRI, p = p0 + l;
    double* r = srecs + l * LD;
    if (p < M) {
        const int t = ptri[p];
        const int ia = tri[3 * t], ib = tri[3 * t + 1], ic = tri[3 * t + 2];
        if (!MIRROR && threadIdx.x >= TRI) {
            const int k = threadIdx.x / TRI - 1;
            double gg[3], hh[3];
            singular_sums<false>(x, ia, ib, ic, k, gg, hh);  // gg[m]: the column of vertex (m + k) % 3
#pragma unroll
            for (int m = 0; m < 3; ++m) r[PR_SING + 3 * k + (m + k) % 3] = gg[m];
        } else {
            const double ax = x[3 * ia], ay = x[3 * ia + 1], az = x[3 * ia + 2];
            const double abx = x[3 * ib] - ax, aby = x[3 * ib + 1] - ay, abz = x[3 * ib + 2] - az;
            const double acx = x[3 * ic] - ax, acy = x[3 * ic + 1] - ay, acz = x[3 * ic + 2] - az;
            const double bcx = x[3 * ic] - x[3 * ib], bcy = x[3 * ic + 1] - x[3 * ib + 1], bcz = x[3 * ic + 2] - x[3 * ib + 2];
            const double nx = aby * bcz - abz * bcy, ny = abz * bcx - abx * bcz, nz = abx * bcy - aby * bcx;
            const double ab2 = abx * abx + aby * aby + abz * abz, ac2 = acx * acx + acy * acy + acz * acz;
            const double bc2 = bcx * bcx + bcy * bcy + bcz * bcz;
            const int sl = pslot[p], col = PATCH_ROWS * (int)sizeof(double);
            r[0] = __hiloint2double((sl >> 8 & 255) * col, (sl & 255) * col);
            r[1] = __hiloint2double(0, (sl >> 16 & 255) * col);
            r[2] = ax;
            r[3] = ay;
            r[4] = az;
            r[5] = 2.0 * abx;
            r[6] = 2.0 * aby;
            r[7] = 2.0 * abz;
            r[8] = 2.0 * acx;
            r[9] = 2.0 * acy;
            r[10] = 2.0 * acz;
            r[11] = ab2;
            r[12] = ac2;
            r[13] = -nx;
            r[14] = -ny;
            r[15] = -nz;
            r[16] = sqrt(nx * nx + ny * ny + nz * nz);
            const double fa = phi[ia], fb = phi[ib], fc = phi[ic];
#pragma unroll
            for (int e = 0; e < 7; ++e) {
                const int k = c_porder[e];
                const double u = c_quv[k][0], v = c_quv[k][1], l0 = 1.0 - u, l1 = u - v;
                r[PR_W + e] = -(l0 * l1 * ab2 + l0 * v * ac2 + l1 * v * bc2);
                r[PR_PHI + e] = c_qc[k][0] * fa + c_qc[k][1] * fb + c_qc[k][2] * fc;
                if (MIRROR) r[PR_YX + e] = ax + u * abx + v * bcx;
            }
        }
    }
    __syncthreads();
    const int words = min(TRI, M - p0) * PREC;
    for (int e = threadIdx.x; e < words; e += 128) prec[(size_t)p0 * PREC + e] = srecs[e / PREC * LD + e % PREC];
}

// One regular (row, triangle) pair: g_k (to be scaled by the area), and hb takes the row's share of b,
// sum over the points of w (phi(y) - phi_i) * (-area (y - x).n / r^3).  wphi: w phi_i for the three weights.
// 112 FP64 operations, 49 of them the seven 1/r and 1/r^3.
template <bool MIRROR>
__device__ __forceinline__ void patch_pair(const double* __restrict__ rec, double xi0, double xi1, double xi2,
                                           const double (&wphi)[3], double (&g)[3], double& hb) {
    // two entries per shared-memory load (the record is 16-byte aligned)
    double r[MIRROR ? 38 : 32];
#pragma unroll
    for (int k = 2; k < (MIRROR ? 38 : 32); k += 2) {
        const double2 v = *reinterpret_cast<const double2*>(rec + k);
        r[k] = v.x;
        r[k + 1] = v.y;
    }
    const double ax = r[2] - xi0, ay = r[3] - xi1, az = r[4] - xi2;
    const double A = fma(ax, ax, fma(ay, ay, __dmul_rn(az, az)));
    const double B = fma(ax, r[5], fma(ay, r[6], fma(az, r[7], r[11])));
    const double C = fma(ax, r[8], fma(ay, r[9], fma(az, r[10], r[12])));
    const double sh = fma(ax, r[13], fma(ay, r[14], __dmul_rn(az, r[15])));  // -area (y - x).n, y in the plane
    const double BC = B + C;
    double kg[7], hs = 0.0, hm = 0.0;
    auto point = [&](int e, double r2, double wp) {
        const double inv = rsqrt_fp64(r2);
        const double f = r[PR_PHI + e] - wp;
        kg[e] = inv;
        const double inv3 = __dmul_rn(__dmul_rn(inv, inv), inv);
        hs = e ? fma(inv3, f, hs) : __dmul_rn(inv3, f);
        if (MIRROR) {
            // image point (-y.x, y.y, y.z), image normal (-n.x, n.y, n.z) (Integrator.hpp:211-229):
            // |y' - x|^2 = |y - x|^2 + 4 x.x y.x
            const double inm = rsqrt_fp64(fma(4.0 * xi0, r[PR_YX + e], r2));
            kg[e] += inm;
            const double inm3 = __dmul_rn(__dmul_rn(inm, inm), inm);
            hm = e ? fma(inm3, f, hm) : __dmul_rn(inm3, f);
        }
    };
    point(0, fma(1.0 / 3.0, BC, A + r[PR_W]), wphi[0]);
#pragma unroll
    for (int o = 0; o < 2; ++o) {
        const double P = fma(c_pbeta[o], BC, A);
        const int e = 1 + 3 * o;
        point(e, P + r[PR_W + e], wphi[1 + o]);
        point(e + 1, fma(c_pdiff[o], B, P + r[PR_W + e + 1]), wphi[1 + o]);
        point(e + 2, fma(c_pdiff[o], C, P + r[PR_W + e + 2]), wphi[1 + o]);
    }
    // sum_q w_q basis_k(q) K(q), as orbit_sums
    const double SA = (kg[2] + kg[3]) + kg[1], SB = (kg[5] + kg[6]) + kg[4];
    const double K = fma(c_orb[0], kg[0], fma(c_orb[1], SA, __dmul_rn(c_orb[3], SB)));
#pragma unroll
    for (int k = 0; k < 3; ++k) g[k] = fma(c_orb[2], kg[1 + k], fma(c_orb[4], kg[4 + k], K));
    hb = fma(hs, sh, hb);
    if (MIRROR) hb = fma(hm, fma(2.0 * xi0, r[13], sh), hb);  // (y' - x).n' = (a - x).n + 2 x.x n.x
}

template <int ROWS>
constexpr size_t patch_smem() {
    return sizeof(double) * ((size_t)PT_MAX * PREC + (size_t)PCOLS * ROWS);
}

// One CTA per tile {patch, first row} of the work list, ROWS rows of the patch's block, one row per
// thread.  G, the halo columns and the row partials are addressed through the patch's PatchInfo, so
// the same kernel serves a single system (one block) and a batch of independent bubbles.
// What bounds it: the pair loop, and there the register reads.  Measured (B200): an FP64 operation takes two issue
// cycles of its SM quarter, three if it reads three different registers; beside one with two or three register
// operands no other instruction issues for free, beside one with a single one (constants, repeated or just used
// operands) some do.  So a pair's 112 FP64 operations and its other instructions add up, and more warps change
// nothing (32 instead of 24 per SM with narrower patches: 4593 and 4602 us at N = 16002).  The shared-memory pipe
// is 70 % busy beside it (records read as broadcasts).  Hence: no singular test in tiles without singular pairs,
// column offsets ready in the record, two triangles per turn of the loop, y0^2 in rsqrt_fp64.  At N = 16002
// 4.48 -> 4.10 ms, at N = 4002 311 -> 285 us, with the wall image at N = 1442 80 -> 74 us (four triangles per
// turn: 4.19 ms).  Measured slower at N = 4002: two rows per thread with half the threads (a record read then
// serves two rows, 299 us), and a persistent form that defers tickets and finishing sums by a tile (423 us before
// these); starting the SM's three CTAs apart changes nothing.
template <bool MIRROR, int ROWS, int MINB>
__global__ void __launch_bounds__(ROWS, MINB)
    k_assemble_patch(const int2* __restrict__ work, const PatchInfo* __restrict__ pinfo,
                     const double* __restrict__ prec, const int* __restrict__ patch_col,
                     const long long* __restrict__ patch_dst, const double* __restrict__ x,
                     const double* __restrict__ phi, double* __restrict__ G, double* __restrict__ halo,
                     double* __restrict__ bp, const double* __restrict__ x0, double* __restrict__ gp,
                     int* __restrict__ err, const int* __restrict__ patch_pk, const PartialCol* __restrict__ pcol,
                     unsigned* __restrict__ halo_tick) {
    extern __shared__ __align__(16) double psmem[];
    double* srec = psmem;                  // [PT_MAX][PREC], the patch's records
    double* acc = psmem + PT_MAX * PREC;   // [PCOLS][ROWS], this CTA's rows of the patch's columns
    __shared__ __align__(8) uint64_t bar;
    __shared__ int s_pk[PCOLS], s_v[PCOLS], s_nc, s_near;
    __shared__ double* s_dst[PCOLS];
    __shared__ double s_x0[PCOLS];
    const int tid = threadIdx.x;
    const int2 wk = work[blockIdx.x];
    const int p = wk.x;
    const PatchInfo P = pinfo[p];
    const int i = wk.y + tid;  // row (global vertex index)
    if (tid == 0) copy_bar_init(&bar);
    __syncthreads();
    if (tid == 0) bulk_copy_g2s(srec, prec + (size_t)P.t0 * PREC, (uint32_t)(P.nt * PREC * sizeof(double)), &bar);
    if (tid < PCOLS) {
        const int v = patch_col[p * PCOLS + tid];
        const long long h = patch_dst[p * PCOLS + tid];
        s_dst[tid] = h < 0 ? G + P.mbase + (long long)(v - P.vbase) * P.n : halo + h;  // where the column goes
        s_pk[tid] = patch_pk[p * PCOLS + tid];
        const unsigned used = __ballot_sync(0xffffffffu, v >= 0);  // the used slots come first
        const unsigned near = __ballot_sync(0xffffffffu, v >= wk.y && v < wk.y + ROWS);
        if (tid == 0) {
            s_nc = __popc(used);
            s_near = near != 0u;
        }
        s_v[tid] = v;
        s_x0[tid] = x0 && v >= 0 ? x0[v] : 0.0;
    }
#pragma unroll 8
    for (int s = 0; s < PCOLS; ++s) acc[s * ROWS + tid] = 0.0;
    const bool row = i < P.vbase + P.n;
    double xi0 = 0.0, xi1 = 0.0, xi2 = 0.0, phii = 0.0;
    if (row) {
        xi0 = x[3 * i];
        xi1 = x[3 * i + 1];
        xi2 = x[3 * i + 2];
        phii = phi[i];
    }
    if (!__syncthreads_and(copy_bar_wait(&bar, 0, COPY_WAIT_POLLS))) {
        // the records did not arrive in time: record the error, let the copy land (bounded) before the
        // CTA's shared memory is released, and leave this tile unwritten (the host reports the error)
        if (tid == 0) {
            atomicExch(err, 1);
            copy_bar_wait(&bar, 0, COPY_WAIT_POLLS);
        }
        return;
    }
    double hb = 0.0;  // the row's share of b over this patch's regular pairs
    const double wphi[3] = {__dmul_rn(c_pw[0], phii), __dmul_rn(c_pw[1], phii), __dmul_rn(c_pw[2], phii)};
    // A tile with a vertex of the patch among its rows has singular pairs (without the wall image their G entries
    // come with the records, and the double layer of the flat own triangle vanishes; with it,
    // k_singular_diag<true, true> adds both); the other tiles run the loop without the test.
    char* mine = reinterpret_cast<char*>(acc + tid);
    const auto pairs = [&](auto near) {
        int own = -1;  // the row's own column of the patch
        if (decltype(near)::value)
            for (int s = 0; s < s_nc; ++s)
                if (s_v[s] == i) own = s * ROWS * (int)sizeof(double);
#pragma unroll 2
        for (int t = 0; t < (row ? P.nt : 0); ++t) {
            const double* r = srec + t * PREC;
            const int4 id = *reinterpret_cast<const int4*>(r);
            double* a0 = reinterpret_cast<double*>(mine + id.x);
            double* a1 = reinterpret_cast<double*>(mine + id.y);
            double* a2 = reinterpret_cast<double*>(mine + id.z);
            if (decltype(near)::value && (own == id.x || own == id.y || own == id.z)) {
                if (!MIRROR) {
                    const double* sg = r + PR_SING + (own == id.x ? 0 : (own == id.y ? 3 : 6));
                    *a0 += sg[0];
                    *a1 += sg[1];
                    *a2 += sg[2];
                }
                continue;
            }
            double g[3];
            patch_pair<MIRROR>(r, xi0, xi1, xi2, wphi, g, hb);
            const double area = r[16];
            *a0 = fma(g[0], area, *a0);
            *a1 = fma(g[1], area, *a1);
            *a2 = fma(g[2], area, *a2);
        }
    };
    if (s_near)
        pairs(std::true_type{});
    else
        pairs(std::false_type{});
    const int il = i - P.vbase;
    if (row) {
        double gs = 0.0;
        const int nc = s_nc;
#pragma unroll 4
        for (int s = 0; s < nc; ++s) s_dst[s][il] = acc[s * ROWS + tid];
        if (x0) {
#pragma unroll 4
            for (int s = 0; s < nc; ++s) gs = fma(acc[s * ROWS + tid], s_x0[s], gs);
        }
        const long long po = P.pbase + (long long)il * P.np + P.lp;  // the row's partials are contiguous
        bp[po] = hb;
        if (x0) gp[po] = gs;
    }
    // shared vertices: one ticket per (vertex, row tile); the CTA drawing the last one sums the halo
    // slices of this row tile in increasing patch order (every slice was written before its ticket)
    const int rt = (wk.y - P.vbase) / ROWS;
    __threadfence();
    __syncthreads();
    __shared__ int s_nfin;
    static_assert(PCOLS == 32, "the finishing slots are drawn by one warp");
    static_assert(PT_MAX * PREC * sizeof(double) >= PCOLS * sizeof(PartialCol), "finishing slots fit the records");
    PartialCol* s_pc = reinterpret_cast<PartialCol*>(srec);  // the records are no longer read
    if (tid < PCOLS) {
        const int k = s_pk[tid];
        bool fin = false;
        PartialCol pc;
        if (k >= 0) {
            pc = pcol[k];
            fin = atomicAdd(&halo_tick[pc.tick + rt], 1u) == (unsigned)(pc.cnt - 1);
        }
        // the finishing columns, compacted in slot order
        const unsigned m = __ballot_sync(0xffffffffu, fin);
        if (fin) s_pc[__popc(m & ((1u << tid) - 1u))] = pc;
        if (tid == 0) s_nfin = __popc(m);
    }
    __syncthreads();
    const int nfin = s_nfin;
    if (nfin > 0) __threadfence();  // the other patches' slices, written before their tickets
    // four columns at a time, the first four slices of each loaded before any is summed (the slices
    // sit in L2: one round trip per four columns instead of one per column)
    constexpr int FC = 4, FS = 4;
    for (int f0 = 0; f0 < (row ? nfin : 0); f0 += FC) {
        double v[FC][FS];
#pragma unroll
        for (int f = 0; f < FC; ++f) {
            const PartialCol& pc = s_pc[f0 + f < nfin ? f0 + f : f0];
            const double* h = halo + pc.hpos + il;
#pragma unroll
            for (int c2 = 0; c2 < FS; ++c2) v[f][c2] = (f0 + f < nfin && c2 < pc.cnt) ? __ldcg(h + (size_t)c2 * pc.n) : 0.0;
        }
#pragma unroll
        for (int f = 0; f < FC; ++f) {
            if (f0 + f >= nfin) break;
            const PartialCol& pc = s_pc[f0 + f];
            double sum = v[f][0];
#pragma unroll
            for (int c2 = 1; c2 < FS; ++c2)
                if (c2 < pc.cnt) sum += v[f][c2];
            const double* h = halo + pc.hpos + il;
            for (int c2 = FS; c2 < pc.cnt; ++c2) sum += __ldcg(h + (size_t)c2 * pc.n);
            G[pc.gpos + il] = sum;
        }
    }
    if (tid < nfin) halo_tick[s_pc[tid].tick + rt] = 0u;  // for the next assembly
}

// The G-only singular pass of a batch: rows of block vblk[i], its patches' row partials.
template <bool MIRROR>
__global__ void __launch_bounds__(32 * SD_WARPS)
    k_singular_diag_batch_g(int N, const int* __restrict__ vblk, const BlockInfo* __restrict__ blk,
                            const double* __restrict__ bp, const double* __restrict__ x, const int* __restrict__ tri,
                            const int* __restrict__ csr_off, const int* __restrict__ csr_idx,
                            const double* __restrict__ phi, double* __restrict__ G, double* __restrict__ b) {
    const int i = blockIdx.x * SD_WARPS + (threadIdx.x >> 5);
    if (i >= N) return;
    const BlockInfo B = blk[vblk[i]];
    singular_diag_row<MIRROR, true>(i, i - B.vbase, B.n, B.mbase, B.vbase, B.npatch, nullptr, bp + B.ppbase, x, tri,
                                    csr_off, csr_idx, phi, G, nullptr, b, nullptr, nullptr, nullptr);
}

// b_i (and r0_i = b_i - (G x0)_i) of the G-only assembly without the wall image, one warp per row:
// the tiles already hold every pair of the row, so what is left is the sum of the row's patch partials
// (lane l takes patches l, l + 32, ..., the lanes add in a fixed butterfly order) and the 4 pi term,
// b_i = sum_j H(i, j) (phi_j - phi_i) - 4 pi phi_i (ColocSim.cpp:85-97).
__device__ __forceinline__ void rhs_finish_row(int i, int il, int np, const double* __restrict__ bp,
                                               const double* __restrict__ phi, double* __restrict__ b,
                                               const double* __restrict__ x0, const double* __restrict__ gp,
                                               double* __restrict__ r0) {
    const int lane = threadIdx.x & 31;
    const size_t pr = (size_t)il * np;  // the row's partials, contiguous
    double bs = 0.0, gx = 0.0;
    for (int g = lane; g < np; g += 32) bs += bp[pr + g];
    if (x0)
        for (int g = lane; g < np; g += 32) gx += gp[pr + g];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        bs += __shfl_xor_sync(0xffffffffu, bs, o);
        gx += __shfl_xor_sync(0xffffffffu, gx, o);
    }
    if (lane) return;
    const double bi = fma(-4.0 * 3.14159265358979323846, phi[i], bs);
    if (b) b[i] = bi;
    if (x0) r0[i] = bi - gx;
}

__global__ void __launch_bounds__(32 * SD_WARPS)
    k_rhs_finish(int N, int np, const double* __restrict__ bp, const double* __restrict__ phi,
                 double* __restrict__ b, const double* __restrict__ x0, const double* __restrict__ gp,
                 double* __restrict__ r0) {
    const int i = blockIdx.x * SD_WARPS + (threadIdx.x >> 5);
    if (i >= N) return;
    rhs_finish_row(i, i, np, bp, phi, b, x0, gp, r0);
}

__global__ void __launch_bounds__(32 * SD_WARPS)
    k_rhs_finish_batch(int N, const int* __restrict__ vblk, const BlockInfo* __restrict__ blk,
                       const double* __restrict__ bp, const double* __restrict__ phi, double* __restrict__ b) {
    const int i = blockIdx.x * SD_WARPS + (threadIdx.x >> 5);
    if (i >= N) return;
    const BlockInfo B = blk[vblk[i]];
    rhs_finish_row(i, i - B.vbase, B.npatch, bp + B.ppbase, phi, b, nullptr, nullptr, nullptr);
}

template <bool MIRROR>
static bool prepare_patch_t() {
    static std::atomic<uint64_t> attr{0};
    return once_per_device(attr, [] {
        return cudaFuncSetAttribute(k_assemble_patch<MIRROR, PATCH_ROWS, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)patch_smem<PATCH_ROWS>()) == cudaSuccess;
    });
}

// Kernel attributes and __constant__ tables of the G-only assembly, outside any stream capture.
void prepare_assemble_g(Ctx& c) {
    upload_constants();
    if (c.prm.mirror)
        prepare_patch_t<true>();
    else
        prepare_patch_t<false>();
}

// G (the context's G) and b = H phi after the 4 pi rule for positions x, potential phi, without H; with
// x0 (may be null; single systems) also r0 = b - G x0.  No pinned vertices.
void launch_assemble_g(Ctx& c, const double* x, const double* phi, double* b, cudaStream_t s, const double* x0,
                       double* r0) {
    const Topology& T = c.topo;
    const int N = (int)T.N, M = (int)T.M;
    if (!r0 || c.batch) x0 = nullptr;
    prepare_assemble_g(c);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (c.prof) {
        e0 = c.take_event();
        e1 = c.take_event();
        cudaEventRecord(e0, s);
    }
    // records (and, without the wall image, the singular pairs)
    if (c.prm.mirror)
        KLAUNCH(), k_patch_records<true><<<(M + PR_TRI<true> - 1) / PR_TRI<true>, 128,
                                           sizeof(double) * PR_TRI<true> * (PREC + 1), s>>>(M, x, phi, T.tri, T.patch_tri,
                                                                                          T.patch_slot, c.prec);
    else
        KLAUNCH(), k_patch_records<false><<<(M + PR_TRI<false> - 1) / PR_TRI<false>, 128,
                                            sizeof(double) * PR_TRI<false> * (PREC + 1), s>>>(
                       M, x, phi, T.tri, T.patch_tri, T.patch_slot, c.prec);
    constexpr size_t sm = patch_smem<PATCH_ROWS>();
    if (c.prm.mirror)
        KLAUNCH(), k_assemble_patch<true, PATCH_ROWS, 3><<<T.nwork, PATCH_ROWS, sm, s>>>(
                       T.pwork, T.pinfo, c.prec, T.patch_col, T.patch_dst, x, phi, c.G, c.halo, c.bp, x0, c.gp,
                       c.asm_err, T.patch_pk, T.pcol, T.halo_tick);
    else
        KLAUNCH(), k_assemble_patch<false, PATCH_ROWS, 3><<<T.nwork, PATCH_ROWS, sm, s>>>(
                       T.pwork, T.pinfo, c.prec, T.patch_col, T.patch_dst, x, phi, c.G, c.halo, c.bp, x0, c.gp,
                       c.asm_err, T.patch_pk, T.pcol, T.halo_tick);
    const int nbs = (N + SD_WARPS - 1) / SD_WARPS, nt = 32 * SD_WARPS;
    if (c.batch) {
        if (c.prm.mirror)
            KLAUNCH(), k_singular_diag_batch_g<true><<<nbs, nt, 0, s>>>(N, c.vblk, c.blk, c.bp, x, T.tri, T.csr_off,
                                                                        T.csr_idx, phi, c.G, b);
        else
            KLAUNCH(), k_rhs_finish_batch<<<nbs, nt, 0, s>>>(N, c.vblk, c.blk, c.bp, phi, b);
    } else if (c.prm.mirror) {
        KLAUNCH(), k_singular_diag<true, true><<<nbs, nt, 0, s>>>(N, T.npatch, nullptr, c.bp, x, T.tri, T.csr_off,
                                                                  T.csr_idx, phi, c.G, nullptr, b, x0, c.gp, r0);
    } else {
        KLAUNCH(), k_rhs_finish<<<nbs, nt, 0, s>>>(N, T.npatch, c.bp, phi, b, x0, c.gp, r0);
    }
    if (c.prof) {  // the profile's assembly time: records, tiles (with the shared columns' sums), singular pairs, 4 pi rule
        cudaEventRecord(e1, s);
        c.ev_asm.emplace_back(e0, e1);
    }
}

}  // namespace bemb
