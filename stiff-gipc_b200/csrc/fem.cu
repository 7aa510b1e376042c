// fem.cu -- the Hessian producer of one implicit-Euler Newton iteration on the GPU: per-tet
// stable Neo-Hookean gradient and PSD-projected Hessian (12x12, written as the 10 upper 3x3
// blocks of the tet), lumped mass, the kinetic term and IPC plane barriers, as the device
// triplets and gradient that GlobalLinearSystem::solve_linear_system receives.
//
// The reference builds these in femEnergy.cu:1719-1855 (_calculate_fem_gradient_hessian, its
// SNH variants and Eigen-SVD eigensystem projection) and GIPC.cu:6524-6551 (ground barrier).
// This file follows the formulation of the synthetic scenes (stgipc/scenes.py: SNH of Smith
// et al. 2018 without the log term, psi = mu/2 (|F|^2 - 3) + lam/2 (J - alpha)^2,
// alpha = 1 + mu / lam, whose 9x9 Hessian in F is projected to PSD by clamping negative
// eigenvalues), and the reference's plane barrier on the squared distance.
#include "solver.hpp"

namespace stg
{
namespace
{
constexpr int FT = 128;  // threads per CTA

__device__ __forceinline__ double det3(const double (&M)[3][3])
{
    return M[0][0] * (M[1][1] * M[2][2] - M[1][2] * M[2][1]) - M[0][1] * (M[1][0] * M[2][2] - M[1][2] * M[2][0]) +
           M[0][2] * (M[1][0] * M[2][1] - M[1][1] * M[2][0]);
}

// ---------------------------------------------------------------------------------------
// The PSD projection in closed form.  With F = U diag(s) V^T (U, V proper rotations, s signed)
// the 9x9 Hessian mu I + lam g g^T + k d2J/dF2, k = lam (J - alpha), splits (Smith et al. 2018,
// section 4) into three 2x2 problems on u_p v_q^T +- u_q v_p^T with eigenvalues mu -+ k s_r
// ({p, q, r} = {0, 1, 2}: one of each pair at most is negative when mu > 0) and one 3x3 problem
// on the u_p v_p^T.  Clamping means adding -lambda Q (x) Q for every negative eigenpair, which
// in the 12 vertex coordinates is a rank-one update.  The eigenvectors come from a one-sided
// Jacobi SVD of F (backward stable, so the blocks keep the accuracy of a full eigen-solve).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ double dot3(const double (&a)[3], const double (&b)[3])
{
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// c, s of the rotation that diagonalises [[app, apq], [apq, aqq]]; apq * apq > 0 (where it
// vanishes in 64 bits, d * d may too, and t is no tangent)
__device__ __forceinline__ void jacobi_cs(double app, double aqq, double apq, double& c, double& s, double& t)
{
    const double d = aqq - app, w = 2.0 * apq;
    // t = sign(d) w / (|d| + sqrt(d^2 + w^2)): tan of the smaller angle, no overflow of d / w
    t = w / (fabs(d) + sqrt(d * d + w * w));
    if(d < 0.0) t = -t;
    c = rsqrt(t * t + 1.0);
    s = t * c;
}

// A: rows are the columns of F on entry, F V on exit (orthogonal rows); V: rows v_p
__device__ __forceinline__ void svd_rotate(double (&A)[3][3], double (&V)[3][3], int p, int q, bool& more)
{
    const double app = dot3(A[p], A[p]), aqq = dot3(A[q], A[q]), apq = dot3(A[p], A[q]);
    if(!(apq * apq > 4e-31 * (app * aqq))) return;
    more = true;
    double c, s, t;
    jacobi_cs(app, aqq, apq, c, s, t);
#pragma unroll
    for(int i = 0; i < 3; i++)
    {
        const double x = A[p][i], y = A[q][i], v = V[p][i], w = V[q][i];
        A[p][i] = c * x - s * y;
        A[q][i] = s * x + c * y;
        V[p][i] = c * v - s * w;
        V[q][i] = s * v + c * w;
    }
}

// signed SVD F = sum_p s_p u_p v_p^T; s[2] has the smallest magnitude and the sign of det F
__device__ __forceinline__ void svd3(const double (&F)[3][3], double (&U)[3][3], double (&sv)[3], double (&V)[3][3])
{
    double A[3][3];
#pragma unroll
    for(int p = 0; p < 3; p++)
#pragma unroll
        for(int i = 0; i < 3; i++)
        {
            A[p][i] = F[i][p];
            V[p][i] = p == i ? 1.0 : 0.0;
        }
    bool more = true;
    for(int sweep = 0; sweep < 12 && more; sweep++)
    {
        more = false;
        svd_rotate(A, V, 0, 1, more);
        svd_rotate(A, V, 0, 2, more);
        svd_rotate(A, V, 1, 2, more);
    }
    double n0 = dot3(A[0], A[0]), n1 = dot3(A[1], A[1]), n2 = dot3(A[2], A[2]);
    // the smallest column last: swapped with column 2, one of the two negated (V stays proper)
#pragma unroll
    for(int p = 0; p < 2; p++)
    {
        const bool sw = p == 0 ? (n0 < n2 && n0 <= n1) : (n1 < n2);
        if(!sw) continue;
#pragma unroll
        for(int i = 0; i < 3; i++)
        {
            const double x = A[p][i], v = V[p][i];
            A[p][i] = A[2][i];
            A[2][i] = -x;
            V[p][i] = V[2][i];
            V[2][i] = -v;
        }
        const double nn = p == 0 ? n0 : n1;
        if(p == 0)
            n0 = n2;
        else
            n1 = n2;
        n2 = nn;
    }
    // A column below 1e-100 of the other counts as zero: it changes nothing, but its direction is
    // not one of the orthogonal basis (svd_rotate's squares vanish before such a column is
    // orthogonal, and a lone column may stand in either place).  A rank of one leaves it first.
    if(n0 < 1e-200 * n1)
    {
#pragma unroll
        for(int i = 0; i < 3; i++)
        {
            const double x = A[0][i], v = V[0][i];
            A[0][i] = A[1][i];
            A[1][i] = -x;
            V[0][i] = V[1][i];
            V[1][i] = -v;
        }
        const double nn = n0;
        n0 = n1;
        n1 = nn;
    }
    sv[0] = sqrt(n0);
    sv[1] = sqrt(n1);
    const bool has0 = n0 > 0.0, has1 = n1 > 1e-200 * n0;
    const double i0 = has0 ? 1.0 / sv[0] : 0.0, i1 = has1 ? 1.0 / sv[1] : 0.0;
#pragma unroll
    for(int i = 0; i < 3; i++)
    {
        U[0][i] = A[0][i] * i0;
        U[1][i] = A[1][i] * i1;
    }
    // a rank below two leaves u_0 or u_1 free: any orthonormal completion
    if(!has0) U[0][0] = 1.0;
    if(!has1)
    {
        const bool ax = fabs(U[0][0]) < 0.6;  // an axis away from u_0, made orthogonal to it
        const double e[3] = {ax ? 1.0 : 0.0, ax ? 0.0 : 1.0, 0.0};
        const double d = dot3(U[0], e);
        double w[3], n = 0.0;
#pragma unroll
        for(int i = 0; i < 3; i++)
        {
            w[i] = e[i] - d * U[0][i];
            n += w[i] * w[i];
        }
        n = rsqrt(n);
#pragma unroll
        for(int i = 0; i < 3; i++) U[1][i] = w[i] * n;
    }
    U[2][0] = U[0][1] * U[1][2] - U[0][2] * U[1][1];
    U[2][1] = U[0][2] * U[1][0] - U[0][0] * U[1][2];
    U[2][2] = U[0][0] * U[1][1] - U[0][1] * U[1][0];
    sv[2] = dot3(U[2], A[2]);
}

// a gradient share with the tet's lumped mass share: one 32-byte sector per (tet, vertex)
__device__ __forceinline__ void st_share(double* p, double a, double b, double c, double d)
{
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}
__device__ __forceinline__ void ld_share(const double* p, double& a, double& b, double& c, double& d)
{
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p));
}

// mu = E / mu_div, lam = E nu / lam_div
struct Material
{
    double nu, mu_div, lam_div, rho, dt;
};

// One thread per tet: the 10 upper blocks (column-major, upper orientation) into the triplets
// at t * 10 + kk, the four gradient shares with the mass share, and the tet's place in each
// vertex's incidence list (counted here, filled by k_fem_fill).  The blocks of a warp's 32
// tets are contiguous; they pass through shared memory, five blocks a tet at a time (45
// doubles: an odd stride, no bank conflicts), and leave in 360-byte runs.
constexpr int FT_ROW = 45;
constexpr int FT_SMEM = (FT / 32) * 32 * FT_ROW * (int)sizeof(double);

__global__ void __launch_bounds__(FT, 3) k_fem_tet(const double* __restrict__ rest, const double* __restrict__ pos,
                                                const int* __restrict__ tets, const double* __restrict__ E, int T,
                                                Material mat, int* rows, int* cols, double* blocks, double* share,
                                                int* cnt, int4* place)
{
    extern __shared__ double fsm[];
    const int lane = threadIdx.x & 31;
    double* sw = fsm + (threadIdx.x >> 5) * (32 * FT_ROW);
    const int t0 = blockIdx.x * FT + (threadIdx.x & ~31), t = t0 + lane;
    if(t0 >= T) return;
    const int nt = min(32, T - t0);
    const bool on = lane < nt;
    int v[4] = {0, 0, 0, 0};
    double d[4][3], F[3][3], g[3][3], U[3][3], V[3][3], sv[3];
    double mu = 0, lam = 0, k = 0, w = 0;
    if(on)
    {
#pragma unroll
        for(int a = 0; a < 4; a++) v[a] = tets[4 * (size_t)t + a];
        int4 pl;
        pl.x = atomicAdd(cnt + v[0], 1);
        pl.y = atomicAdd(cnt + v[1], 1);
        pl.z = atomicAdd(cnt + v[2], 1);
        pl.w = atomicAdd(cnt + v[3], 1);
        place[t] = pl;
        double Dm[3][3], Ds[3][3];
#pragma unroll
        for(int r = 0; r < 3; r++)
        {
            const double r0 = rest[3 * (size_t)v[0] + r], p0 = pos[3 * (size_t)v[0] + r];
#pragma unroll
            for(int a = 0; a < 3; a++)
            {
                Dm[r][a] = rest[3 * (size_t)v[a + 1] + r] - r0;
                Ds[r][a] = pos[3 * (size_t)v[a + 1] + r] - p0;
            }
        }
        const double dd = det3(Dm);
        const double vol = fabs(dd) / 6.0;
        // d[a][j]: dF_ij / dx_a,i; rows 1..3 are Dm^-1 = adj(Dm) / det
        d[1][0] = (Dm[1][1] * Dm[2][2] - Dm[1][2] * Dm[2][1]) / dd;
        d[1][1] = (Dm[0][2] * Dm[2][1] - Dm[0][1] * Dm[2][2]) / dd;
        d[1][2] = (Dm[0][1] * Dm[1][2] - Dm[0][2] * Dm[1][1]) / dd;
        d[2][0] = (Dm[1][2] * Dm[2][0] - Dm[1][0] * Dm[2][2]) / dd;
        d[2][1] = (Dm[0][0] * Dm[2][2] - Dm[0][2] * Dm[2][0]) / dd;
        d[2][2] = (Dm[0][2] * Dm[1][0] - Dm[0][0] * Dm[1][2]) / dd;
        d[3][0] = (Dm[1][0] * Dm[2][1] - Dm[1][1] * Dm[2][0]) / dd;
        d[3][1] = (Dm[0][1] * Dm[2][0] - Dm[0][0] * Dm[2][1]) / dd;
        d[3][2] = (Dm[0][0] * Dm[1][1] - Dm[0][1] * Dm[1][0]) / dd;
#pragma unroll
        for(int j = 0; j < 3; j++) d[0][j] = -(d[1][j] + d[2][j] + d[3][j]);
#pragma unroll
        for(int i = 0; i < 3; i++)
#pragma unroll
            for(int j = 0; j < 3; j++) F[i][j] = Ds[i][0] * d[1][j] + Ds[i][1] * d[2][j] + Ds[i][2] * d[3][j];
        mu = E[t] / mat.mu_div;
        lam = E[t] * mat.nu / mat.lam_div;
        // cofactor g = dJ/dF
        g[0][0] = F[1][1] * F[2][2] - F[1][2] * F[2][1];
        g[0][1] = F[1][2] * F[2][0] - F[1][0] * F[2][2];
        g[0][2] = F[1][0] * F[2][1] - F[1][1] * F[2][0];
        g[1][0] = F[0][2] * F[2][1] - F[0][1] * F[2][2];
        g[1][1] = F[0][0] * F[2][2] - F[0][2] * F[2][0];
        g[1][2] = F[0][1] * F[2][0] - F[0][0] * F[2][1];
        g[2][0] = F[0][1] * F[1][2] - F[0][2] * F[1][1];
        g[2][1] = F[0][2] * F[1][0] - F[0][0] * F[1][2];
        g[2][2] = F[0][0] * F[1][1] - F[0][1] * F[1][0];
        k = lam * (det3(F) - (1.0 + mu / lam));
        w = vol * mat.dt * mat.dt;
        const double ms = mat.rho * vol / 4.0;
#pragma unroll
        for(int a = 0; a < 4; a++)
        {
            double f[3];
#pragma unroll
            for(int i = 0; i < 3; i++)
                f[i] = w * (d[a][0] * (mu * F[i][0] + k * g[i][0]) + d[a][1] * (mu * F[i][1] + k * g[i][1]) +
                            d[a][2] * (mu * F[i][2] + k * g[i][2]));
            st_share(share + 4 * (4 * (size_t)t + a), f[0], f[1], f[2], ms);
        }
        svd3(F, U, sv, V);
    }
    // G[a] = g d_a, vd[p][a] = v_p . d_a; the negative eigenpairs of the three 2x2 problems:
    // weight -lambda / 2 (the vectors carry 1 / sqrt 2 each) and sign sg of the vectors
    // y_r[a] = u_p vd[q][a] + sg u_q vd[p][a], formed where they are used
    double G[4][3], vd[3][4], wt[3], sg[3];
    bool diag = false;
    double Mq[6] = {0, 0, 0, 0, 0, 0};
    if(on)
    {
#pragma unroll
        for(int a = 0; a < 4; a++)
#pragma unroll
            for(int i = 0; i < 3; i++)
            {
                G[a][i] = dot3(g[i], d[a]);
                vd[i][a] = dot3(V[i], d[a]);
            }
#pragma unroll
        for(int r = 0; r < 3; r++)
        {
            const double ks = k * sv[r], lm = mu - fabs(ks);
            wt[r] = lm < 0.0 ? -0.5 * lm : 0.0;
            sg[r] = ks < 0.0 ? -1.0 : 1.0;  // mu + ks on the antisymmetric vector
        }
        // the 3x3 problem, positive definite for all but strongly compressed or inverted tets:
        // its leading minors decide
        const double s12 = sv[1] * sv[2], s02 = sv[0] * sv[2], s01 = sv[0] * sv[1];
        Mq[0] = mu + lam * s12 * s12;
        Mq[1] = k * sv[2] + lam * s12 * s02;
        Mq[2] = k * sv[1] + lam * s12 * s01;
        Mq[3] = mu + lam * s02 * s02;
        Mq[4] = k * sv[0] + lam * s02 * s01;
        Mq[5] = mu + lam * s01 * s01;
        const double m2 = Mq[0] * Mq[3] - Mq[1] * Mq[1];
        const double m3 = Mq[0] * (Mq[3] * Mq[5] - Mq[4] * Mq[4]) - Mq[1] * (Mq[1] * Mq[5] - Mq[4] * Mq[2]) +
                          Mq[2] * (Mq[1] * Mq[4] - Mq[3] * Mq[2]);
        diag = !(Mq[0] > 0.0 && m2 > 0.0 && m3 > 0.0) || mu < 0.0;
    }
    // its eigenpairs by cyclic Jacobi; z[m][a] = sum_p W_mp u_p (v_p . d_a) for negative ones
    double ev[3] = {0, 0, 0}, W[3][3];
    if(diag)
    {
        double M[3][3] = {{Mq[0], Mq[1], Mq[2]}, {Mq[1], Mq[3], Mq[4]}, {Mq[2], Mq[4], Mq[5]}};
#pragma unroll
        for(int i = 0; i < 3; i++)
#pragma unroll
            for(int j = 0; j < 3; j++) W[i][j] = i == j ? 1.0 : 0.0;
        const double nrm = Mq[0] * Mq[0] + Mq[3] * Mq[3] + Mq[5] * Mq[5] +
                           2.0 * (Mq[1] * Mq[1] + Mq[2] * Mq[2] + Mq[4] * Mq[4]);
        for(int sweep = 0; sweep < 12; sweep++)
        {
            const double off = M[0][1] * M[0][1] + M[0][2] * M[0][2] + M[1][2] * M[1][2];
            if(!(off > 1e-33 * nrm)) break;
#pragma unroll
            for(int pq = 0; pq < 3; pq++)
            {
                const int p = pq == 2 ? 1 : 0, q = pq == 0 ? 1 : 2, o = 3 - p - q;
                const double apq = M[p][q];
                if(!(apq * apq > 0.0)) continue;
                double c, s, tt;
                jacobi_cs(M[p][p], M[q][q], apq, c, s, tt);
                M[p][p] -= tt * apq;
                M[q][q] += tt * apq;
                M[p][q] = M[q][p] = 0.0;
                const double x = M[p][o], z = M[q][o];
                M[p][o] = M[o][p] = c * x - s * z;
                M[q][o] = M[o][q] = s * x + c * z;
#pragma unroll
                for(int i = 0; i < 3; i++)
                {
                    const double a = W[p][i], b = W[q][i];
                    W[p][i] = c * a - s * b;
                    W[q][i] = s * a + c * b;
                }
            }
        }
#pragma unroll
        for(int m = 0; m < 3; m++) ev[m] = M[m][m] < 0.0 ? -M[m][m] : 0.0;
    }
#pragma unroll
    for(int half = 0; half < 2; half++)
    {
        if(on)
        {
            int kk = 0;
#pragma unroll
            for(int a = 0; a < 4; a++)
#pragma unroll
                for(int b = a; b < 4; b++, kk++)
                {
                    if(kk / 5 != half) continue;
                    // block (a, b): w (mu d_a.d_b I + lam G_a G_b^T + k [F (d_a x d_b)]_x + the
                    // clamped parts)
                    const double dm = mu * dot3(d[a], d[b]);
                    double B[3][3];
#pragma unroll
                    for(int i = 0; i < 3; i++)
#pragma unroll
                        for(int q = 0; q < 3; q++) B[i][q] = lam * G[a][i] * G[b][q] + (i == q ? dm : 0.0);
                    if(a != b)
                    {
                        const double x0 = d[a][1] * d[b][2] - d[a][2] * d[b][1], x1 = d[a][2] * d[b][0] - d[a][0] * d[b][2],
                                     x2 = d[a][0] * d[b][1] - d[a][1] * d[b][0];
                        const double c0 = k * (F[0][0] * x0 + F[0][1] * x1 + F[0][2] * x2),
                                     c1 = k * (F[1][0] * x0 + F[1][1] * x1 + F[1][2] * x2),
                                     c2 = k * (F[2][0] * x0 + F[2][1] * x1 + F[2][2] * x2);
                        B[0][1] += c2;
                        B[1][0] -= c2;
                        B[0][2] -= c1;
                        B[2][0] += c1;
                        B[1][2] += c0;
                        B[2][1] -= c0;
                    }
#pragma unroll
                    for(int r = 0; r < 3; r++)
                    {
                        if(!(wt[r] > 0.0)) continue;
                        const int p = r == 0 ? 1 : 0, q = r == 2 ? 1 : 2;
                        double yb[3];
#pragma unroll
                        for(int j = 0; j < 3; j++) yb[j] = vd[q][b] * U[p][j] + sg[r] * vd[p][b] * U[q][j];
#pragma unroll
                        for(int i = 0; i < 3; i++)
                        {
                            const double ya = wt[r] * (vd[q][a] * U[p][i] + sg[r] * vd[p][a] * U[q][i]);
#pragma unroll
                            for(int j = 0; j < 3; j++) B[i][j] = fma(ya, yb[j], B[i][j]);
                        }
                    }
                    if(diag)
                    {
                        // a negative modulus: the other eigenpair of each 2x2 problem too
#pragma unroll
                        for(int r = 0; r < 3; r++)
                        {
                            const int p = r == 0 ? 1 : 0, q = r == 2 ? 1 : 2;
                            const double lm = mu + fabs(k * sv[r]);
                            if(!(lm < 0.0)) continue;
                            const double aa = vd[q][a], ab = -sg[r] * vd[p][a], ba = vd[q][b], bb = -sg[r] * vd[p][b];
#pragma unroll
                            for(int i = 0; i < 3; i++)
#pragma unroll
                                for(int j = 0; j < 3; j++)
                                    B[i][j] -= 0.5 * lm * (aa * U[p][i] + ab * U[q][i]) * (ba * U[p][j] + bb * U[q][j]);
                        }
#pragma unroll
                        for(int m = 0; m < 3; m++)
                        {
                            if(!(ev[m] > 0.0)) continue;
                            double za[3], zb[3];
#pragma unroll
                            for(int i = 0; i < 3; i++)
                            {
                                za[i] = zb[i] = 0.0;
#pragma unroll
                                for(int p = 0; p < 3; p++)
                                {
                                    za[i] += W[m][p] * U[p][i] * vd[p][a];
                                    zb[i] += W[m][p] * U[p][i] * vd[p][b];
                                }
                            }
#pragma unroll
                            for(int i = 0; i < 3; i++)
#pragma unroll
                                for(int q = 0; q < 3; q++) B[i][q] = fma(ev[m] * za[i], zb[q], B[i][q]);
                        }
                    }
                    const bool swap = v[a] > v[b];
                    double* o = sw + lane * FT_ROW + 9 * (kk % 5);
                    // column-major storage of the upper-oriented block (B^T when swapped)
#pragma unroll
                    for(int r = 0; r < 3; r++)
#pragma unroll
                        for(int c = 0; c < 3; c++) o[3 * c + r] = w * (swap ? B[c][r] : B[r][c]);
                }
        }
        __syncwarp();
        double* out = blocks + 90 * (size_t)t0 + FT_ROW * half;
        for(int e = lane, tt = 0, r = lane; e < nt * FT_ROW; e += 32, r += 32)
        {
            if(r >= FT_ROW) r -= FT_ROW, tt++;
            out[90 * (size_t)tt + r] = sw[e];
        }
        __syncwarp();
    }
    int* si = reinterpret_cast<int*>(sw);
    if(on)
    {
        int kk = 0;
#pragma unroll
        for(int a = 0; a < 4; a++)
#pragma unroll
            for(int b = a; b < 4; b++, kk++)
            {
                si[10 * lane + kk] = min(v[a], v[b]);
                si[320 + 10 * lane + kk] = max(v[a], v[b]);
            }
    }
    __syncwarp();
    for(int e = lane; e < 10 * nt; e += 32)
    {
        rows[10 * (size_t)t0 + e] = si[e];
        cols[10 * (size_t)t0 + e] = si[320 + e];
    }
}

__global__ void k_fem_fill(const int* __restrict__ tets, int T, const int* __restrict__ start,
                           const int* __restrict__ place, int* inc)
{
    for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < 4 * T; i += gridDim.x * blockDim.x)
        inc[start[tets[i]] + place[i]] = i;  // i = 4 t + a
}

// Per vertex: incident (tet, slot) entries in increasing order, then the gradient and mass
// gathered in that order (eight 32-byte shares in flight), the kinetic term, plane barriers,
// and the vertex's diagonal triplet.  Lists of up to 32 entries (a Kuhn mesh has 24) are sorted
// in registers by a network, without divergence; longer ones in place by insertion, which takes
// as many steps as the slowest lane of the warp.
constexpr int FV = 64;

__global__ void __launch_bounds__(FV) k_fem_vertex(const int* __restrict__ start, int* inc,
                                                   const double* __restrict__ share, const double* __restrict__ pos,
                                                   const double* __restrict__ vel, const double* __restrict__ xtilde,
                                                   int V, int T, double dt, double gy, const double* __restrict__ planes,
                                                   int nplanes, int* rows, int* cols, double* blocks, double* b)
{
    const int v = blockIdx.x * FV + threadIdx.x;
    if(v >= V) return;
    const int s0 = start[v], s1 = start[v + 1], n = s1 - s0;
    double g0 = 0, g1 = 0, g2 = 0, m = 0;
    if(n <= 32)
    {
        int k[32];
#pragma unroll
        for(int u = 0; u < 32; u++) k[u] = u < n ? inc[s0 + u] : 0x7fffffff;
        sort32(k);
#pragma unroll
        for(int p = 0; p < 32; p += 8)
        {
            double f[8][4];
#pragma unroll
            for(int u = 0; u < 8; u++)
                if(p + u < n) ld_share(share + 4 * (size_t)k[p + u], f[u][0], f[u][1], f[u][2], f[u][3]);
#pragma unroll
            for(int u = 0; u < 8; u++)
                if(p + u < n)
                {
                    g0 += f[u][0];
                    g1 += f[u][1];
                    g2 += f[u][2];
                    m += f[u][3];
                }
        }
    }
    else
    {
        for(int p = s0 + 1; p < s1; p++)
        {
            const int x = inc[p];
            int q = p - 1;
            while(q >= s0 && inc[q] > x)
            {
                inc[q + 1] = inc[q];
                q--;
            }
            inc[q + 1] = x;
        }
        for(int p = s0; p < s1; p++)
        {
            double f0, f1, f2, f3;
            ld_share(share + 4 * (size_t)inc[p], f0, f1, f2, f3);
            g0 += f0;
            g1 += f1;
            g2 += f2;
            m += f3;
        }
    }
    // kinetic: M (x - x_tilde), x_tilde given, or x_tilde = x + dt v + dt^2 (0, gy, 0) at x = x_n
    if(xtilde)
    {
        g0 += m * (pos[3 * (size_t)v] - xtilde[3 * (size_t)v]);
        g1 += m * (pos[3 * (size_t)v + 1] - xtilde[3 * (size_t)v + 1]);
        g2 += m * (pos[3 * (size_t)v + 2] - xtilde[3 * (size_t)v + 2]);
    }
    else
    {
        g0 += m * (-dt * vel[3 * (size_t)v]);
        g1 += m * (-dt * vel[3 * (size_t)v + 1] - dt * dt * gy);
        g2 += m * (-dt * vel[3 * (size_t)v + 2]);
    }
    double Hb[9] = {m, 0, 0, 0, m, 0, 0, 0, m};
    const double px = pos[3 * (size_t)v], py = pos[3 * (size_t)v + 1], pz = pos[3 * (size_t)v + 2];
    for(int k = 0; k < nplanes; k++)
    {
        const double* pl = planes + 6 * k;  // normal xyz, offset, dhat, kappa
        const double dist = px * pl[0] + py * pl[1] + pz * pl[2] - pl[3];
        const double dhat = pl[4], kappa = pl[5];
        if(!(dist < dhat)) continue;
        // IPC plane barrier on the squared distance (GIPC.cu:6524-6551)
        const double d2 = dist * dist, dh2 = dhat * dhat, tt = d2 - dh2, lg = log(d2 / dh2);
        const double gb = tt * lg * -2.0 - (tt * tt) / d2;
        const double hb = (lg * -2.0 - tt * 4.0 / d2) + 1.0 / (d2 * d2) * (tt * tt);
        const double gr = kappa * gb * 2.0 * dist, sc = kappa * (4.0 * hb * d2 + 2.0 * gb);
        g0 += gr * pl[0];
        g1 += gr * pl[1];
        g2 += gr * pl[2];
        for(int r = 0; r < 3; r++)
            for(int c = 0; c < 3; c++) Hb[3 * c + r] += sc * pl[r] * pl[c];
    }
    b[3 * (size_t)v] = g0;
    b[3 * (size_t)v + 1] = g1;
    b[3 * (size_t)v + 2] = g2;
    const size_t o = 10 * (size_t)T + v;
    rows[o] = v;
    cols[o] = v;
    for(int e = 0; e < 9; e++) blocks[9 * o + e] = Hb[e];
}

size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

// incremental potential of the Newton iteration's objective, per CTA: dt^2 vol psi(F) per tet
// with its vertices' shares of the inertia 1/2 m |x - x_tilde|^2 (m is the lumped mass, a
// quarter of every incident tet's, so no incidence list is needed), and kappa b(d^2) per
// vertex.  One launch: every CTA walks the tets, then the vertices, and leaves its partial in
// part[blockIdx.x].
__global__ void __launch_bounds__(256) k_fem_energy(const double* __restrict__ rest, const double* __restrict__ pos,
                                                    const double* __restrict__ xtilde, const int* __restrict__ tets,
                                                    const double* __restrict__ E, int T, int V, double nu, double rho,
                                                    double dt, const double* __restrict__ planes, int nplanes,
                                                    double* part, int* violations)
{
    __shared__ double red[8];
    double e = 0;
    for(int t = blockIdx.x * 256 + threadIdx.x; t < T; t += gridDim.x * 256)
    {
        int v[4];
        for(int a = 0; a < 4; a++) v[a] = tets[4 * (size_t)t + a];
        double Dm[3][3], Ds[3][3], q2 = 0;
        for(int r = 0; r < 3; r++)
        {
            const double r0 = rest[3 * (size_t)v[0] + r], p0 = pos[3 * (size_t)v[0] + r];
            const double q0 = p0 - xtilde[3 * (size_t)v[0] + r];
            q2 += q0 * q0;
            for(int a = 0; a < 3; a++)
            {
                const double p = pos[3 * (size_t)v[a + 1] + r], q = p - xtilde[3 * (size_t)v[a + 1] + r];
                Dm[r][a] = rest[3 * (size_t)v[a + 1] + r] - r0;
                Ds[r][a] = p - p0;
                q2 += q * q;
            }
        }
        const double dd = det3(Dm), vol = fabs(dd) / 6.0;
        // F = Ds Dm^-1: |F|^2 and det F = det Ds / det Dm
        double Di[3][3];
        Di[0][0] = (Dm[1][1] * Dm[2][2] - Dm[1][2] * Dm[2][1]) / dd;
        Di[0][1] = (Dm[0][2] * Dm[2][1] - Dm[0][1] * Dm[2][2]) / dd;
        Di[0][2] = (Dm[0][1] * Dm[1][2] - Dm[0][2] * Dm[1][1]) / dd;
        Di[1][0] = (Dm[1][2] * Dm[2][0] - Dm[1][0] * Dm[2][2]) / dd;
        Di[1][1] = (Dm[0][0] * Dm[2][2] - Dm[0][2] * Dm[2][0]) / dd;
        Di[1][2] = (Dm[0][2] * Dm[1][0] - Dm[0][0] * Dm[1][2]) / dd;
        Di[2][0] = (Dm[1][0] * Dm[2][1] - Dm[1][1] * Dm[2][0]) / dd;
        Di[2][1] = (Dm[0][1] * Dm[2][0] - Dm[0][0] * Dm[2][1]) / dd;
        Di[2][2] = (Dm[0][0] * Dm[1][1] - Dm[0][1] * Dm[1][0]) / dd;
        double F[3][3], f2 = 0;
        for(int i = 0; i < 3; i++)
            for(int j = 0; j < 3; j++)
            {
                F[i][j] = Ds[i][0] * Di[0][j] + Ds[i][1] * Di[1][j] + Ds[i][2] * Di[2][j];
                f2 += F[i][j] * F[i][j];
            }
        const double mu = E[t] / (2.0 * (1.0 + nu)), lam = E[t] * nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
        const double J = det3(F), alpha = 1.0 + mu / lam;
        e += vol * dt * dt * (0.5 * mu * (f2 - 3.0) + 0.5 * lam * (J - alpha) * (J - alpha));
        e += 0.5 * (rho * vol / 4.0) * q2;
    }
    for(int v = blockIdx.x * 256 + threadIdx.x; v < V && nplanes > 0; v += gridDim.x * 256)
    {
        for(int k = 0; k < nplanes; k++)
        {
            const double* pl = planes + 6 * k;
            const double dist = pos[3 * (size_t)v] * pl[0] + pos[3 * (size_t)v + 1] * pl[1] + pos[3 * (size_t)v + 2] * pl[2] - pl[3];
            if(!(dist > 0.0))
            {
                atomicAdd(violations, 1);
                continue;
            }
            if(dist < pl[4])
            {
                const double dd2 = dist * dist, dh2 = pl[4] * pl[4], tt = dd2 - dh2;
                e += pl[5] * (-(tt * tt) * log(dd2 / dh2));
            }
        }
    }
    e = block_sum<256>(e, red);
    if(threadIdx.x == 0) part[blockIdx.x] = e;
}
}  // namespace

constexpr int FEM_PARTS = kSMs * 4 + 8;  // energy: CTA partials + violation count

size_t fem_scratch_bytes(int V, int T)
{
    return a256(sizeof(double) * 16 * (size_t)T) + 2 * a256(sizeof(int) * (V + 1)) + 2 * a256(sizeof(int) * 4 * (size_t)T) +
           a256(sizeof(double) * FEM_PARTS);
}

int fem_newton_system(cudaStream_t s, int V, const double* rest, const double* pos, const double* vel,
                      const double* xtilde, int T, const int* tets, const double* E, double nu, double rho, double dt,
                      double gy, int nplanes, const double* planes, int* rows, int* cols, double* blocks, double* b,
                      void* scratch, size_t bytes)
{
    if(V < 1 || T < 0 || !rest || !pos || (!vel && !xtilde) || (T > 0 && (!tets || !E)) || (nplanes > 0 && !planes) || !rows ||
       !cols || !blocks || !b || !(dt > 0) || !(nu > 0 && nu < 0.5))
    {
        set_error("stg_fem_newton_system: invalid arguments");
        return STG_ERR_INVALID;
    }
    if(!scratch || bytes < fem_scratch_bytes(V, T) || reinterpret_cast<uintptr_t>(scratch) % 256)
    {
        set_error("stg_fem_newton_system: scratch too small or not 256-byte aligned");
        return STG_ERR_INVALID;
    }
    unsigned char* p = static_cast<unsigned char*>(scratch);
    double* share = reinterpret_cast<double*>(p);  // [T][4]{gradient, mass}
    p += a256(sizeof(double) * 16 * (size_t)T);
    int* cnt = reinterpret_cast<int*>(p);
    p += a256(sizeof(int) * (V + 1));
    int* start = reinterpret_cast<int*>(p);
    p += a256(sizeof(int) * (V + 1));
    int* place = reinterpret_cast<int*>(p);
    p += a256(sizeof(int) * 4 * (size_t)T);
    int* inc = reinterpret_cast<int*>(p);
    if(T > 0)
    {
        static thread_local unsigned long long attr_done = 0;
        if(first_on_device(attr_done))
            STG_CUDA_TRY(cudaFuncSetAttribute(k_fem_tet, cudaFuncAttributeMaxDynamicSharedMemorySize, FT_SMEM));
        STG_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(int) * (V + 1), s));
        const Material mat{nu, 2.0 * (1.0 + nu), (1.0 + nu) * (1.0 - 2.0 * nu), rho, dt};
        k_fem_tet<<<div_up(T, FT), FT, FT_SMEM, s>>>(rest, pos, tets, E, T, mat, rows, cols, blocks, share, cnt,
                                                     reinterpret_cast<int4*>(place));
        STG_LAUNCH_CHECK();
        STG_TRY(scan_exclusive(cnt, start, nullptr, V, V, start + V, s));
        k_fem_fill<<<std::max(1, std::min(div_up(4L * T, 256), kSMs * 8)), 256, 0, s>>>(tets, T, start, place, inc);
        STG_LAUNCH_CHECK();
    }
    else
        STG_CUDA_TRY(cudaMemsetAsync(start, 0, sizeof(int) * (V + 1), s));
    k_fem_vertex<<<div_up(V, FV), FV, 0, s>>>(start, inc, share, pos, vel, xtilde, V, T, dt, gy, planes, nplanes, rows,
                                              cols, blocks, b);
    STG_LAUNCH_CHECK();
    return 0;
}

// the incremental potential at pos (CTA partials summed on the host in CTA order); `violations` counts vertices on the wrong side of a plane (energy
// infinite: the caller must reject the step).  Uses the same scratch as fem_newton_system.
int fem_energy(cudaStream_t s, int V, const double* rest, const double* pos, const double* xtilde, int T,
               const int* tets, const double* E, double nu, double rho, double dt, int nplanes, const double* planes,
               void* scratch, size_t bytes, double* energy, int* violations)
{
    if(V < 1 || T < 0 || !rest || !pos || !xtilde || (T > 0 && (!tets || !E)) || (nplanes > 0 && !planes) || !energy)
    {
        set_error("stg_fem_energy: invalid arguments");
        return STG_ERR_INVALID;
    }
    if(!scratch || bytes < fem_scratch_bytes(V, T) || reinterpret_cast<uintptr_t>(scratch) % 256)
    {
        set_error("stg_fem_energy: scratch too small or not 256-byte aligned");
        return STG_ERR_INVALID;
    }
    double* part = static_cast<double*>(scratch);
    const int g = std::max(1, std::min(div_up(std::max(T, V), 256), kSMs * 4));
    int* viol = reinterpret_cast<int*>(part + g);
    STG_CUDA_TRY(cudaMemsetAsync(viol, 0, sizeof(int), s));
    k_fem_energy<<<g, 256, 0, s>>>(rest, pos, xtilde, tets, E, T, V, nu, rho, dt, planes, nplanes, part, viol);
    STG_LAUNCH_CHECK();
    // partials and violation count are adjacent: one read-back
    std::vector<double> h(g + 1);
    STG_CUDA_TRY(cudaMemcpyAsync(h.data(), part, sizeof(double) * g + sizeof(int), cudaMemcpyDeviceToHost, s));
    STG_CUDA_TRY(cudaStreamSynchronize(s));
    int hv = 0;
    std::memcpy(&hv, h.data() + g, sizeof(int));
    double e = 0;
    for(int i = 0; i < g; i++) e += h[i];
    *energy = e;
    if(violations) *violations = hv;
    return 0;
}

}  // namespace stg
