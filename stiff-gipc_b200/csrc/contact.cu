// contact.cu -- barrier gradient and Hessian of the contact pairs on sm_100a.
//
// Replaces _calBarrierGradientAndHessian (StiffGIPC/GIPC.cu:3149-4988) as the reference
// builds it (NEWF and RANK 2, GIPC.cu:29-30) for the four unmollified pair types of the
// sign-encoded int4 (GIPC.cuh:49-66):
//   edge-edge       x >= 0, w >= 0            edges (x, y) and (z, w)
//   point-point     x < 0, z < 0, y >= 0      point -x-1 and y
//   point-edge      x < 0, z >= 0, w < 0, y >= 0   point -x-1, edge (y, z)
//   point-triangle  x < 0, z >= 0, w >= 0     point -x-1, triangle (y, z, w)
// With d the pair's distance (the squared-distance formulas of _d_PP / _d_PE / _d_PT / _d_EE,
// mlbvh.cu:229-257), dHat the squared activation distance and s = d / sqrt(dHat), the
// barrier energy is kappa dHat^2 (s^2 - 1)^2 ln^2(s^2) for s < 1.  The gradient is E'(s) ds/dx
// and the Hessian the rank-one E''(s) ds/dx ds/dx^T (GIPC.cu:3187-3403: PFPx's last column is
// ds/dx), with E''(s) evaluated at s^2 = 1e-6 below that (the reference's gassThreshold,
// GIPC.cu:3171); E'' >= 0 on s < 1, so the Hessian is positive semi-definite as it stands.
// ds/dx is the forward derivative of the distance formula.  The mollified near-parallel
// edge-edge encodings (x >= 0 with w < 0; x < 0 with y < 0 and z < 0 or w < 0) are not
// produced here: such a pair gets zero blocks and counts in *skipped.
//
// Output per pair, in fixed slots (no atomics): 10 upper 3x3 blocks (column-major) for the
// local vertex pairs (i <= j) of up to four vertices (unused slots: a zero block on the first
// vertex's diagonal) and 12 gradient entries (3 per local vertex).
#include "solver.hpp"

namespace stg
{

__device__ __forceinline__ void v_cross(const double* a, const double* b, double* r)
{
    r[0] = a[1] * b[2] - a[2] * b[1];
    r[1] = a[2] * b[0] - a[0] * b[2];
    r[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ double v_dot(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// squared distance of the pair's type (_d_PP / _d_PE / _d_PT / _d_EE, mlbvh.cu:229-257)
__device__ __forceinline__ double squared_distance(int type, const double (&x)[4][3])
{
    // type 0: u; 1: |u x v|^2 / |w|^2; 2 and 3: (w . (u x v))^2 / |u x v|^2
    double u[3], v[3], w[3], n[3];
#pragma unroll
    for(int k = 0; k < 3; k++)
    {
        u[k] = type == 0 ? x[0][k] - x[1][k] : (type == 2 ? x[2][k] - x[1][k] : x[1][k] - x[0][k]);
        v[k] = type == 1 ? x[2][k] - x[0][k] : (type == 2 ? x[3][k] - x[1][k] : x[3][k] - x[2][k]);
        w[k] = type == 1 ? x[2][k] - x[1][k] : (type == 2 ? x[0][k] - x[1][k] : x[2][k] - x[0][k]);
    }
    if(type == 0) return v_dot(u, u);
    v_cross(u, v, n);
    if(type == 1) return v_dot(n, n) / v_dot(w, w);
    const double a = v_dot(w, n);
    return a * a / v_dot(n, n);
}

// E'(s) and E''(s) of kappa dHat^2 (s^2 - 1)^2 ln^2(s^2) (RANK 2, GIPC.cu:3226-3230, 3285-3303)
__device__ __forceinline__ void barrier_derivs(double s, double dhat, double kappa, double& e1, double& e2)
{
    const double I = s * s, lI = log(I);
    e1 = s * 2.0 * (2.0 * kappa * dhat * dhat * lI * (I - 1.0) * (I + I * lI - 1.0)) / I;
    const double Ic = I < 1e-6 ? 1e-6 : I, l = log(Ic);
    e2 = -(4.0 * kappa * dhat * dhat *
           (4.0 * Ic + l - 3.0 * Ic * Ic * l * l + 6.0 * Ic * l - 2.0 * Ic * Ic + Ic * l * l - 7.0 * Ic * Ic * l - 2.0)) /
         Ic;
}

// Squared distance and its gradient: the forward derivative of the formulas of squared_distance
// with its zeros left out.  A vertex moves the difference vectors u, v, w by su, sv, sw (0 or
// +-1) times a unit vector e_k, so of n = u x v only the two components beside k change.  Every
// term and sum is the one that differentiating with all 12 partials forms, in its order, with
// p2 for the derivative of a square (x' x + x x').
__device__ __forceinline__ double p2(double dx, double x) { return fma(dx, x, dx * x); }

// derivative of the components k + 1 and k + 2 of u x v
__device__ __forceinline__ void d_cross(const double* u, const double* v, int k, double su, double sv, double& d1, double& d2)
{
    const int k1 = (k + 1) % 3, k2 = (k + 2) % 3;
    d1 = sv * u[k2] - su * v[k2];
    d2 = su * v[k1] - sv * u[k1];
}

__device__ __forceinline__ double distance2_gradient(int type, const double (&x)[4][3], double (&g)[4][3])
{
    if(type == 0)
    {
        double d[3];
#pragma unroll
        for(int k = 0; k < 3; k++)
        {
            d[k] = x[0][k] - x[1][k];
            g[0][k] = 2.0 * d[k];
            g[1][k] = -2.0 * d[k];
        }
        return v_dot(d, d);
    }
    if(type == 1)
    {
        // |u x v|^2 / |e|^2, u = x1 - x0, v = x2 - x0, e = x2 - x1
        double u[3], v[3], e[3], n[3];
#pragma unroll
        for(int k = 0; k < 3; k++) u[k] = x[1][k] - x[0][k], v[k] = x[2][k] - x[0][k], e[k] = x[2][k] - x[1][k];
        v_cross(u, v, n);
        const double den = v_dot(e, e), q = v_dot(n, n) / den, ib = 1.0 / den;
#pragma unroll
        for(int m = 0; m < 3; m++)
#pragma unroll
            for(int k = 0; k < 3; k++)
            {
                const double su = m == 0 ? -1.0 : (m == 1 ? 1.0 : 0.0), sv = m == 0 ? -1.0 : (m == 2 ? 1.0 : 0.0);
                const double se = m == 1 ? -1.0 : (m == 2 ? 1.0 : 0.0);
                double d1, d2;
                d_cross(u, v, k, su, sv, d1, d2);
                const double dn = p2(d1, n[(k + 1) % 3]) + p2(d2, n[(k + 2) % 3]);
                g[m][k] = fma(-q, 2.0 * se * e[k], dn) * ib;
            }
        return q;
    }
    // (w . n)^2 / |n|^2 with n = u x v: point-triangle u = x2 - x1, v = x3 - x1, w = x0 - x1;
    // edge-edge u = x1 - x0, v = x3 - x2, w = x2 - x0
    double u[3], v[3], w[3], n[3];
#pragma unroll
    for(int k = 0; k < 3; k++)
    {
        u[k] = type == 2 ? x[2][k] - x[1][k] : x[1][k] - x[0][k];
        v[k] = type == 2 ? x[3][k] - x[1][k] : x[3][k] - x[2][k];
        w[k] = type == 2 ? x[0][k] - x[1][k] : x[2][k] - x[0][k];
    }
    v_cross(u, v, n);
    const double a = v_dot(w, n), den = v_dot(n, n), q = a * a / den, ib = 1.0 / den;
#pragma unroll
    for(int m = 0; m < 4; m++)
    {
        const double su = type == 2 ? (m == 1 ? -1.0 : (m == 2 ? 1.0 : 0.0)) : (m == 0 ? -1.0 : (m == 1 ? 1.0 : 0.0));
        const double sv = type == 2 ? (m == 1 ? -1.0 : (m == 3 ? 1.0 : 0.0)) : (m == 2 ? -1.0 : (m == 3 ? 1.0 : 0.0));
        const double sw = type == 2 ? (m == 0 ? 1.0 : (m == 1 ? -1.0 : 0.0)) : (m == 0 ? -1.0 : (m == 2 ? 1.0 : 0.0));
#pragma unroll
        for(int k = 0; k < 3; k++)
        {
            const int k1 = (k + 1) % 3, k2 = (k + 2) % 3;
            double d1, d2, t[3];
            d_cross(u, v, k, su, sv, d1, d2);
            t[k] = sw * n[k];
            t[k1] = __dmul_rn(w[k1], d1);
            t[k2] = __dmul_rn(w[k2], d2);
            const double da = t[0] + t[1] + t[2];
            const double dn = p2(d1, n[k1]) + p2(d2, n[k2]);
            g[m][k] = fma(-q, dn, p2(da, a)) * ib;
        }
    }
    return q;
}

// One thread per pair.  A warp's 32 pairs' outputs are contiguous (720, 96 and 40 bytes a pair)
// and pass through shared memory, the blocks five at a time (45 doubles a pair: an odd stride),
// so that they leave in long runs; written by each thread in place, every store instruction
// touched 32 sectors for 8 bytes each.  30,001 pairs (27 MB out) took 24.6 us that way, with a
// gradient that carried all 12 partials through every operation (122 registers); 9.2 us now,
// 2.9 TB/s written.
constexpr int CT = 64, CT_ROW = 45;

__global__ void __launch_bounds__(CT) k_contact_barrier(int ncp, const int4* __restrict__ pairs,
                                                        const double* __restrict__ x, int nv, int block_offset,
                                                        double dhat, double kappa, int* rows, int* cols, double* blocks,
                                                        double* grad, int* skipped)
{
    __shared__ double sm[CT / 32][32 * CT_ROW];
    const int lane = threadIdx.x & 31;
    double* sw = sm[threadIdx.x >> 5];
    const int p0 = blockIdx.x * CT + (threadIdx.x & ~31), np = min(32, ncp - p0);
    if(np <= 0) return;
    const int p = p0 + lane;
    const bool on = lane < np;
    int vid[4] = {0, 0, 0, 0}, cnt = 0;
    bool ok = false;
    double h[12] = {0.0}, lam = 0.0, e1 = 0.0;
    if(on)
    {
        const int4 q = pairs[p];
        int type = -1;
        if(q.x >= 0)
        {
            if(q.w >= 0)
            {
                type = 3;
                vid[0] = q.x, vid[1] = q.y, vid[2] = q.z, vid[3] = q.w, cnt = 4;
            }
        }
        else if(q.y >= 0)
        {
            const int v0 = -q.x - 1;
            if(q.z < 0)
                type = 0, vid[0] = v0, vid[1] = q.y, cnt = 2;
            else if(q.w < 0)
                type = 1, vid[0] = v0, vid[1] = q.y, vid[2] = q.z, cnt = 3;
            else
                type = 2, vid[0] = v0, vid[1] = q.y, vid[2] = q.z, vid[3] = q.w, cnt = 4;
        }
        ok = type >= 0;
#pragma unroll
        for(int i = 0; i < 4; i++) ok = ok && (i >= cnt || (vid[i] >= 0 && vid[i] < nv));
#pragma unroll
        for(int i = 0; i < 4; i++)
#pragma unroll
            for(int j = i + 1; j < 4; j++) ok = ok && (j >= cnt || vid[i] != vid[j]);
        if(ok)
        {
            double v[4][3], g[4][3] = {};
#pragma unroll
            for(int i = 0; i < 4; i++)
#pragma unroll
                for(int k = 0; k < 3; k++) v[i][k] = i < cnt ? x[3 * (size_t)vid[i] + k] : 0.0;
            const double d2 = distance2_gradient(type, v, g);
            const double d = sqrt(d2), rs = 1.0 / sqrt(dhat);
            const double s = d * rs;
            if(s < 1.0 && s > 0.0)
            {
                barrier_derivs(s, dhat, kappa, e1, lam);
                const double f = 0.5 / d;  // dd/dx = f dd2/dx
#pragma unroll
                for(int k = 0; k < 12; k++) h[k] = g[k / 3][k % 3] * f * rs;
            }
        }
        else if(skipped)
            atomicAdd(skipped, 1);
    }
    // the 10 upper blocks (i <= j) of lam h h^T, oriented upper in the global numbering: element
    // (a, b) = lam h[3i + a] h[3j + b], column-major, the transposed block when the order swaps
#pragma unroll
    for(int half = 0; half < 2; half++)
    {
        int slot = 0;
#pragma unroll
        for(int i = 0; i < 4; i++)
#pragma unroll
            for(int j = i; j < 4; j++, slot++)
            {
                if(slot / 5 != half) continue;
                const bool used = ok && j < cnt, sw_ = used && vid[i] > vid[j];
                double* B = sw + lane * CT_ROW + 9 * (slot % 5);
#pragma unroll
                for(int a = 0; a < 3; a++)
#pragma unroll
                    for(int b = 0; b < 3; b++) B[sw_ ? a * 3 + b : b * 3 + a] = used ? lam * h[3 * i + a] * h[3 * j + b] : 0.0;
            }
        __syncwarp();
        double* out = blocks + 90 * (size_t)p0 + CT_ROW * half;
        for(int e = lane, t = 0, r = lane; e < np * CT_ROW; e += 32, r += 32)
        {
            if(r >= CT_ROW) r -= CT_ROW, t++;
            out[90 * (size_t)t + r] = sw[e];
        }
        __syncwarp();
    }
    // gradient, 3 per local vertex (13 doubles a pair in shared memory), then the block indices
    int* si = reinterpret_cast<int*>(sw + 32 * 13);
#pragma unroll
    for(int k = 0; k < 12; k++) sw[13 * lane + k] = e1 * h[k];
    int slot = 0;
#pragma unroll
    for(int i = 0; i < 4; i++)
#pragma unroll
        for(int j = i; j < 4; j++, slot++)
        {
            const bool used = ok && j < cnt;
            si[10 * lane + slot] = block_offset + (used ? min(vid[i], vid[j]) : (ok ? vid[0] : 0));
            si[320 + 10 * lane + slot] = block_offset + (used ? max(vid[i], vid[j]) : (ok ? vid[0] : 0));
        }
    __syncwarp();
    for(int e = lane; e < 12 * np; e += 32) grad[12 * (size_t)p0 + e] = sw[e + e / 12];
    for(int e = lane; e < 10 * np; e += 32)
    {
        rows[10 * (size_t)p0 + e] = si[e];
        cols[10 * (size_t)p0 + e] = si[320 + e];
    }
}

// per-pair barrier energy kappa dHat^2 (s^2 - 1)^2 ln^2(s^2) for s < 1 (the reference's
// barrier at RANK 2, GIPC.cu:3226-3230 integrated); unsupported or invalid pairs give 0
__global__ void k_contact_energy(int ncp, const int4* __restrict__ pairs, const double* __restrict__ x, int nv,
                                 double dhat, double kappa, double* energy)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if(p >= ncp) return;
    const int4 q = pairs[p];
    int vid[4] = {0, 0, 0, 0}, cnt = 0, type = -1;
    if(q.x >= 0)
    {
        if(q.w >= 0) type = 3, vid[0] = q.x, vid[1] = q.y, vid[2] = q.z, vid[3] = q.w, cnt = 4;
    }
    else if(q.y >= 0)
    {
        vid[0] = -q.x - 1, vid[1] = q.y;
        if(q.z < 0)
            type = 0, cnt = 2;
        else if(q.w < 0)
            type = 1, vid[2] = q.z, cnt = 3;
        else
            type = 2, vid[2] = q.z, vid[3] = q.w, cnt = 4;
    }
    bool ok = type >= 0;
    for(int i = 0; i < cnt; i++) ok = ok && vid[i] >= 0 && vid[i] < nv;
    for(int i = 0; i < cnt; i++)
        for(int j = i + 1; j < cnt; j++) ok = ok && vid[i] != vid[j];
    double e = 0.0;
    if(ok)
    {
        double v[4][3];
#pragma unroll
        for(int i = 0; i < 4; i++)
#pragma unroll
            for(int k = 0; k < 3; k++) v[i][k] = x[3 * (size_t)vid[i < cnt ? i : 0] + k];
        const double I = squared_distance(type, v) / dhat;
        if(I < 1.0)
        {
            const double l = log(I);
            e = kappa * dhat * dhat * (I - 1.0) * (I - 1.0) * l * l;
        }
    }
    energy[p] = e;
}

}  // namespace stg

extern "C" int stg_contact_energy(int ncp, const int32_t* pairs, const double* x, int num_verts, double dhat,
                                  double kappa, double* energy, void* stream)
{
    if(ncp < 0 || num_verts < 0 || !(dhat > 0.0) || !(kappa >= 0.0) || (ncp > 0 && (!pairs || !x || !energy)))
    {
        stg::set_error("stg_contact_energy: invalid arguments");
        return STG_ERR_INVALID;
    }
    if(ncp == 0) return STG_OK;
    stg::k_contact_energy<<<(ncp + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(
        ncp, reinterpret_cast<const int4*>(pairs), x, num_verts, dhat, kappa, energy);
    STG_CUDA_TRY(cudaGetLastError());
    return STG_OK;
}

extern "C" int stg_contact_barrier(int ncp, const int32_t* pairs, const double* x, int num_verts, int block_offset,
                                   double dhat, double kappa, int32_t* rows, int32_t* cols, double* blocks,
                                   double* grad, int* skipped, void* stream)
{
    if(ncp < 0 || num_verts < 0 || block_offset < 0 || !(dhat > 0.0) || !(kappa >= 0.0) ||
       (ncp > 0 && (!pairs || !x || !rows || !cols || !blocks || !grad)))
    {
        stg::set_error("stg_contact_barrier: invalid arguments");
        return STG_ERR_INVALID;
    }
    if(ncp == 0) return STG_OK;
    stg::k_contact_barrier<<<(ncp + stg::CT - 1) / stg::CT, stg::CT, 0, static_cast<cudaStream_t>(stream)>>>(
        ncp, reinterpret_cast<const int4*>(pairs), x, num_verts, block_offset, dhat, kappa, rows, cols, blocks, grad,
        skipped);
    STG_CUDA_TRY(cudaGetLastError());
    return STG_OK;
}
