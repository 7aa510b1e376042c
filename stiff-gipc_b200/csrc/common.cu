// common.cu -- error state and the exclusive scan used by the build stages.
#include "common.cuh"

#include <cooperative_groups.h>

namespace stg
{

static thread_local std::string g_error = "no error";

void set_error(const std::string& msg) { g_error = msg; }
const char* last_error() { return g_error.c_str(); }

// Exclusive scan.  A round scans 16 values per thread of 1,024 (16,384), read and written as
// int4 when both arrays are 16-byte aligned.  One CTA takes 2.7 us for up to one round, then
// about 3.6 us per round (latency of one SM: 30 us at 117,649 values); so more values than
// SCAN_ONE go to one cluster of CL CTAs, each scanning a contiguous part: the parts' sums are
// exchanged over distributed shared memory, and a part of one round keeps its values in
// registers in between.
constexpr int SCAN_PT = 16, SCAN_ROUND = SCAN_PT * 1024, SCAN_CL = 8, SCAN_ONE = SCAN_ROUND;

__device__ __forceinline__ void scan_load(const int* in, int idx, int end, bool vec, int (&v)[SCAN_PT])
{
    if(vec && idx + SCAN_PT <= end)
    {
#pragma unroll
        for(int q = 0; q < SCAN_PT / 4; q++)
        {
            const int4 t = reinterpret_cast<const int4*>(in + idx)[q];
            v[4 * q] = t.x;
            v[4 * q + 1] = t.y;
            v[4 * q + 2] = t.z;
            v[4 * q + 3] = t.w;
        }
    }
    else
    {
#pragma unroll
        for(int q = 0; q < SCAN_PT; q++) v[q] = idx + q < end ? in[idx + q] : 0;
    }
}

// this thread's offset inside the round and the round's total (every thread gets it)
__device__ __forceinline__ int scan_round(const int (&v)[SCAN_PT], int* warp_incl, int& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int local = 0;
#pragma unroll
    for(int q = 0; q < SCAN_PT; q++) local += v[q];
    int x = local;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if(lane >= o) x += y;
    }
    if(lane == 31) warp_incl[warp] = x;
    __syncthreads();
    if(warp == 0)
    {
        int w = warp_incl[lane];
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if(lane >= o) w += y;
        }
        warp_incl[lane] = w;
    }
    __syncthreads();
    const int e = (warp > 0 ? warp_incl[warp - 1] : 0) + x - local;
    total = warp_incl[31];
    __syncthreads();
    return e;
}

template <int CL>
__global__ void __launch_bounds__(1024) k_scan_exclusive(const int* in, int* out, const int* n_dev, int n_host, int* total)
{
    __shared__ int warp_incl[32];
    __shared__ int part_sum;
    int n = n_host;
    if(n_dev)
    {
        const int v = *n_dev;
        n = n_host < 0 ? (v + (-n_host) - 1) / (-n_host) : v;
    }
    const bool vec = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    // this CTA's part [b, e): a multiple of SCAN_PT values per CTA keeps the int4 alignment
    const int len = CL == 1 ? n : ((n + CL - 1) / CL + SCAN_PT - 1) / SCAN_PT * SCAN_PT;
    const int b = CL == 1 ? 0 : min(n, (int)blockIdx.x * len), e = CL == 1 ? n : min(n, b + len);
    int v[SCAN_PT], off = 0, carry = 0, rt = 0;
    if(CL > 1)
    {
        int sum = 0;
        for(int base = b; base < e; base += SCAN_ROUND)
        {
            scan_load(in, base + threadIdx.x * SCAN_PT, e, vec, v);
            off = scan_round(v, warp_incl, rt);
            sum += rt;
        }
        if(threadIdx.x == 0) part_sum = sum;
        auto cluster = cooperative_groups::this_cluster();
        cluster.sync();
        int all = 0;
        for(int r = 0; r < CL; r++)
        {
            const int x = *cluster.map_shared_rank(&part_sum, r);
            if(r < (int)blockIdx.x) carry += x;
            all += x;
        }
        cluster.sync();  // no CTA leaves while another reads its sum
        if(blockIdx.x == 0 && threadIdx.x == 0 && total) *total = all;
    }
    const bool kept = CL > 1 && e - b <= SCAN_ROUND;  // values and offsets still in registers
    for(int base = b; base < e; base += SCAN_ROUND)
    {
        const int idx = base + threadIdx.x * SCAN_PT;
        if(!kept)
        {
            scan_load(in, idx, e, vec, v);
            off = scan_round(v, warp_incl, rt);
        }
        int x = carry + off;
#pragma unroll
        for(int q = 0; q < SCAN_PT; q++)
        {
            const int t = v[q];
            v[q] = x;
            x += t;
        }
        if(vec && idx + SCAN_PT <= e)
        {
#pragma unroll
            for(int q = 0; q < SCAN_PT / 4; q++)
                reinterpret_cast<int4*>(out + idx)[q] = make_int4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
        else
        {
#pragma unroll
            for(int q = 0; q < SCAN_PT; q++)
                if(idx + q < e) out[idx + q] = v[q];
        }
        carry += rt;
    }
    if(CL == 1 && threadIdx.x == 0 && total) *total = carry;
}

int scan_exclusive(const int* in, int* out, const int* n_dev, int n_host, int n_max, int* total, cudaStream_t s)
{
    if(n_max <= SCAN_ONE)
    {
        k_scan_exclusive<1><<<1, 1024, 0, s>>>(in, out, n_dev, n_host, total);
        STG_LAUNCH_CHECK();
        return 0;
    }
    cudaLaunchAttribute at = {};
    const cudaLaunchConfig_t cfg = cluster_config(SCAN_CL, SCAN_CL, 1024, 0, s, &at);
    STG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_scan_exclusive<SCAN_CL>, in, out, n_dev, n_host, total));
    return 0;
}

}  // namespace stg
