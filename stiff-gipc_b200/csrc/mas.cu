// mas.cu -- multilevel additive Schwarz (MAS / CEMAS) preconditioner on sm_100a.
//
// Replaces MASPreconditioner (StiffGIPC/MASPreconditioner.cu):
//   hierarchy  ReorderRealtime (1785-1826) and its kernels (29-625, 1132-1548)
//   assembly   PrepareHessian_bcoo (1829-2075) + __inverse6_P96x96 (630-726)
//   apply      preconditioning (2248-2289): __buildMultiLevelR_optimized_new (729-847),
//              _schwarzLocalXSym6 (957-1027), __collectFinalZ_new (850-879)
//
// Bank size B (BANKSIZE, eigen_data.h:17) is a template parameter: 16 (CEMAS as shipped) or
// 32 (Morton-ordered GPU MAS).  Integer results (masks, coarse ids, tables) are bit-exact
// with the reference's intended semantics; the reference's warp-synchronous shared-memory
// races are replaced by explicit barriers:
//   * in-bank closure (_preparePrefixSumL0_new / _nextLevelCluster) reads the original
//     masks from shared memory written before a __syncthreads;
//   * the union of coarse connectivity masks (_buildConnectMaskLx_new) is formed with
//     atomicOr on the node mask (OR is order independent);
//   * component leaders and counts use ballots instead of racy shared atomics.
// Restriction sums are computed per bank in lane order (deterministic) instead of float
// atomics, and the coarse-level Galerkin blocks are formed level by level with the
// deterministic sort/merge of convert.cu instead of FP64 atomics (see the assembly section).
#include "solver.hpp"
#include "bank_dev.cuh"
#include "mas_index.cuh"

namespace stg
{


// group-local ballot: the B lanes of this lane's bank
template <int B>
__device__ __forceinline__ unsigned group_ballot(bool pred)
{
    const unsigned all = __ballot_sync(0xffffffffu, pred);
    if(B == 32) return all;
    const int shift = (threadIdx.x & 31) & ~(B - 1);
    return (all >> shift) & ((1u << B) - 1u);
}

// ---------------------------------------------------------------------------------------
// hierarchy
// ---------------------------------------------------------------------------------------
// _buildCML0_new (MASPreconditioner.cu:62-98): in-bank neighbour bits; inter-bank neighbours
// are compacted to the front of the vertex's list.
template <int B>
__global__ void k_mas_l0_mask(const int* __restrict__ part_map, const int* __restrict__ real_map,
                              const unsigned* __restrict__ nstart, unsigned* nnum, unsigned* nlist, unsigned* fine_mask,
                              int M)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if(s >= M) return;
    const int v = part_map[s];
    if(v < 0) return;
    const int bank = s / B, lane = s % B;
    unsigned msk = 1u << lane;
    unsigned nk = 0;
    const unsigned st = nstart[v], num = nnum[v];
    for(unsigned i = 0; i < num; i++)
    {
        const unsigned u = nlist[st + i];
        const int su = real_map[u];
        if(su / B == bank)
            msk |= 1u << (su % B);
        else
            nlist[st + nk++] = u;
    }
    nnum[v] = nk;
    fine_mask[v] = msk;
}

// _buildCollisionConnection_new (MASPreconditioner.cu:1132-1548).  coarse == nullptr: level 0
// (ids via real_map, OR into conn[vertex]); otherwise the previous level's coarse table
// (OR into conn[coarse id]).
template <int B>
__device__ __forceinline__ void contact_connect(unsigned* conn, const int* coarse, const int* __restrict__ real_map,
                                                const int4 q, int node_offset, int V)
{
    int v[4] = {q.x, q.y, q.z, q.w};
    int cnt = 4;
    if(v[0] >= 0)
    {
        if(v[3] < 0) v[3] = -v[3] - 1;
    }
    else
    {
        v[0] = -v[0] - 1;
        if(v[2] < 0)
        {
            if(v[1] < 0)
            {
                v[1] = -v[1] - 1;
                v[2] = -v[2] - 1;
                v[3] = -v[3] - 1;
            }
            else
                cnt = 2;
        }
        else if(v[3] < 0)
        {
            if(v[1] < 0)
            {
                v[1] = -v[1] - 1;
                v[3] = -v[3] - 1;
            }
            else
                cnt = 3;
        }
    }
    int vid[4], cpv[4];
    unsigned msk[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for(int i = 0; i < 4; i++)
    {
        const int id = v[i] - node_offset;
        vid[i] = (i < cnt && id >= 0 && id < V) ? id : -1;
        cpv[i] = vid[i] >= 0 ? (coarse ? __ldcg(coarse + vid[i]) : real_map[vid[i]]) : -1;
    }
#pragma unroll
    for(int i = 0; i < 4; i++)
#pragma unroll
        for(int j = i + 1; j < 4; j++)
        {
            const int a = cpv[i], b = cpv[j];
            if(a == b || a < 0 || b < 0) continue;
            if(a / B == b / B)
            {
                msk[i] |= 1u << (b % B);
                msk[j] |= 1u << (a % B);
            }
        }
#pragma unroll
    for(int i = 0; i < 4; i++)
    {
        if(coarse)
        {
            if(cpv[i] >= 0 && msk[i]) atomicOr(conn + cpv[i], msk[i]);
        }
        else if(vid[i] >= 0 && msk[i])
            atomicOr(conn + vid[i], msk[i]);
    }
}

template <int B>
__global__ void k_mas_contacts(unsigned* conn, const int* __restrict__ coarse, const int* __restrict__ real_map,
                               const int4* __restrict__ pairs, int ncp, int node_offset, int V)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if(p < ncp) contact_connect<B>(conn, coarse, real_map, pairs[p], node_offset, V);
}

// Reachable set of `lane` through the bank's original masks (the visit loop of
// _preparePrefixSumL0_new / _nextLevelCluster), masks read from shared memory.
__device__ __forceinline__ unsigned bank_closure(const unsigned* orig, int lane, unsigned start)
{
    unsigned conn = start, visited = 1u << lane;
    for(;;)
    {
        const unsigned todo = visited ^ conn;
        if(!todo) break;
        const int nv = __ffs(todo) - 1;
        visited |= 1u << nv;
        conn |= orig[nv];
    }
    return conn;
}

// _preparePrefixSumL0_new (MASPreconditioner.cu:159-214): closure + component count per bank.
template <int B>
__global__ void __launch_bounds__(256) k_mas_l0_closure(const int* __restrict__ part_map, unsigned* fine_mask,
                                                        int* prefix_orig, int M)
{
    __shared__ unsigned orig[256];
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = s % B;
    const int v = s < M ? part_map[s] : -1;
    orig[threadIdx.x] = v >= 0 ? fine_mask[v] : 0u;
    __syncthreads();
    bool leader = false;
    if(v >= 0)
    {
        const unsigned* bank_orig = orig + (threadIdx.x & ~(B - 1));
        const unsigned c = bank_closure(bank_orig, lane, bank_orig[lane]);
        fine_mask[v] = c;
        leader = __popc(c & lanemask_lt(lane)) == 0;
    }
    const unsigned lm = group_ballot<B>(leader);
    if(lane == 0 && s < M) prefix_orig[s / B] = __popc(lm);
}

// _buildLevel1_new (MASPreconditioner.cu:270-328): level-1 ids in leader-lane order.
template <int B>
__global__ void k_mas_l1_assign(const int* __restrict__ part_map, const unsigned* __restrict__ fine_mask,
                                const int* __restrict__ prefix_sum_orig, int* coarse_tables, int* going_next, int M)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = s % B;
    const int v = s < M ? part_map[s] : -1;
    const unsigned c = v >= 0 ? fine_mask[v] : 0u;
    const bool leader = v >= 0 && __popc(c & lanemask_lt(lane)) == 0;
    const unsigned elected = group_ballot<B>(leader);
    if(v < 0) return;
    const int lead = __ffs(c) - 1;
    const int id = __popc(elected & lanemask_lt(lead)) + prefix_sum_orig[s / B];
    coarse_tables[v] = id;
    going_next[v] = id + M;
}

// _buildConnectMaskLx_new (MASPreconditioner.cu:401-470) with union semantics.
template <int B>
__global__ void k_mas_lx_mask(const int* __restrict__ part_map, const unsigned* __restrict__ nstart, unsigned* nnum,
                              unsigned* nlist, const int* __restrict__ prev, unsigned* next_mask, int M)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if(s >= M) return;
    const int v = part_map[s];
    if(v < 0) return;
    const unsigned c = (unsigned)prev[v];
    unsigned msk = 0, nk = 0;
    const unsigned st = nstart[v], num = nnum[v];
    for(unsigned i = 0; i < num; i++)
    {
        const unsigned u = nlist[st + i];
        const unsigned cu = (unsigned)prev[u];
        if(c / B == cu / B)
            msk |= 1u << (cu % B);
        else
            nlist[st + nk++] = u;
    }
    nnum[v] = nk;
    if(msk) atomicOr(next_mask + c, msk);
}

// _nextLevelCluster (MASPreconditioner.cu:473-520): closure over level-l banks.
// ls: level sizes (count, begin) pairs; level = l.
template <int B>
__global__ void __launch_bounds__(256) k_mas_lx_closure(unsigned* next_mask, unsigned* closed, int* next_prefix,
                                                        const int* __restrict__ ls, int level)
{
    __shared__ unsigned orig[256];
    const int number = ls[2 * level], begin = ls[2 * level + 1];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = i % B;
    const bool valid = i < number;
    orig[threadIdx.x] = valid ? ((1u << lane) | next_mask[i]) : 0u;
    __syncthreads();
    bool leader = false;
    if(valid)
    {
        const unsigned* bank_orig = orig + (threadIdx.x & ~(B - 1));
        const unsigned c = bank_closure(bank_orig, lane, bank_orig[lane]);
        next_mask[i] = c;
        closed[begin + i] = c;
        leader = __popc(c & lanemask_lt(lane)) == 0;
    }
    const unsigned lm = group_ballot<B>(leader);
    if(lane == 0 && i < number) next_prefix[i / B] = __popc(lm);
}

// _prefixSumLx (MASPreconditioner.cu:522-566): next-level ids; also records the level size.
template <int B>
__global__ void k_mas_lx_assign(unsigned* next_mask, const int* __restrict__ next_prefix_sum, int* going_next,
                                int* lead_of, int* ls, int level)
{
    const int number = ls[2 * level], begin = ls[2 * level + 1];
    const int rounded = (number + B - 1) / B * B;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = i % B;
    const bool valid = i < number;
    const unsigned c = valid ? next_mask[i] : 0u;
    const bool leader = valid && __popc(c & lanemask_lt(lane)) == 0;
    const unsigned elected = group_ballot<B>(leader);
    if(i == 0) ls[2 * (level + 1) + 1] = begin + rounded;
    if(!valid) return;
    const int lead = __ffs(c) - 1;
    const int id = __popc(elected & lanemask_lt(lead)) + next_prefix_sum[i / B];
    next_mask[i] = (unsigned)id;
    going_next[begin + i] = id + begin + rounded;
    if(leader) lead_of[id + begin + rounded] = begin + i;
}

// _computeNextLevel (MASPreconditioner.cu:568-579)
__global__ void k_mas_compute_next(int* coarse_tables, const unsigned* __restrict__ next_mask, int level, int V)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if(v >= V) return;
    coarse_tables[(size_t)level * V + v] = (int)next_mask[coarse_tables[(size_t)(level - 1) * V + v]];
}

// _aggregationKernel (MASPreconditioner.cu:581-608)
__global__ void k_mas_aggregate(const int* __restrict__ going_next, int* coarse_table, int L, int V)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if(v >= V) return;
    int cur = v;
    for(int l = 0; l < L - 1; l++)
    {
        cur = going_next[cur];
        coarse_table[(size_t)v * (L - 1) + l] = cur;
    }
}

// scan driver: n = ceil(ls[2*level] / div) when ls != nullptr
__global__ void k_set_level1(int* ls, const int* total, int M)
{
    ls[2] = *total;
    ls[3] = M;
}

// ---------------------------------------------------------------------------------------
// The whole hierarchy in one launch, for meshes of up to MB_MAX_SLOTS slots: one cluster of 16
// CTAs of 1,024 threads, the steps of the kernels above separated by cluster barriers (0.5 us)
// instead of launches (about 4 us each, 6 a level: 122 us for 343 vertices and 152 us for 4,913,
// of which the kernels' work was a few microseconds a level).  Larger meshes keep the separate
// kernels, whose neighbour walks need the whole GPU.  Same integers: a component's id is the
// number of component leaders before its own in slot order.
// ---------------------------------------------------------------------------------------
constexpr int MB_CL = 16, MB_T = 1024, MB_ROUNDS = 2, MB_MAX_SLOTS = MB_CL * MB_T * MB_ROUNDS;

struct MasBuildArgs
{
    const int* part_map;
    const int* real_map;
    const unsigned* nstart;
    const unsigned* nnum_init;
    const unsigned* nlist_init;
    unsigned* nnum;
    unsigned* nlist;
    unsigned* fine_mask;
    int* prefix_orig;
    int* coarse_tables;
    int* going_next;
    unsigned* closed;
    int* lead;
    int* coarse_table;
    unsigned* next_mask;  // two buffers of V + B
    int* ls;
    const int4* pairs;
    int ncp, node_offset, V, M, L;
};

__device__ __forceinline__ void mb_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int B>
__global__ void __launch_bounds__(MB_T) k_mas_build_small(MasBuildArgs A)
{
    __shared__ unsigned orig[MB_T];
    __shared__ int wcnt[MB_T / 32];
    __shared__ int part;
    const int rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gt = rank * MB_T + tid, gn = MB_CL * MB_T;

    // closure of the banks over nodes [0, number) and ids in leader order: load(i, msk) gives
    // node i's mask (false: no node), done(i, c, id, leader) stores.  Returns the id count.
    auto level_pass = [&](int number, auto load, auto done, int* bank_count) -> int {
        const int span = (number + 31) / 32 * 32;
        const int chunk = ((span + MB_CL - 1) / MB_CL + 31) / 32 * 32;
        const int lo = min(span, rank * chunk), hi = min(span, lo + chunk);
        unsigned c[MB_ROUNDS], ball[MB_ROUNDS];
        int base[MB_ROUNDS], carry = 0;
        bool valid[MB_ROUNDS];
#pragma unroll
        for(int r = 0; r < MB_ROUNDS; r++)
        {
            const int i = lo + r * MB_T + tid;
            unsigned m = 0u;
            valid[r] = i < hi && i < number && load(i, m);
            orig[tid] = valid[r] ? m : 0u;
            __syncthreads();
            c[r] = 0u;
            bool leader = false;
            if(valid[r])
            {
                const unsigned* bo = orig + (tid & ~(B - 1));
                c[r] = bank_closure(bo, tid % B, bo[tid % B]);
                leader = __popc(c[r] & lanemask_lt(tid % B)) == 0;
            }
            ball[r] = __ballot_sync(0xffffffffu, leader);
            if(lane == 0) wcnt[warp] = __popc(ball[r]);
            if(bank_count && i < hi && i < number && tid % B == 0)
                bank_count[i / B] = __popc(B == 32 ? ball[r] : (ball[r] >> (lane & ~(B - 1))) & ((1u << (B & 31)) - 1u));
            __syncthreads();
            int x = wcnt[lane];
#pragma unroll
            for(int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if(lane >= o) x += y;
            }
            base[r] = carry + (warp > 0 ? __shfl_sync(0xffffffffu, x, max(warp - 1, 0)) : 0);
            carry += __shfl_sync(0xffffffffu, x, 31);
            __syncthreads();
        }
        if(tid == 0) part = carry;
        mb_barrier();
        // lane q reads CTA q's count: one round trip for all of them
        static_assert(MB_CL <= 32, "one lane per CTA");
        int mine = 0;
        if(lane < MB_CL)
        {
            unsigned a, v;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                         : "=r"(a)
                         : "r"((unsigned)__cvta_generic_to_shared(&part)), "r"(lane));
            asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
            mine = (int)v;
        }
        const int total = __reduce_add_sync(0xffffffffu, mine);
        const int off = __reduce_add_sync(0xffffffffu, lane < rank ? mine : 0);
#pragma unroll
        for(int r = 0; r < MB_ROUNDS; r++)
            if(valid[r])
            {
                const int ld = (lane & ~(B - 1)) + __ffs(c[r]) - 1;
                done(lo + r * MB_T + tid, c[r], off + base[r] + __popc(ball[r] & lanemask_lt(ld)), ld == lane);
            }
        return total;
    };
    // neighbours eight at a time: all their loads in flight before the list is compacted
    auto neighbours = [&](const unsigned* list, unsigned st, unsigned num, auto key, auto mine) -> unsigned {
        unsigned nk = 0;
        for(unsigned i0 = 0; i0 < num; i0 += 8)
        {
            unsigned u[8];
            int k[8];
#pragma unroll
            for(int q = 0; q < 8; q++) u[q] = i0 + q < num ? __ldcg(list + st + i0 + q) : 0u;
#pragma unroll
            for(int q = 0; q < 8; q++) k[q] = i0 + q < num ? key(u[q]) : 0;
#pragma unroll
            for(int q = 0; q < 8; q++)
                if(i0 + q < num && !mine(k[q])) A.nlist[st + nk++] = u[q];
        }
        return nk;
    };

    for(int i = gt; i < A.M; i += gn)
    {
        const int v = A.part_map[i];
        if(v < 0) continue;
        unsigned msk = 1u << (i % B);
        A.nnum[v] = neighbours(
            A.nlist_init, A.nstart[v], A.nnum_init[v], [&](unsigned u) { return A.real_map[u]; },
            [&](int su) {
                if(su / B != i / B) return false;
                msk |= 1u << (su % B);
                return true;
            });
        A.fine_mask[v] = msk;
    }
    mb_barrier();
    if(A.ncp > 0)
    {
        for(int p = gt; p < A.ncp; p += gn) contact_connect<B>(A.fine_mask, nullptr, A.real_map, A.pairs[p], A.node_offset, A.V);
        mb_barrier();
    }
    const bool table = A.L > 1;
    int number = level_pass(
        A.M,
        [&](int i, unsigned& m) {
            const int v = A.part_map[i];
            if(v >= 0) m = __ldcg(A.fine_mask + v);
            return v >= 0;
        },
        [&](int i, unsigned c, int id, bool) {
            const int v = A.part_map[i];
            A.fine_mask[v] = c;
            A.coarse_tables[v] = id;
            A.going_next[v] = id + A.M;
            if(table) A.coarse_table[(size_t)v * (A.L - 1)] = id + A.M;
        },
        A.prefix_orig);
    int begin = A.M;
    if(gt == 0)
    {
        A.ls[0] = A.ls[1] = 0;
        A.ls[2] = number;
        A.ls[3] = begin;
    }
    for(int level = 1; level < A.L; level++)
    {
        unsigned* nm = A.next_mask + (size_t)(level & 1) * (A.V + B);
        const int* prev = A.coarse_tables + (size_t)(level - 1) * A.V;
        for(int i = gt; i < number; i += gn) nm[i] = 0u;
        mb_barrier();
        for(int i = gt; i < A.M; i += gn)
        {
            const int v = A.part_map[i];
            if(v < 0) continue;
            const unsigned c = (unsigned)__ldcg(prev + v);
            unsigned msk = 0u;
            A.nnum[v] = neighbours(
                A.nlist, A.nstart[v], __ldcg(A.nnum + v), [&](unsigned u) { return __ldcg(prev + u); },
                [&](int cu) {
                    if(c / B != (unsigned)cu / B) return false;
                    msk |= 1u << (cu % B);
                    return true;
                });
            if(msk) atomicOr(nm + c, msk);
        }
        for(int p = gt; p < A.ncp; p += gn) contact_connect<B>(nm, prev, A.real_map, A.pairs[p], A.node_offset, A.V);
        mb_barrier();
        const int next = begin + (number + B - 1) / B * B;
        const int total = level_pass(
            number,
            [&](int i, unsigned& m) {
                m = (1u << (i % B)) | __ldcg(nm + i);
                return true;
            },
            [&](int i, unsigned c, int id, bool leader) {
                A.closed[begin + i] = c;
                nm[i] = (unsigned)id;
                A.going_next[begin + i] = id + next;
                if(leader) A.lead[id + next] = begin + i;
            },
            nullptr);
        mb_barrier();
        for(int v = gt; v < A.V; v += gn)
        {
            const int id = (int)__ldcg(nm + __ldcg(prev + v));
            A.coarse_tables[(size_t)level * A.V + v] = id;
            if(level < A.L - 1) A.coarse_table[(size_t)v * (A.L - 1) + level] = id + next;
        }
        number = total;
        begin = next;
        if(gt == 0)
        {
            A.ls[2 * (level + 1)] = number;
            A.ls[2 * (level + 1) + 1] = begin;
        }
    }
    mb_barrier();  // no CTA leaves while another may read its part
}

// ---------------------------------------------------------------------------------------
// assembly (PrepareHessian_bcoo) and inverse
// ---------------------------------------------------------------------------------------
// PrepareHessian_bcoo (MASPreconditioner.cu:1829-2075) accumulates, for every level l, the
// bank-diagonal blocks of the Galerkin operator P_l^T A P_l: block (a, b) of a level-l bank
// is the sum of A(u, v) over all fine pairs with coarse_l(u) = a, coarse_l(v) = b.  The
// reference walks every BCOO entry and every in-bank level-0 pair up the levels with FP64
// atomics, which serialise on the few coarse blocks every pair reaches.  Here the same sums
// are formed level by level: A_1 = aggregate(A_0), A_{l+1} = aggregate(A_l) (aggregate =
// map both indices to the coarse node and merge duplicates with the deterministic sorter of
// convert.cu), and each level's bank blocks are read off A_l.  Level-0 in-bank entries with
// slot(col) < slot(row) are not stored by the reference (lambda 1 only stores col >= row
// slots, and lambda 2 propagates the stored bank matrix); they are left out here too.

// level-0 bank blocks (lambda 1, level-0 branch): direct stores, entries are unique
template <int B>
__global__ void k_mas_store_l0(const int* __restrict__ rows, const int* __restrict__ cols,
                               const double* __restrict__ blocks, int nnzb, int offset, int V,
                               const int* __restrict__ real_map, double* mat)
{
    const int NS = nsym(B);
    for(int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnzb; k += gridDim.x * blockDim.x)
    {
        const int rr = rows[k] - offset, cc = cols[k] - offset;
        if(rr < 0 || rr >= V || cc < 0 || cc >= V) continue;
        const int sc = real_map[cc], sr = real_map[rr];
        if(sc / B != sr / B || sc < sr) continue;
        const double* H = blocks + 9 * (size_t)k;
        double* D = mat + ((size_t)(sc / B) * NS + upper_index(B, sr % B, sc % B)) * 9;
#pragma unroll
        for(int e = 0; e < 9; e++) D[e] = H[e];
    }
}

// A_0 (FEM range of the BCOO) -> level-1 triplets; masked entries get row -1
template <int B>
__global__ void k_mas_agg_l0(const int* __restrict__ rows, const int* __restrict__ cols, const double* __restrict__ blocks,
                             int nnzb, int offset, int V, const int* __restrict__ real_map, const int* __restrict__ c1,
                             int* orow, int* ocol, double* oblk)
{
    for(int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnzb; k += gridDim.x * blockDim.x)
    {
        const int rr = rows[k] - offset, cc = cols[k] - offset;
        bool use = rr >= 0 && rr < V && cc >= 0 && cc < V;
        if(use)
        {
            const int sc = real_map[cc], sr = real_map[rr];
            use = !(sc / B == sr / B && sc < sr);
        }
        if(!use)
        {
            orow[k] = -1;
            ocol[k] = 0;
            continue;
        }
        coarse_triplet(rr, cc, c1[rr], c1[cc], blocks + 9 * (size_t)k, orow + k, ocol + k, oblk + 9 * (size_t)k);
    }
}

// A_l -> level-(l+1) triplets through going_next (global ids) of level-l nodes
__global__ void k_mas_agg_lx(const int* __restrict__ rows, const int* __restrict__ cols, const double* __restrict__ blocks,
                             int nnz, const int* __restrict__ going_next, int begin, int begin_next, int* orow, int* ocol,
                             double* oblk)
{
    for(int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += gridDim.x * blockDim.x)
    {
        const int u = rows[k], v = cols[k];
        coarse_triplet(u, v, going_next[begin + u] - begin_next, going_next[begin + v] - begin_next,
                       blocks + 9 * (size_t)k, orow + k, ocol + k, oblk + 9 * (size_t)k);
    }
}

// bank-diagonal blocks of A_l (level-local ids, upper) into the packed bank matrices
template <int B>
__global__ void k_mas_extract(const int* __restrict__ rows, const int* __restrict__ cols, const double* __restrict__ blocks,
                              int nnz, int begin, double* mat)
{
    const int NS = nsym(B);
    for(int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += gridDim.x * blockDim.x)
    {
        const int ga = begin + rows[k], gb = begin + cols[k];
        if(ga / B != gb / B) continue;
        double* D = mat + ((size_t)(ga / B) * NS + upper_index(B, ga % B, gb % B)) * 9;
        const double* H = blocks + 9 * (size_t)k;
#pragma unroll
        for(int e = 0; e < 9; e++) D[e] = H[e];
    }
}

// The coarse levels' aggregation in one launch, from the triplets of the first level that has
// at most CHAIN_CAP of them: one CTA sorts a level's triplets by (row, col, index) in shared
// memory (32-bit keys where the level's nodes fit 10 bits), stages three of the nine values of
// all blocks at a time there, sums every run in that order (one thread per value), writes the
// level's operator and bank blocks, and maps it to the next level's triplets.  As separate
// launches a level costs 10 launches and a read-back, about 55 us, for a few thousand triplets;
// here all three levels from 2,197 triplets take 57 us (65 with 64-bit keys alone and runs summed
// from device memory).
// The sums and their order are those of convert_into.
constexpr int CHAIN_CAP = 4096, CHAIN_T = 1024;
constexpr int CHAIN_SMEM = CHAIN_CAP * (8 + 2 + 3 * 8) + 16;
constexpr int CHAIN_NODES32 = 1023;  // nodes that 10-bit rows and columns of a 32-bit key can name

// bitonic sort of P keys (a power of two) in shared memory
template <typename K>
__device__ __forceinline__ void chain_sort(K* key, int P)
{
    for(int k = 2; k <= P; k <<= 1)
        for(int j = k >> 1; j > 0; j >>= 1)
        {
            for(int t = threadIdx.x; t < P / 2; t += CHAIN_T)
            {
                const int a = 2 * t - (t & (j - 1)), b = a + j;  // pairs (a, a ^ j), a & j == 0
                const K x = key[a], y = key[b];
                if((x > y) == ((a & k) == 0)) key[a] = y, key[b] = x;
            }
            __syncthreads();
        }
}

struct ChainArgs
{
    int* tr_rows;
    int* tr_cols;
    double* tr_blocks;
    int count, level, L;      // triplets of `level`, levels
    int begin[kMaxLevels + 1], nodes[kMaxLevels + 1];
    const int* going_next;
    int* rows;                // scratch for one level's operator
    int* cols;
    double* blocks;
    double* mat;
};

template <int B>
__global__ void __launch_bounds__(CHAIN_T) k_mas_chain(ChainArgs A)
{
    extern __shared__ unsigned long long ckey[];
    double* stage = reinterpret_cast<double*>(ckey + CHAIN_CAP);  // [3 * CHAIN_CAP], first the 32-bit keys
    unsigned short* ustart = reinterpret_cast<unsigned short*>(stage + 3 * CHAIN_CAP);  // [CHAIN_CAP + 1]
    __shared__ int wcnt[CHAIN_T / 32];
    __shared__ int live;
    const int NS = nsym(B);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int n = A.count;
    for(int level = A.level;; level++)
    {
        if(tid == 0) live = 0;
        int P = 1;
        while(P < n) P <<= 1;
        __syncthreads();
        const bool small = A.nodes[level] <= CHAIN_NODES32;
        unsigned* k32 = reinterpret_cast<unsigned*>(stage);
        int kept = 0;
        for(int i = tid; i < P; i += CHAIN_T)
        {
            const int r = i < n ? __ldcg(A.tr_rows + i) : -1;
            const unsigned c = r >= 0 ? (unsigned)__ldcg(A.tr_cols + i) : 0u;
            kept += r >= 0;
            if(small)
                k32[i] = r >= 0 ? ((unsigned)r << 22) | (c << 12) | (unsigned)i : ~0u;
            else
                ckey[i] = r >= 0 ? ((unsigned long long)r << 40) | ((unsigned long long)c << 20) | (unsigned)i : ~0ull;
        }
        if(kept) atomicAdd(&live, kept);
        __syncthreads();
        if(small)
        {
            static_assert(CHAIN_CAP <= 4096, "12-bit indices");
            chain_sort(k32, P);
            for(int i = tid; i < P; i += CHAIN_T)
            {
                const unsigned k = k32[i];
                ckey[i] = ((unsigned long long)(k >> 22) << 40) | ((unsigned long long)((k >> 12) & 1023u) << 20) | (k & 4095u);
            }
            __syncthreads();
        }
        else
            chain_sort(ckey, P);
        // run starts: each thread owns a stretch of PT keys, a block scan numbers the runs
        const int m = live, PT = (m + CHAIN_T - 1) / CHAIN_T, i0 = min(m, tid * PT), i1 = min(m, i0 + PT);
        int heads = 0;
        for(int i = i0; i < i1; i++) heads += i == 0 || (ckey[i] >> 20) != (ckey[i - 1] >> 20);
        int x = heads;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if(lane >= o) x += y;
        }
        if(lane == 31) wcnt[warp] = x;
        __syncthreads();
        int w = wcnt[lane];
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if(lane >= o) w += y;
        }
        const int runs = __shfl_sync(0xffffffffu, w, 31);
        int u = x - heads + (warp > 0 ? __shfl_sync(0xffffffffu, w, max(warp - 1, 0)) : 0);
        for(int i = i0; i < i1; i++)
            if(i == 0 || (ckey[i] >> 20) != (ckey[i - 1] >> 20))
            {
                ustart[u] = (unsigned short)i;
                A.rows[u] = (int)(ckey[i] >> 40);
                A.cols[u] = (int)(ckey[i] >> 20) & 0xfffff;
                u++;
            }
        __syncthreads();
        const int begin = A.begin[level];
        for(int p = 0; p < 9; p += 3)
        {
            // values p .. p + 2 of every block in sorted order: independent loads, so that the
            // runs (a diagonal block's holds up to about 100 blocks) sum from shared memory
#pragma unroll 4
            for(int t = tid; t < 3 * m; t += CHAIN_T)
            {
                const int i = t / 3;
                stage[t] = __ldcg(A.tr_blocks + 9 * (size_t)((unsigned)ckey[i] & 0xfffffu) + p + (t - 3 * i));
            }
            __syncthreads();
            for(int t = tid; t < 3 * runs; t += CHAIN_T)
            {
                const int q = t / 3, e = t - 3 * q;
                const int s0 = ustart[q], s1 = q + 1 < runs ? ustart[q + 1] : m;
                double acc = stage[3 * s0 + e];
                for(int i = s0 + 1; i < s1; i++) acc += stage[3 * i + e];
                A.blocks[9 * (size_t)q + p + e] = acc;
                const int ga = begin + (int)(ckey[s0] >> 40), gb = begin + ((int)(ckey[s0] >> 20) & 0xfffff);
                if(ga / B == gb / B) A.mat[((size_t)(ga / B) * NS + upper_index(B, ga % B, gb % B)) * 9 + p + e] = acc;
            }
            __syncthreads();
        }
        if(level + 1 >= A.L || runs == 0) return;
        const int next = A.begin[level + 1];
        for(int i = tid; i < runs; i += CHAIN_T)
        {
            const int r = __ldcg(A.rows + i), c = __ldcg(A.cols + i);
            double H[9];
#pragma unroll
            for(int e = 0; e < 9; e++) H[e] = __ldcg(A.blocks + 9 * (size_t)i + e);
            coarse_triplet(r, c, A.going_next[begin + r] - next, A.going_next[begin + c] - next, H, A.tr_rows + i,
                           A.tr_cols + i, A.tr_blocks + 9 * (size_t)i);
        }
        n = runs;
        __syncthreads();
    }
}

// __inverse6_P96x96 (MASPreconditioner.cu:630-726): in-place Gauss-Jordan without pivoting
// of each bank's dense 3B x 3B matrix in FP64 (zero diagonal -> 1 for padding), lower
// triangle of the diagonal 3x3 blocks mirrored from the upper one, upper blocks stored FP32.
// One CTA per bank, thread i owns column i.  The pivot row is scaled by the correctly rounded
// reciprocal of the pivot (the reference divides; k_mas_invert16 does the same as here, so
// both bank sizes follow one order, the CPU oracle's ORC_ORDER_FIXED).
template <int B>
__global__ void __launch_bounds__(3 * B) k_mas_invert(const double* __restrict__ mat, float* inv, int nbanks)
{
    constexpr int N = 3 * B;
    const int NS = nsym(B);
    extern __shared__ double sm[];
    double* A = sm;            // N*N row-major
    double* colm = sm + N * N; // N
    const int bk = blockIdx.x;
    const int i = threadIdx.x;
    const double* Mb = mat + (size_t)bk * NS * 9;
    for(int j = 0; j < N; j++)
    {
        const int rowId = j / 3, colId = i / 3;
        double v;
        if(colId >= rowId)
            v = Mb[upper_index(B, rowId, colId) * 9 + (i % 3) * 3 + (j % 3)];
        else
            v = Mb[upper_index(B, colId, rowId) * 9 + (j % 3) * 3 + (i % 3)];
        if(i == j && v == 0.0) v = 1.0;
        A[j * N + i] = v;
    }
    for(int j = 0; j < N; j++)
    {
        __syncthreads();
        const double rt = A[j * N + j];
        colm[i] = A[i * N + j];
        __syncthreads();
        A[i * N + j] = (i == j) ? 1.0 : 0.0;
        __syncthreads();
        A[j * N + i] = __dmul_rn(A[j * N + i], 1.0 / rt);
        __syncthreads();
        const double aji = A[j * N + i];
        for(int k = 0; k < N; k++)
        {
            if(k == j) continue;
            A[k * N + i] = fma(-colm[k], aji, A[k * N + i]);
        }
    }
    __syncthreads();
    if(i % 3 < 2)
        A[(i + 1) * N + i] = A[i * N + i + 1];
    else
        A[i * N + i - 2] = A[(i - 2) * N + i];
    __syncthreads();
    float* P = inv + (size_t)bk * NS * 9;
    for(int j = 0; j < N; j++)
    {
        const int rowId = j / 3, colId = i / 3;
        if(colId >= rowId) P[upper_index(B, rowId, colId) * 9 + (i % 3) * 3 + (j % 3)] = (float)A[j * N + i];
    }
}

// The same Gauss-Jordan for 16-banks, one warp per bank: lane (bi, bj) of a 4 x 8 grid holds
// rows 12 bi .. 12 bi + 11, columns 6 bj .. 6 bj + 5 in registers (72 doubles).  Pivot j: the
// lanes of its column publish column j, those of its row scale row j by the reciprocal of the
// pivot and publish it; then every lane updates its tile with fma(-colm[k], A[j][i], A[k][i])
// as k_mas_invert does: 18 shared-memory reads for 72 FMAs and warp barriers only.  (A CTA of
// 256 threads per bank with 3x3 tiles read 6 values for 9 FMAs and took two CTA barriers a
// pivot: 456 us for 8,163 banks, against 50 us of FP64 FMAs.)  Scaling by the reciprocal
// instead of dividing changes the last bit of some FP64 entries against the reference's
// per-element division; k_mas_invert scales the same way, and the CPU oracle
// (ORC_ORDER_FIXED) restates it.
constexpr int INV_WARPS = 4;

__global__ void __launch_bounds__(32 * INV_WARPS, 2) k_mas_invert16(const double* __restrict__ mat, float* inv, int nbanks)
{
    constexpr int B = 16, TR = 12, TC = 6;
    const int NS = nsym(B);
    __shared__ double rowj[INV_WARPS][2][3 * B], colj[INV_WARPS][2][3 * B];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bk = blockIdx.x * INV_WARPS + w;
    if(bk >= nbanks) return;
    const int bi = lane >> 3, bj = lane & 7;
    const double* Mb = mat + (size_t)bk * NS * 9;
    double a[TR][TC];
#pragma unroll
    for(int p = 0; p < TR / 3; p++)
#pragma unroll
        for(int q = 0; q < TC / 3; q++)
        {
            const int rb = 4 * bi + p, cb = 2 * bj + q;
            const bool up = cb >= rb;  // else the mirror block, transposed
            const double* H = Mb + upper_index(B, min(rb, cb), max(rb, cb)) * 9;  // column-major
#pragma unroll
            for(int r = 0; r < 3; r++)
#pragma unroll
                for(int cc = 0; cc < 3; cc++)
                {
                    double v = up ? H[cc * 3 + r] : H[r * 3 + cc];
                    if(r == cc && rb == cb && v == 0.0) v = 1.0;
                    a[3 * p + r][3 * q + cc] = v;
                }
        }
    for(int pb = 0; pb < 4; pb++)
    {
#pragma unroll
        for(int pr = 0; pr < TR; pr++)
        {
            const int j = TR * pb + pr;
            double* cj = colj[w][pr & 1];
            double* rj = rowj[w][pr & 1];
            const bool my_col = bj == 2 * pb + pr / TC, my_row = bi == pb;
            // 1: the old column j
            if(my_col)
            {
#pragma unroll
                for(int k = 0; k < TR; k++) cj[TR * bi + k] = a[k][pr % TC];
            }
            __syncwarp();
            // 2: row j after the column replacement (e_j) and the scaling by the pivot's reciprocal
            if(my_row)
            {
                const double rinv = 1.0 / cj[j];
#pragma unroll
                for(int cc = 0; cc < TC; cc++)
                {
                    const double x = my_col && cc == pr % TC ? 1.0 : a[pr][cc];
                    a[pr][cc] = __dmul_rn(x, rinv);
                    rj[TC * bj + cc] = a[pr][cc];
                }
            }
            __syncwarp();
            // 3: every other row (column j replaced by e_j)
            double rv[TC];
#pragma unroll
            for(int cc = 0; cc < TC; cc++) rv[cc] = rj[TC * bj + cc];
#pragma unroll
            for(int k = 0; k < TR; k++)
            {
                if(k == pr && my_row) continue;
                const double cm = cj[TR * bi + k];
#pragma unroll
                for(int cc = 0; cc < TC; cc++)
                {
                    const double old = my_col && cc == pr % TC ? 0.0 : a[k][cc];
                    a[k][cc] = fma(-cm, rv[cc], old);
                }
            }
            // the next pivot writes the other buffers; this pivot's are reused two pivots later,
            // after two more barriers
        }
    }
    float* P = inv + (size_t)bk * NS * 9;
#pragma unroll
    for(int p = 0; p < TR / 3; p++)
#pragma unroll
        for(int q = 0; q < TC / 3; q++)
        {
            const int rb = 4 * bi + p, cb = 2 * bj + q;
            if(cb < rb) continue;
            float* D = P + upper_index(B, rb, cb) * 9;
#pragma unroll
            for(int r = 0; r < 3; r++)
#pragma unroll
                for(int cc = 0; cc < 3; cc++)
                {
                    // lower triangle of a diagonal 3x3 block mirrored from the upper one
                    D[cc * 3 + r] = (float)(rb == cb && r > cc ? a[3 * p + cc][3 * q + r] : a[3 * p + r][3 * q + cc]);
                }
        }
}

// ---------------------------------------------------------------------------------------
// apply
// ---------------------------------------------------------------------------------------
// Level 0 + level 1 of __buildMultiLevelR_optimized_new (MASPreconditioner.cu:729-847):
// slot values (FP32) and, for each level-0 component, the sum of its members in lane order.
template <int B>
__global__ void k_mas_restrict0(const double* __restrict__ r, const int* __restrict__ part_map,
                                const unsigned* __restrict__ fine_mask, const int* __restrict__ going_next, float* R, int M,
                                const int* done)
{
    if(done && *done) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = s % B;
    const int v = s < M ? part_map[s] : -1;
    float r0 = 0.f, r1 = 0.f, r2 = 0.f;
    unsigned msk = 0;
    if(v >= 0)
    {
        r0 = (float)r[3 * v];
        r1 = (float)r[3 * v + 1];
        r2 = (float)r[3 * v + 2];
        msk = fine_mask[v];
    }
    if(s < M) st4(R + 4 * (size_t)s, r0, r1, r2);
    float a0 = 0.f, a1 = 0.f, a2 = 0.f;
#pragma unroll
    for(int b = 0; b < B; b++)
    {
        const float x0 = group_shfl<B>(r0, b);
        const float x1 = group_shfl<B>(r1, b);
        const float x2 = group_shfl<B>(r2, b);
        if(msk & (1u << b))
        {
            a0 += x0;
            a1 += x1;
            a2 += x2;
        }
    }
    if(v >= 0 && __popc(msk & lanemask_lt(lane)) == 0)
    {
        const int g = going_next[v];
        st4(R + 4 * (size_t)g, a0, a1, a2);
    }
}

// Levels l -> l+1 (l >= 1): each component of a level-l bank sums its nodes in lane order.
template <int B>
__global__ void k_mas_restrict_lx(float* R, const unsigned* __restrict__ closed, const int* __restrict__ going_next,
                                  int number, int begin, const int* done)
{
    if(done && *done) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = i % B;
    const bool valid = i < number;
    float r0 = 0.f, r1 = 0.f, r2 = 0.f;
    unsigned msk = 0;
    if(valid)
    {
        ld4(R + 4 * (size_t)(begin + i), r0, r1, r2);
        msk = closed[begin + i];
    }
    float a0 = 0.f, a1 = 0.f, a2 = 0.f;
#pragma unroll
    for(int b = 0; b < B; b++)
    {
        const float x0 = group_shfl<B>(r0, b);
        const float x1 = group_shfl<B>(r1, b);
        const float x2 = group_shfl<B>(r2, b);
        if(msk & (1u << b))
        {
            a0 += x0;
            a1 += x1;
            a2 += x2;
        }
    }
    if(valid && __popc(msk & lanemask_lt(lane)) == 0)
    {
        const int g = going_next[begin + i];
        st4(R + 4 * (size_t)g, a0, a1, a2);
    }
}

// _schwarzLocalXSym6 (MASPreconditioner.cu:957-1027): z_b = P_b r_b for every bank of every
// level, with the row arithmetic of bank_dev.cuh (the PCG loop's phase D gives the same bits).
// 16-banks: one warp per bank (4 per CTA), lane (a, h) forms half h of block row a; the
// packed inverse (4,896 B) and the 16 residual slots are staged per warp with 16-byte loads.
constexpr int SCHWARZ16_WARPS = 4;

__global__ void __launch_bounds__(SCHWARZ16_WARPS * 32) k_mas_schwarz16(const float* __restrict__ inv,
                                                                        const float* __restrict__ R, float* Z,
                                                                        int nbanks, const int* done)
{
    if(done && *done) return;
    __shared__ __align__(16) float P[SCHWARZ16_WARPS][136 * 9];
    __shared__ float4 rs[SCHWARZ16_WARPS][16];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bk = blockIdx.x * SCHWARZ16_WARPS + w;
    if(bk >= nbanks) return;
    const float4* src = reinterpret_cast<const float4*>(inv + (size_t)bk * 136 * 9);
    float4* dst = reinterpret_cast<float4*>(P[w]);
    for(int t = lane; t < 136 * 9 / 4; t += 32) dst[t] = __ldg(src + t);
    if(lane < 16) rs[w][lane] = *reinterpret_cast<const float4*>(R + 4 * ((size_t)bk * 16 + lane));
    __syncwarp();
    const int a = lane & 15, h = lane >> 4;
    float z0, z1, z2;
    bank16_half(P[w], rs[w], a, h, z0, z1, z2);
    bank16_join(z0, z1, z2);
    if(h == 0) st4(Z + ((size_t)bk * 16 + a) * 4, z0, z1, z2);
}

// 32-banks: one CTA of 1,024 threads per bank, thread (a, c) forms the block product of
// block (a, c) and the 32 lanes of row a sum them with the xor butterfly.
__global__ void __launch_bounds__(1024) k_mas_schwarz32(const float* __restrict__ inv, const float* __restrict__ R,
                                                        float* Z, const int* done)
{
    if(done && *done) return;
    constexpr int B = 32, NS = B * (B + 1) / 2;
    __shared__ __align__(16) float P[NS * 9];
    __shared__ float r[3 * B];
    const int bk = blockIdx.x;
    const float4* src = reinterpret_cast<const float4*>(inv + (size_t)bk * NS * 9);
    float4* dst = reinterpret_cast<float4*>(P);
    for(int t = threadIdx.x; t < NS * 9 / 4; t += B * B) dst[t] = __ldg(src + t);
    if(threadIdx.x < B) ld4(R + 4 * ((size_t)bk * B + threadIdx.x), r[3 * threadIdx.x], r[3 * threadIdx.x + 1], r[3 * threadIdx.x + 2]);
    __syncthreads();
    const int a = threadIdx.x / B, c = threadIdx.x % B;
    const int lo = min(a, c), hi = max(a, c);
    float z0, z1, z2;
    blk_mul3(P + upper_index(B, lo, hi) * 9, c < a, r[3 * c], r[3 * c + 1], r[3 * c + 2], z0, z1, z2);
    warp_butterfly3(z0, z1, z2);
    if(c == 0) st4(Z + ((size_t)bk * B + a) * 4, z0, z1, z2);
}

// __collectFinalZ_new (MASPreconditioner.cu:850-879): Z_v = sum over levels (FP32) -> FP64.
__global__ void k_mas_prolong(const float* __restrict__ Z, const int* __restrict__ real_map,
                              const int* __restrict__ coarse_table, int L, int V, double* z)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if(v >= V) return;
    const int s = real_map[v];
    float c0, c1, c2;
    ld4(Z + 4 * (size_t)s, c0, c1, c2);
    for(int l = 1; l < L; l++)
    {
        const int now = coarse_table[(size_t)v * (L - 1) + l - 1];
        float t0, t1, t2;
        ld4(Z + 4 * (size_t)now, t0, t1, t2);
        c0 += t0;
        c1 += t1;
        c2 += t2;
    }
    z[3 * v] = c0;
    z[3 * v + 1] = c1;
    z[3 * v + 2] = c2;
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
static int num_levels(int n, int B)
{
    int nLevel = 1;
    int levelSz = (n + B - 1) / B * B;
    while(levelSz > B)
    {
        levelSz /= B;
        nLevel++;
        levelSz = (levelSz + B - 1) / B * B;
    }
    nLevel = nLevel + 1;
    return nLevel > kMaxLevels ? kMaxLevels : nLevel;
}

int Solver::mas_init(int V, int node_offset, const uint32_t* ns, const uint32_t* nn, const uint32_t* nl, int nls,
                     const int* pm, int pms, const int* rm)
{
    MasState& m = mas;
    const int B = cfg.bank_size;
    if(V < 1 || pms < V || pms % B != 0 || nls < 0)
    {
        set_error("stg_mas_init: need vert_num >= 1, part_map_size >= vert_num and a multiple of bank_size");
        return STG_ERR_INVALID;
    }
    // host-side validation of the maps (an out-of-range id would be an out-of-bounds access)
    for(int s = 0; s < pms; s++)
        if(pm[s] < -1 || pm[s] >= V)
        {
            set_error("stg_mas_init: part_map entry out of range");
            return STG_ERR_INVALID;
        }
    for(int v = 0; v < V; v++)
        if(rm[v] < 0 || rm[v] >= pms || pm[rm[v]] != v)
        {
            set_error("stg_mas_init: real_map is not the inverse of part_map");
            return STG_ERR_INVALID;
        }
    for(int v = 0; v < V; v++)
        if((long)ns[v] + nn[v] > nls)
        {
            set_error("stg_mas_init: neighbour list overruns neighbor_list_size");
            return STG_ERR_INVALID;
        }
    for(int e = 0; e < nls; e++)
        if(nl[e] >= (uint32_t)V)
        {
            set_error("stg_mas_init: neighbour id out of range");
            return STG_ERR_INVALID;
        }
    m.bank = B;
    m.V = V;
    m.M = pms;
    m.identity = true;
    for(int s = 0; s < pms && m.identity; s++) m.identity = pm[s] == (s < V ? s : -1);
    m.nb0 = pms / B;
    m.node_offset = node_offset;
    m.nlist_size = nls;
    m.L = num_levels(std::max(pms, V), B);
    const int L = m.L;
    cudaStream_t s = stream;
    STG_TRY(m.nstart.resize(V));
    STG_TRY(m.nnum_init.resize(V));
    STG_TRY(m.nnum.resize(V));
    STG_TRY(m.nlist_init.resize(std::max(nls, 1)));
    STG_TRY(m.nlist.resize(std::max(nls, 1)));
    STG_TRY(m.part_map.resize(pms));
    STG_TRY(m.real_map.resize(V));
    STG_TRY(m.fine_mask.resize(V));
    STG_TRY(m.next_mask.resize(2 * (size_t)(V + B)));
    STG_TRY(m.prefix_orig.resize(m.nb0 + 1));
    STG_TRY(m.prefix_sum_orig.resize(m.nb0 + 1));
    STG_TRY(m.next_prefix.resize(V / B + 2));
    STG_TRY(m.next_prefix_sum.resize(V / B + 2));
    STG_TRY(m.coarse_tables.resize((size_t)L * V));
    m.gn_size = pms + L * (V + B);  // >= total clusters: level l >= 1 holds <= V nodes, rounded to B
    STG_TRY(m.going_next.resize(m.gn_size));
    STG_TRY(m.closed.resize(m.gn_size));
    STG_TRY(m.lead.resize(m.gn_size));
    STG_TRY(m.coarse_table.resize((size_t)V * std::max(L - 1, 1)));
    STG_TRY(m.level_size_d.resize(kMaxLevels + 2));
    STG_TRY(m.scratch.resize(kMaxLevels + 2));
    STG_CUDA_TRY(cudaMemcpyAsync(m.nstart.data(), ns, sizeof(unsigned) * V, cudaMemcpyHostToDevice, s));
    STG_CUDA_TRY(cudaMemcpyAsync(m.nnum_init.data(), nn, sizeof(unsigned) * V, cudaMemcpyHostToDevice, s));
    if(nls > 0) STG_CUDA_TRY(cudaMemcpyAsync(m.nlist_init.data(), nl, sizeof(unsigned) * nls, cudaMemcpyHostToDevice, s));
    STG_CUDA_TRY(cudaMemcpyAsync(m.part_map.data(), pm, sizeof(int) * pms, cudaMemcpyHostToDevice, s));
    STG_CUDA_TRY(cudaMemcpyAsync(m.real_map.data(), rm, sizeof(int) * V, cudaMemcpyHostToDevice, s));
    STG_CUDA_TRY(cudaMemsetAsync(m.going_next.data(), 0, sizeof(int) * m.gn_size, s));
    STG_CUDA_TRY(cudaMemsetAsync(m.closed.data(), 0, sizeof(unsigned) * m.gn_size, s));
    STG_CUDA_TRY(cudaMemsetAsync(m.lead.data(), 0, sizeof(int) * m.gn_size, s));
    STG_CUDA_TRY(cudaStreamSynchronize(s));
    m.inited = true;
    m.built = m.assembled = false;
    return 0;
}

// one cluster's launch configuration; false where such clusters do not fit the device
template <int B>
static int build_small_fits(bool* fits)
{
    static thread_local unsigned long long seen = 0;
    static thread_local bool ok[64];
    int dev = 0;
    STG_CUDA_TRY(cudaGetDevice(&dev));
    if(first_on_device(seen))
    {
        cudaLaunchAttribute at = {};
        const cudaLaunchConfig_t cfg = cluster_config(MB_CL, MB_CL, MB_T, 0, nullptr, &at);
        int n = 0;
        STG_CUDA_TRY(cudaFuncSetAttribute(k_mas_build_small<B>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        ok[dev & 63] = cudaOccupancyMaxActiveClusters(&n, k_mas_build_small<B>, &cfg) == cudaSuccess && n > 0;
        cudaGetLastError();
    }
    *fits = ok[dev & 63];
    return 0;
}

// reads the level sizes back and derives the bank counts
static int mas_sizes(Solver& S, int B)
{
    MasState& m = S.mas;
    STG_CUDA_TRY(cudaMemcpyAsync(m.level_size, m.level_size_d.data(), sizeof(int) * 2 * (m.L + 1), cudaMemcpyDeviceToHost,
                                 S.stream));
    STG_CUDA_TRY(cudaStreamSynchronize(S.stream));
    m.total_clusters = m.level_size[2 * m.L + 1];
    m.nbanks = m.total_clusters / B;
    if(m.total_clusters > m.gn_size || m.total_clusters % B != 0)
    {
        set_error("MAS build produced an inconsistent cluster count");
        return STG_ERR_INVALID;
    }
    m.built = true;
    return 0;
}

template <int B>
static int mas_build_t(Solver& S, const int* contacts, int ncp)
{
    MasState& m = S.mas;
    cudaStream_t s = S.stream;
    const int V = m.V, M = m.M, L = m.L;
    int* ls = reinterpret_cast<int*>(m.level_size_d.data());
    bool small = M <= MB_MAX_SLOTS;
    if(small) STG_TRY(build_small_fits<B>(&small));
    if(small)
    {
        MasBuildArgs A{m.part_map.data(), m.real_map.data(), m.nstart.data(), m.nnum_init.data(), m.nlist_init.data(),
                       m.nnum.data(), m.nlist.data(), m.fine_mask.data(), m.prefix_orig.data(), m.coarse_tables.data(),
                       m.going_next.data(), m.closed.data(), m.lead.data(), m.coarse_table.data(), m.next_mask.data(),
                       ls, reinterpret_cast<const int4*>(contacts), ncp, m.node_offset, V, M, L};
        cudaLaunchAttribute at = {};
        const cudaLaunchConfig_t cfg = cluster_config(MB_CL, MB_CL, MB_T, 0, s, &at);
        STG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_mas_build_small<B>, A));
        S.launches++;
        return mas_sizes(S, B);
    }
    STG_CUDA_TRY(cudaMemcpyAsync(m.nlist.data(), m.nlist_init.data(), sizeof(unsigned) * std::max(m.nlist_size, 1),
                                 cudaMemcpyDeviceToDevice, s));
    STG_CUDA_TRY(cudaMemcpyAsync(m.nnum.data(), m.nnum_init.data(), sizeof(unsigned) * V, cudaMemcpyDeviceToDevice, s));
    STG_CUDA_TRY(cudaMemsetAsync(ls, 0, sizeof(int2) * (kMaxLevels + 2), s));
    const int gM = div_up(M, 256), gV = div_up(V, 256);
    const int4* pairs = reinterpret_cast<const int4*>(contacts);
    k_mas_l0_mask<B><<<gM, 256, 0, s>>>(m.part_map.data(), m.real_map.data(), m.nstart.data(), m.nnum.data(),
                                        m.nlist.data(), m.fine_mask.data(), M);
    STG_LAUNCH_CHECK();
    if(ncp > 0)
    {
        k_mas_contacts<B><<<div_up(ncp, 256), 256, 0, s>>>(m.fine_mask.data(), nullptr, m.real_map.data(), pairs, ncp,
                                                          m.node_offset, V);
        STG_LAUNCH_CHECK();
        S.launches++;
    }
    k_mas_l0_closure<B><<<gM, 256, 0, s>>>(m.part_map.data(), m.fine_mask.data(), m.prefix_orig.data(), M);
    STG_LAUNCH_CHECK();
    STG_TRY(scan_exclusive(m.prefix_orig.data(), m.prefix_sum_orig.data(), nullptr, m.nb0, m.nb0, m.scratch.data(), s));
    k_set_level1<<<1, 1, 0, s>>>(ls, m.scratch.data(), M);
    STG_LAUNCH_CHECK();
    k_mas_l1_assign<B><<<gM, 256, 0, s>>>(m.part_map.data(), m.fine_mask.data(), m.prefix_sum_orig.data(),
                                          m.coarse_tables.data(), m.going_next.data(), M);
    STG_LAUNCH_CHECK();
    S.launches += 5;
    const int gN = div_up(V + B, 256);
    for(int level = 1; level < L; level++)
    {
        const int* prev = m.coarse_tables.data() + (size_t)(level - 1) * V;
        STG_CUDA_TRY(cudaMemsetAsync(m.next_mask.data(), 0, sizeof(unsigned) * (V + B), s));
        k_mas_lx_mask<B><<<gM, 256, 0, s>>>(m.part_map.data(), m.nstart.data(), m.nnum.data(), m.nlist.data(), prev,
                                            m.next_mask.data(), M);
        STG_LAUNCH_CHECK();
        if(ncp > 0)
        {
            k_mas_contacts<B><<<div_up(ncp, 256), 256, 0, s>>>(m.next_mask.data(), prev, m.real_map.data(), pairs, ncp,
                                                              m.node_offset, V);
            STG_LAUNCH_CHECK();
            S.launches++;
        }
        k_mas_lx_closure<B><<<gN, 256, 0, s>>>(m.next_mask.data(), m.closed.data(), m.next_prefix.data(), ls, level);
        STG_LAUNCH_CHECK();
        // n = ceil(ls[2*level] / B) banks
        STG_TRY(scan_exclusive(m.next_prefix.data(), m.next_prefix_sum.data(), ls + 2 * level, -B, V / B + 1,
                               ls + 2 * (level + 1), s));
        k_mas_lx_assign<B><<<gN, 256, 0, s>>>(m.next_mask.data(), m.next_prefix_sum.data(), m.going_next.data(),
                                              m.lead.data(), ls, level);
        STG_LAUNCH_CHECK();
        k_mas_compute_next<<<gV, 256, 0, s>>>(m.coarse_tables.data(), m.next_mask.data(), level, V);
        STG_LAUNCH_CHECK();
        S.launches += 5;
    }
    if(L > 1)
    {
        k_mas_aggregate<<<gV, 256, 0, s>>>(m.going_next.data(), m.coarse_table.data(), L, V);
        STG_LAUNCH_CHECK();
        S.launches++;
    }
    return mas_sizes(S, B);
}

int Solver::mas_build(const int* contacts, int ncp)
{
    if(!mas.inited)
    {
        set_error("MAS not initialised (stg_mas_init)");
        return STG_ERR_NOT_READY;
    }
    if(cfg.bank_size == 32) return mas_build_t<32>(*this, contacts, ncp);
    return mas_build_t<16>(*this, contacts, ncp);
}

int convert_into(Solver& S, ConvertScratch& cv, int count, const int* rows, const int* cols, const double* blocks,
                 int nrows, bool skip_negative, DBuf<int>& out_rows, DBuf<int>& out_cols, DBuf<double>& out_blocks,
                 DBuf<int>& row_ptr, int* unique, bool fuse = false);

template <int B>
static int mas_assemble_t(Solver& S, int offset)
{
    MasState& m = S.mas;
    cudaStream_t s = S.stream;
    const int NS = nsym(B);
    const size_t nvals = (size_t)m.nbanks * NS * 9;
    STG_TRY(m.mat.resize(nvals));
    STG_TRY(m.inv.resize(nvals));
    // R, Z: one {x y z 0} float4 slot per node of every level
    STG_TRY(m.R.resize((size_t)m.total_clusters * 4));
    STG_TRY(m.Z.resize((size_t)m.total_clusters * 4));
    // the fine convert of stg_solve_linear_system already stored level 0 and emitted the
    // level-1 triplets (ConvFuse) when it ran for this offset
    const bool fused = m.l0_fused && m.l0_offset == offset;
    m.l0_fused = false;
    if(!fused) STG_CUDA_TRY(cudaMemsetAsync(m.mat.data(), 0, nvals * sizeof(double), s));
    STG_CUDA_TRY(cudaMemsetAsync(m.R.data(), 0, sizeof(float) * 4 * m.total_clusters, s));
    const int nnzb = S.bcoo.nnzb;
    const int g = std::max(1, std::min(div_up(nnzb, 256), kSMs * 16));
    if(nnzb > 0 && !fused)
    {
        k_mas_store_l0<B><<<g, 256, 0, s>>>(S.bcoo.R(), S.bcoo.C(), S.bcoo.B(), nnzb, offset, m.V, m.real_map.data(),
                                            m.mat.data());
        STG_LAUNCH_CHECK();
        S.launches++;
    }
    bool learned_captured = false;
    S.learned.graph_ready = false;
    if(m.L > 1 && nnzb > 0)
    {
        // level 1 from the fine matrix
        if(!fused)
        {
            STG_TRY(m.tr_rows.resize(nnzb));
            STG_TRY(m.tr_cols.resize(nnzb));
            STG_TRY(m.tr_blocks.resize((size_t)nnzb * 9));
            k_mas_agg_l0<B><<<g, 256, 0, s>>>(S.bcoo.R(), S.bcoo.C(), S.bcoo.B(), nnzb, offset, m.V,
                                              m.real_map.data(), m.coarse_tables.data(), m.tr_rows.data(),
                                              m.tr_cols.data(), m.tr_blocks.data());
            STG_LAUNCH_CHECK();
            S.launches++;
        }
        // a level with few enough triplets and nodes (20-bit keys) ends the levels in one launch;
        // the learned level's operator is read back level by level
        auto chain = [&](int level, int count) -> bool {
            return count <= CHAIN_CAP && m.level_size[2 * level] < (1 << 20) && S.learned.level == 0;
        };
        auto run_chain = [&](int level, int count) -> int {
            STG_TRY(m.ga_rows.resize(std::max<size_t>(m.ga_rows.size, count)));
            STG_TRY(m.ga_cols.resize(std::max<size_t>(m.ga_cols.size, count)));
            STG_TRY(m.ga_blocks.resize(std::max<size_t>(m.ga_blocks.size, 9 * (size_t)count)));
            ChainArgs A{m.tr_rows.data(), m.tr_cols.data(), m.tr_blocks.data(), count, level, m.L, {}, {}, m.going_next.data(),
                        m.ga_rows.data(), m.ga_cols.data(), m.ga_blocks.data(), m.mat.data()};
            for(int l = 0; l <= m.L; l++) A.begin[l] = m.level_size[2 * l + 1], A.nodes[l] = m.level_size[2 * l];
            static thread_local unsigned long long seen = 0;
            if(first_on_device(seen))
                STG_CUDA_TRY(cudaFuncSetAttribute(k_mas_chain<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, CHAIN_SMEM));
            k_mas_chain<B><<<1, CHAIN_T, CHAIN_SMEM, s>>>(A);
            STG_LAUNCH_CHECK();
            S.launches++;
            return 0;
        };
        int nnz = 0;
        const bool all = chain(1, nnzb);
        if(all) STG_TRY(run_chain(1, nnzb));
        if(!all) STG_TRY(convert_into(S, m.gcv, nnzb, m.tr_rows.data(), m.tr_cols.data(), m.tr_blocks.data(), m.level_size[2],
                             true, m.ga_rows, m.ga_cols, m.ga_blocks, m.g_rowptr, &nnz));
        for(int level = 1; !all; level++)
        {
            const int begin = m.level_size[2 * level + 1];
            if(level == S.learned.level && nnz > 0)
            {
                // the learned level's Galerkin operator, kept for its graph (built below)
                LearnedState& Ls = S.learned;
                STG_TRY(Ls.urow.resize(nnz));
                STG_TRY(Ls.ucol.resize(nnz));
                STG_TRY(Ls.ublk.resize(9 * (size_t)nnz));
                STG_CUDA_TRY(cudaMemcpyAsync(Ls.urow.data(), m.ga_rows.data(), sizeof(int) * nnz, cudaMemcpyDeviceToDevice, s));
                STG_CUDA_TRY(cudaMemcpyAsync(Ls.ucol.data(), m.ga_cols.data(), sizeof(int) * nnz, cudaMemcpyDeviceToDevice, s));
                STG_CUDA_TRY(cudaMemcpyAsync(Ls.ublk.data(), m.ga_blocks.data(), sizeof(double) * 9 * nnz,
                                             cudaMemcpyDeviceToDevice, s));
                Ls.unnz = nnz;
                learned_captured = true;
            }
            if(nnz > 0)
            {
                k_mas_extract<B><<<std::max(1, std::min(div_up(nnz, 256), kSMs * 16)), 256, 0, s>>>(
                    m.ga_rows.data(), m.ga_cols.data(), m.ga_blocks.data(), nnz, begin, m.mat.data());
                STG_LAUNCH_CHECK();
                S.launches++;
            }
            if(level + 1 >= m.L || nnz == 0) break;
            const int begin_next = m.level_size[2 * (level + 1) + 1];
            STG_TRY(m.tr_rows.resize(nnz));
            STG_TRY(m.tr_cols.resize(nnz));
            STG_TRY(m.tr_blocks.resize((size_t)nnz * 9));
            k_mas_agg_lx<<<std::max(1, std::min(div_up(nnz, 256), kSMs * 16)), 256, 0, s>>>(
                m.ga_rows.data(), m.ga_cols.data(), m.ga_blocks.data(), nnz, m.going_next.data(), begin, begin_next,
                m.tr_rows.data(), m.tr_cols.data(), m.tr_blocks.data());
            STG_LAUNCH_CHECK();
            S.launches++;
            if(chain(level + 1, nnz))
            {
                STG_TRY(run_chain(level + 1, nnz));
                break;
            }
            int nnz2 = 0;
            STG_TRY(convert_into(S, m.gcv, nnz, m.tr_rows.data(), m.tr_cols.data(), m.tr_blocks.data(),
                                 m.level_size[2 * (level + 1)], false, m.gb_rows, m.gb_cols, m.gb_blocks, m.g_rowptr,
                                 &nnz2));
            std::swap(m.ga_rows.ptr, m.gb_rows.ptr);
            std::swap(m.ga_rows.cap, m.gb_rows.cap);
            std::swap(m.ga_cols.ptr, m.gb_cols.ptr);
            std::swap(m.ga_cols.cap, m.gb_cols.cap);
            std::swap(m.ga_blocks.ptr, m.gb_blocks.ptr);
            std::swap(m.ga_blocks.cap, m.gb_blocks.cap);
            nnz = nnz2;
        }
    }
    if(B == 16)
    {
        k_mas_invert16<<<div_up(m.nbanks, INV_WARPS), 32 * INV_WARPS, 0, s>>>(m.mat.data(), m.inv.data(), m.nbanks);
        STG_LAUNCH_CHECK();
    }
    else
    {
        const size_t smem = sizeof(double) * (3 * B * 3 * B + 3 * B);
        if(smem > 48 * 1024)
            STG_CUDA_TRY(cudaFuncSetAttribute(k_mas_invert<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_mas_invert<B><<<m.nbanks, 3 * B, smem, s>>>(m.mat.data(), m.inv.data(), m.nbanks);
        STG_LAUNCH_CHECK();
    }
    S.launches++;
    if(learned_captured)
    {
        LearnedState& Ls = S.learned;
        const int n = m.level_size[2 * Ls.level];
        Ls.begin = m.level_size[2 * Ls.level + 1];
        STG_TRY(net_build_graph(s, Ls.graph, n, Ls.unnz, Ls.urow.data(), Ls.ucol.data(), Ls.ublk.data(), &S.launches));
        Ls.graph.level = Ls.level;
        const size_t bytes = net_scratch_bytes(n, 1);
        STG_TRY(Ls.scratch.resize(bytes));
        STG_TRY(net_carve(Ls.scratch.data(), bytes, n, 1, Ls.buf));
        Ls.graph_ready = true;
    }
    m.assembled = true;
    return 0;
}

int Solver::mas_assemble(int offset)
{
    if(!mas.built)
    {
        set_error("MAS hierarchy not built");
        return STG_ERR_NOT_READY;
    }
    if(cfg.bank_size == 32) return mas_assemble_t<32>(*this, offset);
    return mas_assemble_t<16>(*this, offset);
}

template <int B>
int mas_restrict_solve_t(Solver& S, const double* r, const int* done)
{
    MasState& m = S.mas;
    cudaStream_t s = S.stream;
    k_mas_restrict0<B><<<div_up(m.M, 256), 256, 0, s>>>(r, m.part_map.data(), m.fine_mask.data(), m.going_next.data(),
                                                        m.R.data(), m.M, done);
    STG_LAUNCH_CHECK();
    S.launches++;
    for(int level = 1; level < m.L - 1; level++)
    {
        const int number = m.level_size[2 * level], begin = m.level_size[2 * level + 1];
        if(number < 1) continue;
        k_mas_restrict_lx<B><<<div_up((number + B - 1) / B * B, 256), 256, 0, s>>>(m.R.data(), m.closed.data(),
                                                                                   m.going_next.data(), number, begin, done);
        STG_LAUNCH_CHECK();
        S.launches++;
    }
    if(B == 16)
        k_mas_schwarz16<<<div_up(m.nbanks, SCHWARZ16_WARPS), SCHWARZ16_WARPS * 32, 0, s>>>(m.inv.data(), m.R.data(),
                                                                                          m.Z.data(), m.nbanks, done);
    else
        k_mas_schwarz32<<<m.nbanks, 1024, 0, s>>>(m.inv.data(), m.R.data(), m.Z.data(), done);
    STG_LAUNCH_CHECK();
    S.launches++;
    return 0;
}

// restriction + bank solves; kernels return immediately when *done != 0 (done may be null)
int mas_restrict_solve_guarded(Solver& S, const double* r, const int* done)
{
    if(S.cfg.bank_size == 32) return mas_restrict_solve_t<32>(S, r, done);
    return mas_restrict_solve_t<16>(S, r, done);
}

int mas_restrict_solve(Solver& S, const double* r) { return mas_restrict_solve_guarded(S, r, nullptr); }

int Solver::mas_apply(const double* r, double* z)
{
    if(!mas.assembled)
    {
        set_error("MAS not assembled");
        return STG_ERR_NOT_READY;
    }
    STG_TRY(mas_restrict_solve(*this, r));
    k_mas_prolong<<<div_up(mas.V, 256), 256, 0, stream>>>(mas.Z.data(), mas.real_map.data(), mas.coarse_table.data(),
                                                          mas.L, mas.V, z);
    STG_LAUNCH_CHECK();
    launches++;
    return 0;
}

}  // namespace stg
