// The whole PCG loop of a small system in one cooperative launch.
//
// Below ~30,000 rows an iteration of the launch-per-step loop (b2s_pcg.cu) is
// a chain of five launches that each do a microsecond of work, and the host
// looks at the scalars every few iterations. Here the grid stays resident: a
// thread owns one row of x, r, p and z in registers for the whole solve, a
// warp owns the two MAS banks of its 32 rows and keeps their inverses in
// shared memory, and the steps are separated by grid barriers (three per
// iteration with block Jacobi, five with the MAS). Only p (gathered by the
// SpMV), Ap (its reductions) and the coarse levels' sums and Z go through L2.
// Same arithmetic per entry, stop rules and scalars as the launch-per-step
// loop; the sums add per-block partials in a fixed order.
//
// What crosses blocks inside the launch is read past L1 (ld.cg), after a
// barrier whose arrival releases and whose wait acquires at device scope. The
// bulk copies (TMA) only read inverses, which the launch never writes. Every
// wait is bounded: a barrier or a copy that runs out sets the error flag and
// the block leaves, its copies in flight waited for; the others' barriers then
// run out too. The scalars stay as they were, and the host, which reads the
// flag with them after every launch, ends the call with an error.
#include "b2s_mas_apply.cuh"
#include "b2s_pcg.cuh"

#include <algorithm>

namespace b2s
{

namespace
{
constexpr int SM_THREADS = 256;
constexpr int SM_WARPS   = SM_THREADS / 32;
constexpr int SM_CTAS    = 2;  // per SM (128 registers a thread)
constexpr int SM_COARSE  = 2;  // stages of the level-1 warp and of the level-2 warp
constexpr int SM_L1_WARP = 6, SM_L2_WARP = 7;
constexpr unsigned SM_SPINS = 1u << 22;  // polls of a barrier (seconds; an iteration is ~20 us)

template <typename VT>
struct SmallArgs
{
    int32_t        n;  // rows
    int            kind;
    int64_t        S;
    const int32_t* rows;
    const int32_t* cols;
    const VT*      vals;  // planes
    double*        x;
    VT*            r;
    VT*            p;
    VT*            Ap;
    PcgScalars*    sc;
    double*        partials;  // [3][grid]
    unsigned*      bar;       // zero at launch
    MasView        mv;
    const double*  dinv;
    ApplyArgs      A;
    const uint16_t* comp_mask;  // of the slots
    const int32_t*  new_local;
    const int4*     part_dst;
    double*         part;
    long long      iterations;
    unsigned       polls;  // of a barrier, before it gives up
};

// grid barrier: false when it runs out, or when a warp of this block has given
// up (*s_dead: the block does not arrive)
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned& epoch, unsigned polls, int* err,
                                             const int* s_dead)
{
    __shared__ int s_ok;
    epoch += gridDim.x;
    __syncthreads();
    if(threadIdx.x == 0)
    {
        // arrive: releases the block's writes (ordered before by the block barrier)
        const bool dead = *s_dead != 0;
        if(!dead)
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        int ok = 0;
        for(unsigned i = 0; i < polls && !dead; ++i)
        {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if((int)(v - epoch) >= 0)
            {
                ok = 1;
                break;
            }
        }
        if(!ok)
            atomicOr(err, DERR_TMA_TIMEOUT);
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// this block's sum of v -> partials[blockIdx]
__device__ __forceinline__ void block_partial(double v, double* partials, double* s_red)
{
#pragma unroll
    for(int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    if((threadIdx.x & 31) == 0)
        s_red[threadIdx.x >> 5] = v;
    __syncthreads();
    if(threadIdx.x == 0)
    {
        double t = s_red[0];
#pragma unroll
        for(int w = 1; w < SM_WARPS; ++w)
            t += s_red[w];
        partials[blockIdx.x] = t;
    }
}

// the sum of the blocks' partials, the same in every warp of the grid
__device__ __forceinline__ double sum_partials(const double* partials)
{
    double acc = 0.0;
    for(unsigned b = threadIdx.x & 31; b < gridDim.x; b += 32)
        acc += __ldcg(partials + b);
#pragma unroll
    for(int o = 16; o > 0; o >>= 1)
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

template <typename VT>
__device__ __forceinline__ void load_vec(const VT* p, int64_t i, VT v[3])
{
    if constexpr(sizeof(VT) == 4)
    {
        const float4 q = __ldcg(reinterpret_cast<const float4*>(p) + i);
        v[0] = q.x, v[1] = q.y, v[2] = q.z;
    }
    else
#pragma unroll
        for(int c = 0; c < 3; ++c)
            v[c] = __ldcg(p + 3 * i + c);
}
__device__ __forceinline__ void store_vec(float* p, int64_t i, const float v[3])
{
    reinterpret_cast<float4*>(p)[i] = make_float4(v[0], v[1], v[2], 0.0f);
}
__device__ __forceinline__ void store_vec(double* p, int64_t i, const double v[3])
{
#pragma unroll
    for(int c = 0; c < 3; ++c)
        p[3 * i + c] = v[c];
}
__device__ __forceinline__ void red_vec(float* p, int64_t i, const float v[3])
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + 4 * i), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(0.0f)
                 : "memory");
}
__device__ __forceinline__ void red_vec(double* p, int64_t i, const double v[3])
{
#pragma unroll
    for(int c = 0; c < 3; ++c)
        asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p + 3 * i + c), "d"(v[c]) : "memory");
}

// Ap += A p over this thread's blocks (2 consecutive ones at a time), returns
// its part of p.Ap
template <typename VT>
__device__ __forceinline__ double small_spmv(const SmallArgs<VT>& a)
{
    constexpr int BPT = 2;
    double        dot = 0.0;
    const int64_t n_chunks = a.S / BPT;
    for(int64_t c = (int64_t)blockIdx.x * SM_THREADS + threadIdx.x; c < n_chunks;
        c += (int64_t)gridDim.x * SM_THREADS)
    {
        const int64_t e0 = c * BPT;
        const int2    r2 = __ldg(reinterpret_cast<const int2*>(a.rows + e0));
        const int2    c2 = __ldg(reinterpret_cast<const int2*>(a.cols + e0));
        const int32_t rr[2] = {r2.x, r2.y}, cc[2] = {c2.x, c2.y};
        VT            b[9][BPT];
#pragma unroll
        for(int q = 0; q < 9; ++q)
        {
            if constexpr(sizeof(VT) == 4)
            {
                const float2 v = __ldg(reinterpret_cast<const float2*>(a.vals + (int64_t)q * a.S + e0));
                b[q][0] = v.x, b[q][1] = v.y;
            }
            else
            {
                const double2 v = __ldg(reinterpret_cast<const double2*>(a.vals + (int64_t)q * a.S + e0));
                b[q][0] = v.x, b[q][1] = v.y;
            }
        }
        int32_t cur = -1;
        VT      s[3] = {0, 0, 0}, xi[3] = {0, 0, 0};
#pragma unroll
        for(int k = 0; k < BPT; ++k)
        {
            if(rr[k] < 0)
                break;  // padding: only at the end of the stream
            VT xj[3];
            load_vec(a.p, cc[k], xj);
            if(rr[k] != cur)
            {
                if(cur >= 0)
                    red_vec(a.Ap, cur, s);
                cur = rr[k];
                s[0] = s[1] = s[2] = 0;
                load_vec(a.p, cur, xi);
            }
            // column-major: B(p,q) = b[q*3 + p]
            VT y[3];
#pragma unroll
            for(int i = 0; i < 3; ++i)
            {
                y[i] = b[i][k] * xj[0] + b[3 + i][k] * xj[1] + b[6 + i][k] * xj[2];
                s[i] += y[i];
            }
            const bool   off = cur != cc[k];
            const double d   = (double)xi[0] * (double)y[0] + (double)xi[1] * (double)y[1] + (double)xi[2] * (double)y[2];
            dot += off ? 2.0 * d : d;
            if(off)
            {
                VT t[3];
#pragma unroll
                for(int j = 0; j < 3; ++j)
                    t[j] = b[3 * j][k] * xi[0] + b[3 * j + 1][k] * xi[1] + b[3 * j + 2][k] * xi[2];
                red_vec(a.Ap, cc[k], t);
            }
        }
        if(cur >= 0)
            red_vec(a.Ap, cur, s);
    }
    return dot;
}

// the coarse value of level-1 node n1 with ancestors an: Z_1 + Z_2[..] + ...
__device__ __forceinline__ void coarse_value(const MasView& mv, int n1, int4 an, float w[3])
{
    const int  up[4] = {an.x, an.y, an.z, an.w};
#pragma unroll
    for(int c = 0; c < 3; ++c)
        w[c] = __ldcg(mv.Z + 3 * (int64_t)n1 + c);
#pragma unroll
    for(int k = 0; k < 4; ++k)
        if(up[k] >= 0)
#pragma unroll
            for(int c = 0; c < 3; ++c)
                w[c] += __ldcg(mv.Z + 3 * (int64_t)up[k] + c);
}

// VT double: FP64 vectors, FP32 inverses; float: padded FP32 vectors, BF16
// inverses. MAS: rows in PCG order.
template <typename VT, bool MAS>
__global__ void __launch_bounds__(SM_THREADS, SM_CTAS) k_pcg_small(const __grid_constant__ SmallArgs<VT> a)
{
    constexpr bool     BF = sizeof(VT) == 4;
    constexpr uint32_t SB = stage_bytes<BF>();
    constexpr uint32_t CB = BF ? INV16_BYTES : INV_BYTES;
    extern __shared__ __align__(128) unsigned char s_dyn[];  // MAS: [2 per warp][SB], level 1 [2][SB], level 2 [2][SB]
    __shared__ uint64_t s_bar[SM_WARPS + 2 * SM_COARSE];
    __shared__ double   s_red[2][SM_WARPS];
    __shared__ int      s_dead;  // a warp of this block gave up waiting
    __shared__ float    s_z[MAS ? SM_WARPS : 1][2 * BANK * 3];
    __shared__ float    s_rr[MAS ? SM_THREADS : 1][3], s_lead[MAS ? SM_THREADS : 1][3];
    __shared__ int4     s_dst[MAS ? SM_THREADS : 1];
    __shared__ int      s_n[SM_WARPS];
    const int  lane = threadIdx.x & 31, w = threadIdx.x >> 5, sub = lane & 15;
    const int  i = blockIdx.x * SM_THREADS + threadIdx.x;  // this thread's row
    const bool live = i < a.n, in_bank = MAS && i < a.mv.slots;
    const int  bank0 = (blockIdx.x * SM_WARPS + w) * 2;  // the warp's banks: bank0, bank0 + 1
    const int  n0 = MAS ? a.mv.slots / BANK : 0;
    unsigned   epoch = 0;
    int        u1 = 0, u2 = 0;  // copies run through the level-1 / level-2 stages
    uint32_t   cm = 0;
    int        nl = 0, n1 = -1;
    int4       an = make_int4(-1, -1, -1, -1), to = an;
    bool       stiff[2] = {false, false};
    unsigned char* own = s_dyn + (size_t)2 * w * SB;
    bool           underway = false;  // level-1 warp: its first copy of the iteration is not waited for yet
    if(threadIdx.x == 0)
        s_dead = 0;
    // every block leaves the loop through here when a barrier runs out
    auto barrier = [&]() -> bool
    {
        const bool ok = grid_barrier(a.bar, epoch, a.polls, a.A.err, &s_dead);
        if(MAS && !ok && underway)
            mbar_wait(&s_bar[SM_WARPS + u1 % SM_COARSE], (uint32_t)((u1 / SM_COARSE) & 1), nullptr, 0);
        return ok;
    };
    if constexpr(MAS)
    {
        if(threadIdx.x < SM_WARPS + 2 * SM_COARSE)
        {
            mbar_init(&s_bar[threadIdx.x], 1);
            mbar_fence_init();
        }
        __syncthreads();
        if(lane == 0)
        {
            // the warp's inverses, for the whole solve
            const int nb = min(2, max(0, n0 - bank0));
            if(nb > 0)
            {
                mbar_arrive_expect_tx(&s_bar[w], nb * CB);
                for(int k = 0; k < nb; ++k)
                    bulk_copy_g2s(own + k * SB, a.A.inv + (size_t)(bank0 + k) * CB, CB, &s_bar[w]);
            }
        }
        __syncthreads();
        const bool here = bank0 >= n0 || mbar_wait(&s_bar[w], 0, a.A.err, DERR_TMA_TIMEOUT);
        if(!here)  // once more, for the copy to end before the block does
            mbar_wait(&s_bar[w], 0, nullptr, 0);
        if(!__syncthreads_and(here))
            return;  // the others' first barrier runs out
        if(a.A.stiff)
            for(int k = 0; k < 2; ++k)
                stiff[k] = bank0 + k < n0 && a.A.stiff[bank0 + k] != 0;
        if(in_bank)
        {
            if(a.mv.T > 0)
            {
                cm = a.comp_mask[i];
                nl = a.new_local[i];
                n1 = a.mv.slot_node1[i];
                if(n1 >= 0)
                {
                    an = a.mv.anc[n1 - a.mv.begin1];
                    to = a.part_dst[n1 - a.mv.begin1];
                }
            }
        }
    }
    int2 be2 = make_int2(0, 0);  // level-2 warp: the entries of its first bank
    if constexpr(MAS)
        if(w == SM_L2_WARP && (int)(gridDim.x - 1 - blockIdx.x) < a.A.n2)
            be2 = bank_entries(a.A, (int64_t)a.A.g2 + (gridDim.x - 1 - blockIdx.x), lane);
    VT     r[3] = {0, 0, 0}, p[3] = {0, 0, 0}, z[3];
    double x[3] = {0, 0, 0};
    if(live)
    {
        load_vec(a.r, i, r);
        load_vec(a.p, i, p);
        load_vec(a.x, i, x);
    }
    // the matrix's row (-1: padding slot); a body's rows may lie anywhere in PCG order
    const int  row = (MAS && live) ? a.mv.row_of[i] : i;
    const bool body = a.mv.abd_n > 0 && row >= a.mv.abd_off && row < a.mv.abd_off + 4 * a.mv.abd_n;
    PcgScalars sc   = *a.sc;
    double*    part0 = a.partials;
    double*    part1 = part0 + gridDim.x;
    double*    part2 = part1 + gridDim.x;
    for(long long it = 0; it < a.iterations && sc.converged == 0; ++it)
    {
        // the coarse inverses of this iteration, underway during the SpMV
        if constexpr(MAS)
            if(w == SM_L1_WARP && (int)blockIdx.x < a.A.n1)
            {
                const int slot = u1 % SM_COARSE;
                if(lane == 0)
                {
                    fence_proxy_async_smem();
                    issue_bank_copy<BF>(s_dyn + (size_t)(2 * SM_WARPS + slot) * SB, &s_bar[SM_WARPS + slot], a.A,
                                        (int64_t)a.A.g1 + blockIdx.x, false);
                }
                underway = true;
            }
        // Ap = A p, p.Ap
        block_partial(small_spmv<VT>(a), part0, s_red[0]);
        if(!barrier())
            return;
        sc.pAp   = sum_partials(part0);
        sc.alpha = sc.rz / sc.pAp;
        // x += alpha p, r -= alpha Ap, Ap = 0
        if(live)
        {
            VT ap[3];
            load_vec(a.Ap, i, ap);
            const VT zero[3] = {0, 0, 0};
            store_vec(a.Ap, i, zero);
#pragma unroll
            for(int c = 0; c < 3; ++c)
            {
                x[c] += sc.alpha * (double)p[c];
                if constexpr(BF)
                    r[c] = __fmaf_rn(-(float)sc.alpha, ap[c], r[c]);
                else
                    r[c] -= sc.alpha * ap[c];
            }
            if(body)
                store_vec(a.r, i, r);
        }
        // z = P r
        if(a.kind == B2S_PRECOND_NONE)
#pragma unroll
            for(int c = 0; c < 3; ++c)
                z[c] = r[c];
        if constexpr(MAS)
        {
            // the warp's banks: residuals to shared memory, level-1 sums out
            float* s_r = reinterpret_cast<float*>(own + (lane >> 4) * SB + CB);
#pragma unroll
            for(int c = 0; c < 3; ++c)
                s_r[3 * sub + c] = (float)r[c];
#pragma unroll
            for(int c = 0; c < 3; ++c)
                s_rr[threadIdx.x][c] = (float)r[c];
            __syncthreads();
            if(a.mv.T > 0)
                restrict_coarse<SM_THREADS>(s_rr, cm, nl, to, a.mv.begin1, a.A.R, a.part, s_lead, s_dst, s_n);
            // their products, before the barrier that publishes R_1
#pragma unroll
            for(int k = 0; k < 2; ++k)
                if(bank0 + k < n0)
                {
                    unsigned char* st = own + k * SB;
                    float*         Zk = s_z[w] + k * BANK * 3;
                    const float(*rk)[3] = reinterpret_cast<const float(*)[3]>(st + CB);
                    if(BF && !stiff[k])
                        cluster_product_mma(st, &rk[0][0], lane, Zk);
                    else
                    {
                        float        o[3];
                        const float* Mc = stiff[k] ? a.A.inv32 + (size_t)(bank0 + k) * SYM * 9 :
                                                     reinterpret_cast<const float*>(st);
                        cluster_product(Mc, rk, lane, o);
                        if(lane < 16)
                        {
                            Zk[3 * lane]     = o[0];
                            Zk[3 * lane + 1] = o[1];
                            Zk[3 * lane + 2] = o[2];
                        }
                    }
                }
            __syncwarp();
            if(!barrier())
                return;
            if(w == SM_L1_WARP)
            {
                // level-1 banks blockIdx, blockIdx + grid, ...
                for(int b = blockIdx.x; b < a.A.n1; b += gridDim.x)
                {
                    const int      slot  = u1 % SM_COARSE;
                    unsigned char* st    = s_dyn + (size_t)(2 * SM_WARPS + slot) * SB;
                    uint64_t*      bar   = &s_bar[SM_WARPS + slot];
                    const int64_t  g     = (int64_t)a.A.g1 + b;
                    float*         s_r1  = reinterpret_cast<float*>(st + CB);
                    if(b + (int)gridDim.x < a.A.n1 && lane == 0)
                    {
                        const int ns = (u1 + 1) % SM_COARSE;
                        fence_proxy_async_smem();
                        issue_bank_copy<BF>(s_dyn + (size_t)(2 * SM_WARPS + ns) * SB, &s_bar[SM_WARPS + ns], a.A,
                                            g + gridDim.x, false);
                    }
                    for(int e = lane; e < BANK * 3; e += 32)
                        s_r1[e] = __ldcg(a.A.R + g * (BANK * 3) + e);
                    __syncwarp();  // every lane's entries, for the others in bank_product
                    const bool ok = mbar_wait(bar, (uint32_t)((u1 / SM_COARSE) & 1), a.A.err, DERR_TMA_TIMEOUT);
                    underway      = false;
                    if(!__all_sync(0xffffffffu, ok))
                    {
                        // give up, with the next bank's copy drained
                        if(b + (int)gridDim.x < a.A.n1)
                            mbar_wait(&s_bar[SM_WARPS + (u1 + 1) % SM_COARSE],
                                      (uint32_t)(((u1 + 1) / SM_COARSE) & 1), nullptr, 0);
                        s_dead = 1;
                        break;
                    }
                    bank_product<BF>(a.A, st, g, BF && a.A.stiff != nullptr && a.A.stiff[g] != 0, lane);
                    __syncwarp();
                    ++u1;
                }
            }
            else if(w == SM_L2_WARP)
            {
                // the banks of the levels above: from the last block down, so
                // that few blocks have one of these and a level-1 bank
                for(int b = (int)gridDim.x - 1 - (int)blockIdx.x; b < a.A.n2; b += gridDim.x)
                {
                    const int      slot = u2 % SM_COARSE;
                    unsigned char* st   = s_dyn + (size_t)(2 * SM_WARPS + SM_COARSE + slot) * SB;
                    uint64_t*      bar  = &s_bar[SM_WARPS + SM_COARSE + slot];
                    const int64_t  g    = (int64_t)a.A.g2 + b;
                    if(lane == 0)
                    {
                        fence_proxy_async_smem();
                        issue_bank_copy<BF>(st, bar, a.A, g, false);
                    }
                    take_coarse(a.A, g, b < (int)gridDim.x ? be2 : bank_entries(a.A, g, lane),
                                reinterpret_cast<float*>(st + CB), lane);
                    const bool ok = mbar_wait(bar, (uint32_t)((u2 / SM_COARSE) & 1), a.A.err, DERR_TMA_TIMEOUT);
                    if(!__all_sync(0xffffffffu, ok))
                    {
                        s_dead = 1;
                        break;
                    }
                    bank_product<BF>(a.A, st, g, BF && a.A.stiff != nullptr && a.A.stiff[g] != 0, lane);
                    __syncwarp();
                    ++u2;
                }
            }
            if(!barrier())
                return;
            if(in_bank)
            {
                const float* Zk = s_z[w] + (lane >> 4) * BANK * 3 + 3 * sub;
                float        v[3] = {Zk[0], Zk[1], Zk[2]};
                if(n1 >= 0)
                {
                    float c3[3];
                    coarse_value(a.mv, n1, an, c3);
#pragma unroll
                    for(int c = 0; c < 3; ++c)
                        v[c] += c3[c];
                }
#pragma unroll
                for(int c = 0; c < 3; ++c)
                    z[c] = (VT)v[c];
            }
        }
        else if(a.mv.abd_n > 0 && a.kind != B2S_PRECOND_NONE)
        {
            if(!barrier())
                return;  // the bodies' rows read each other's r
        }
        if(a.kind != B2S_PRECOND_NONE && live && !in_bank)
        {
            if(body)
            {
                // row l of body b: z = (H_b^-1)[3l .. 3l+2][0 .. 11] r_b
                const int     b = (row - a.mv.abd_off) >> 2, l = (row - a.mv.abd_off) & 3;
                const double* Hi = a.mv.abd_inv + (size_t)b * 144 + 36 * l;
                double        t[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for(int q = 0; q < 4; ++q)
                {
                    VT rq[3];
                    load_vec(a.r, MAS ? a.mv.pos[row - l + q] : row - l + q, rq);
#pragma unroll
                    for(int c = 0; c < 3; ++c)
#pragma unroll
                        for(int m = 0; m < 3; ++m)
                            t[m] += Hi[12 * m + 3 * q + c] * (double)rq[c];
                }
#pragma unroll
                for(int c = 0; c < 3; ++c)
                    z[c] = (VT)t[c];
            }
            else
            {
                const double* D  = a.dinv + (size_t)row * 9;
                const double  r0 = r[0], r1 = r[1], r2 = r[2];
                z[0] = (VT)(D[0] * r0 + D[1] * r1 + D[2] * r2);
                z[1] = (VT)(D[3] * r0 + D[4] * r1 + D[5] * r2);
                z[2] = (VT)(D[6] * r0 + D[7] * r1 + D[8] * r2);
            }
        }
        double rz = 0.0, rr = 0.0;
        if(live)
#pragma unroll
            for(int c = 0; c < 3; ++c)
            {
                rz += (double)r[c] * (double)z[c];
                rr += (double)r[c] * (double)r[c];
            }
        block_partial(rz, part1, s_red[0]);
        block_partial(rr, part2, s_red[1]);
        if(!barrier())
            return;
        // the scalars of the iteration, the same in every thread
        sc.rz_new = sum_partials(part1);
        sc.rr     = sum_partials(part2);
        sc.iter += 1;
        const bool hit = (sc.stop_rule == B2S_STOP_RZ) ? (fabs(sc.rz_new) <= sc.rz_tol) : (sc.rr <= sc.rr_tol);
        if(!isfinite(sc.rz_new))
            sc.converged = 3;
        else if(hit)
        {
            sc.converged = 1;
            sc.iter_conv = sc.iter;
        }
        else if(sc.iter >= sc.max_iter - 1)
            sc.converged = 2;
        else
        {
            sc.beta = sc.rz_new / sc.rz;
            sc.rz   = sc.rz_new;
            if(live)
            {
#pragma unroll
                for(int c = 0; c < 3; ++c)
                    if constexpr(BF)
                        p[c] = __fmaf_rn((float)sc.beta, p[c], z[c]);
                    else
                        p[c] = z[c] + sc.beta * p[c];
                store_vec(a.p, i, p);
            }
            if(!barrier())
                return;
        }
    }
    if(live)
    {
        store_vec(a.x, i, x);
        store_vec(a.r, i, r);
    }
    // the fine level of the last apply (b2s_mas_get_nodes; the coarse levels are there)
    if(in_bank)
#pragma unroll
        for(int c = 0; c < 3; ++c)
        {
            a.A.R[3 * (int64_t)i + c] = (float)r[c];
            a.A.Z[3 * (int64_t)i + c] = s_z[w][(lane >> 4) * BANK * 3 + 3 * sub + c];
        }
    if(i == 0)
        *a.sc = sc;
}

// shared memory per block: the MAS stages
template <typename VT>
constexpr size_t small_smem(bool mas)
{
    return mas ? (size_t)(2 * SM_WARPS + 2 * SM_COARSE) * stage_bytes<sizeof(VT) == 4>() : 0;
}

// the grid: a thread per row, and at least a thread per two blocks (one load of
// the SpMV each) up to a block per SM. A second load in turn costs more than
// the arrivals of twice the blocks: with a thread per four blocks the solve of
// 1,331 rows took 1.35 ms against 1.19, of a 128 x 128 cloth (MAS) 1.187 against 1.170.
int small_grid(const Matrix& A)
{
    const int64_t rows = (A.nb + SM_THREADS - 1) / SM_THREADS;
    const int64_t blk  = (A.nnz + 2 * SM_THREADS - 1) / (2 * SM_THREADS);
    return (int)std::max<int64_t>(rows, std::min<int64_t>(blk, NUM_SMS_HINT));
}

template <typename VT>
bool launch(b2s_solver* s, const Matrix& A, int kind, long long iterations, double* x, const VT* vals, VT* r,
            VT* p, VT* Ap)
{
    PcgState&     P   = s->pcg;
    const bool    mas = kind == B2S_PRECOND_MAS;
    const int     grid = small_grid(A);
    SmallArgs<VT> a{};
    a.n    = A.nb;
    a.kind = kind;
    a.S    = A.stride;
    a.rows = A.rows.data();
    a.cols = A.cols.data();
    a.vals = vals;
    a.x    = x;
    a.r    = r;
    a.p    = p;
    a.Ap   = Ap;
    a.sc   = P.sc.data();
    a.mv   = mas_view(s);
    a.dinv = s->dinv.data();
    if(mas)
    {
        a.A         = mas_apply_args(s, sizeof(VT) == 4);
        a.comp_mask = s->mas.comp_mask[0].data();
        a.new_local = s->mas.new_local[0].data();
        a.part_dst  = s->mas.part_dst.data();
        a.part      = s->mas.part.data();
    }
    a.A.err      = device_error_flag(s);
    a.iterations = iterations;
    a.polls      = s->inject_polls < 0 ? SM_SPINS : (unsigned)s->inject_polls;
    try
    {
        P.small_partials.resize(3 * (size_t)grid);
        P.small_bar.resize(1);
    }
    catch(const OutOfMemory&)
    {
        return false;
    }
    a.partials = P.small_partials.data();
    a.bar      = P.small_bar.data();
    B2S_CUDA(cudaMemsetAsync(a.bar, 0, sizeof(unsigned), s->stream));
    const void*  k    = mas ? (const void*)k_pcg_small<VT, true> : (const void*)k_pcg_small<VT, false>;
    const size_t smem = small_smem<VT>(mas);
    B2S_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void* args[] = {&a};
    cudaError_t e = cudaErrorCooperativeLaunchTooLarge;
    if(s->inject_launch > 0)
        --s->inject_launch;
    else
        e = cudaLaunchCooperativeKernel(k, dim3(grid), dim3(SM_THREADS), args, smem, s->stream);
    if(e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported)
    {
        cudaGetLastError();
        return false;
    }
    B2S_CUDA(e);
    B2S_CHECK_LAUNCH();
    return true;
}
}  // namespace

// Whether the one-launch loop takes the system: every block resident at once
// (148 x 2 blocks of 256 rows), and few enough blocks per thread (of one block
// of threads per SM) that the barriers bound the iteration: its two-blocks-a-load
// SpMV streams a matrix slower than the launches' kernels do. Measured, us per
// iteration in one launch / launch by launch (graph), below and above each line:
//   Jacobi, FP64 (6):  227,000 blocks 18.9 / 21.9 (tets), 237,000 31.0 / 29.3 (cloth)
//   Jacobi, mixed (8): 301,000 blocks 17.0 / 19.4 (tets), 362,000 31.8 / 25.8 (cloth)
//   MAS, FP64 (3):      43,000 blocks 20.4 / 25.3 (tets), 121,000 31.9 / 30.8 (cloth)
//   MAS, mixed (5):    121,000 blocks 26.0 / 26.9 (cloth), 237,000 30.5 / 29.7 (cloth)
// At 70,000 rows the launches win by a quarter (cloth 71.7 / 54.6, MAS, FP64).
bool pcg_small_fits(b2s_solver* s, const Matrix& A, int kind, bool ord, bool f32)
{
    const bool mas = kind == B2S_PRECOND_MAS;
    if(A.nnz == 0 || (mas && !ord) || (ord && kind == B2S_PRECOND_JACOBI))
        return false;
    const void*  k    = f32 ? (mas ? (const void*)k_pcg_small<float, true> : (const void*)k_pcg_small<float, false>) :
                              (mas ? (const void*)k_pcg_small<double, true> : (const void*)k_pcg_small<double, false>);
    const size_t smem = f32 ? small_smem<float>(mas) : small_smem<double>(mas);
    const int    per_thread = mas ? (f32 ? 5 : 3) : (f32 ? 8 : 6);
    if(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    {
        cudaGetLastError();
        return false;
    }
    int occ = 0, sms = 0;
    if(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, SM_THREADS, smem) != cudaSuccess ||
       cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device) != cudaSuccess)
    {
        cudaGetLastError();
        return false;
    }
    return (int64_t)small_grid(A) <= (int64_t)occ * sms && A.nnz <= (int64_t)per_thread * SM_THREADS * sms;
}

bool pcg_small_launch(b2s_solver* s, const Matrix& A, int kind, long long iterations, double* x)
{
    PcgState& P = s->pcg;
    return launch<double>(s, A, kind, iterations, x, A.vals.data(), P.r.data(), P.p.data(), P.Ap.data());
}
bool pcg_small_launch_f32(b2s_solver* s, const Matrix& A, int kind, long long iterations, double* x)
{
    PcgState& P = s->pcg;
    return launch<float>(s, A, kind, iterations, x, A.vals32.data(), P.r32.data(), P.p32.data(), P.Ap32.data());
}
}  // namespace b2s
