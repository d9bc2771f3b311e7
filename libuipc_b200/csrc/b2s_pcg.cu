// Preconditioner build/apply dispatch and the PCG loop (FP64 path).
//
// PCG semantics follow LinearFusedPCG::fused_pcg
// (src/backends/cuda/linear_system/linear_fused_pcg.cu:1782-2005) and
// LinearPCG::pcg (src/backends/cuda/linear_system/linear_pcg.cu:558-644):
// x0 = 0 (or the given guess), r = b - A x0, z = P r, p = z; per iteration
// alpha = rz / pAp, x += alpha p, r -= alpha Ap, z = P r, rz' = r.z,
// converged when |rz'| <= tol |rz0| (or, with the relative-residual rule,
// ||r|| <= tol ||b||), beta = rz'/rz, p = z + beta p; max_iter = 2 n; the
// PSD guard re-runs with the preconditioner bypassed when rz0 < 0 or is not
// finite (:1819-1877). The scalars live on the device; the convergence flag
// freezes every kernel once set, so `check_interval` iterations can be
// replayed from one CUDA graph and checked once by the host, as the
// reference's graph block replay does (:1923-1998).
#include "b2s_internal.cuh"
#include "b2s_mas_apply.cuh"
#include "b2s_pcg.cuh"
#include "b2s_reduce.cuh"

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>

namespace b2s
{
void spmv_f64_launch(b2s_solver* s, const Matrix& A, const double* x, double* y, Reduction& red, double* d_dot,
                     const int* stop);
int  spmv_grid(int64_t U);
void mas_apply_levels(b2s_solver* s, const double* r, const int* converged);
void mas_apply_levels_f32(b2s_solver* s, const float* r, const int* converged, bool bf16);
void mas_pack_bf16(b2s_solver* s);
void spmv_f32_launch(b2s_solver* s, const Matrix& A, const float* x, float* y, Reduction& red, double* d_dot,
                     const int* stop);
void pcg_solve_mixed(b2s_solver* s, const double* b, double* x, const b2s_pcg_options& o, b2s_pcg_stats& st_out);
void build_row_groups(b2s_solver* s, Matrix& A);

namespace
{
constexpr int VEC_BLOCK = 256;

int vec_grid(int64_t n)
{
    int64_t g = (n + VEC_BLOCK - 1) / VEC_BLOCK;
    const int64_t cap = (int64_t)NUM_SMS_HINT * 8;
    if(g > cap)
        g = cap;
    return (int)(g < 1 ? 1 : g);
}

__device__ __forceinline__ bool frozen(const PcgScalars* sc) { return sc && sc->converged != 0; }

// 3x3 block Jacobi inverses (row-major), identity where the diagonal block is
// missing or singular. With r2p (MAS on rows off .. off + vn): only the rows
// outside its partition, the others' inverses are never applied
__global__ void k_diag_inverse(int32_t nb, const int32_t* diag_index, const double* vals, int64_t U, double* dinv,
                               const int32_t* __restrict__ r2p, int off, int vn)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= nb || (r2p && i >= off && i < off + vn && r2p[i - off] >= 0))
        return;
    const int k = diag_index[i];
    double*   o = dinv + (size_t)i * 9;
    if(k < 0)
    {
        for(int q = 0; q < 9; ++q)
            o[q] = (q % 4 == 0) ? 1.0 : 0.0;
        return;
    }
    double m[9];  // row-major
#pragma unroll
    for(int p = 0; p < 3; ++p)
#pragma unroll
        for(int q = 0; q < 3; ++q)
            m[p * 3 + q] = vals[(int64_t)(q * 3 + p) * U + k];
    const double c0 = m[4] * m[8] - m[5] * m[7], c1 = m[5] * m[6] - m[3] * m[8], c2 = m[3] * m[7] - m[4] * m[6];
    const double det = m[0] * c0 + m[1] * c1 + m[2] * c2;
    if(!(det != 0.0) || !isfinite(det))
    {
        for(int q = 0; q < 9; ++q)
            o[q] = (q % 4 == 0) ? 1.0 : 0.0;
        return;
    }
    const double id = 1.0 / det;
    o[0] = c0 * id;
    o[1] = (m[2] * m[7] - m[1] * m[8]) * id;
    o[2] = (m[1] * m[5] - m[2] * m[4]) * id;
    o[3] = c1 * id;
    o[4] = (m[0] * m[8] - m[2] * m[6]) * id;
    o[5] = (m[2] * m[3] - m[0] * m[5]) * id;
    o[6] = c2 * id;
    o[7] = (m[1] * m[6] - m[0] * m[7]) * id;
    o[8] = (m[0] * m[4] - m[1] * m[3]) * id;
}

// 12x12 block-Jacobi inverses of the affine bodies (ABDDiagPreconditioner,
// src/backends/cuda/affine_body/abd_diag_preconditioner.cu:15-125: the inverse
// of each body's full 12x12 diagonal Hessian block): body b owns block rows
// off + 4b .. off + 4b + 3; its 10 stored upper 3x3 blocks are gathered from
// the BSR (binary search of the sorted columns), mirrored, and inverted in FP64
// by Gauss-Jordan with partial pivoting (identity when singular). One warp per
// body: lane j < 24 holds column j of [H | I] in registers, the pivot column's
// lane finds the pivot and broadcasts its column. (One thread per body, its
// 12x24 array in local memory, took 122 us for 25 bodies, as long as for one.)
// Out: 144 doubles per body, row-major.
constexpr int ABD_WARPS = 4;
__global__ void __launch_bounds__(ABD_WARPS * 32) k_abd_inverse(int n_bodies, int off,
                                                                const int32_t* __restrict__ rowptr,
                                                                const int32_t* __restrict__ cols,
                                                                const double* __restrict__ vals, int64_t S,
                                                                double* __restrict__ out)
{
    const int lane = threadIdx.x & 31;
    const int b    = blockIdx.x * ABD_WARPS + (threadIdx.x >> 5);
    if(b >= n_bodies)
        return;
    // lanes 0-9 find the 10 upper blocks (bi, bj)
    int pos = -1;
    if(lane < 10)
    {
        const int bi = lane < 4 ? 0 : (lane < 7 ? 1 : (lane < 9 ? 2 : 3));
        const int bj = lane < 4 ? lane : (lane < 7 ? lane - 3 : (lane < 9 ? lane - 5 : 3));
        const int row = off + 4 * b + bi, col = off + 4 * b + bj;
        int       l = rowptr[row], h = rowptr[row + 1];
        const int end = h;
        while(l < h)
        {
            const int m = (l + h) >> 1;
            if(cols[m] < col)
                l = m + 1;
            else
                h = m;
        }
        if(l < end && cols[l] == col)
            pos = l;
    }
    double a[12];
#pragma unroll
    for(int i = 0; i < 12; ++i)
    {
        const int  j = lane < 12 ? lane : 0, bi = i / 3, bj = j / 3;
        const bool up = bi <= bj;
        const int  lo = up ? bi : bj, hi = up ? bj : bi;
        const int  l = __shfl_sync(0xffffffffu, pos, lo * 4 - lo * (lo - 1) / 2 + hi - lo);
        const int  p = up ? i % 3 : j % 3, q = up ? j % 3 : i % 3;
        a[i]         = lane < 12 ? (l >= 0 ? vals[(int64_t)(q * 3 + p) * S + l] : 0.0) : (lane - 12 == i ? 1.0 : 0.0);
    }
    bool ok = true;
#pragma unroll
    for(int c = 0; c < 12; ++c)
    {
        // the pivot of column c: its first largest entry from row c down
        int    piv = c;
        double big = fabs(a[c]), pv = a[c];
#pragma unroll
        for(int r = c + 1; r < 12; ++r)
            if(fabs(a[r]) > big)
            {
                piv = r;
                big = fabs(a[r]);
                pv  = a[r];
            }
        piv = __shfl_sync(0xffffffffu, piv, c);
        pv  = __shfl_sync(0xffffffffu, pv, c);
        if(!(fabs(pv) > 0.0) || !isfinite(pv))
        {
            ok = false;
            break;
        }
#pragma unroll
        for(int r = c + 1; r < 12; ++r)
            if(r == piv)
            {
                const double t = a[c];
                a[c]           = a[r];
                a[r]           = t;
            }
        a[c] *= 1.0 / pv;
        const double ac = a[c];
#pragma unroll
        for(int r = 0; r < 12; ++r)
            if(r != c)
            {
                const double f = __shfl_sync(0xffffffffu, a[r], c);
                if(f != 0.0)
                    a[r] -= f * ac;
            }
    }
    if(lane >= 12 && lane < 24)
#pragma unroll
        for(int i = 0; i < 12; ++i)
            out[(size_t)b * 144 + i * 12 + lane - 12] = ok ? a[i] : (lane - 12 == i ? 1.0 : 0.0);
}

// node i's three entries of r: NS = 3 values per node (FP64 vectors), or 4
// (the padded FP32 vectors of the mixed PCG: one 16-byte load)
template <typename VT, int NS>
__device__ __forceinline__ void load_r(const VT* r, int64_t i, double& a, double& b, double& c)
{
    if constexpr(NS == 4)
    {
        const float4 q = *reinterpret_cast<const float4*>(r + 4 * i);
        a = q.x;
        b = q.y;
        c = q.z;
    }
    else
    {
        a = r[3 * i];
        b = r[3 * i + 1];
        c = r[3 * i + 2];
    }
}

// the MAS value of slot p with level-1 node n1 (-1: none): the fine level's Z
// of the slot plus its coarse nodes' (level 1 up; neighbours mostly share
// them, so these are broadcast hits in L1)
__device__ __forceinline__ void mas_value(const MasView& mv, int p, int n1, double z[3])
{
    float c0 = mv.Z[3 * (int64_t)p], c1 = mv.Z[3 * (int64_t)p + 1], c2 = mv.Z[3 * (int64_t)p + 2];
    if(n1 >= 0)
    {
        const int4 a  = mv.anc[n1 - mv.begin1];
        float      w0 = mv.Z[3 * (int64_t)n1], w1 = mv.Z[3 * (int64_t)n1 + 1], w2 = mv.Z[3 * (int64_t)n1 + 2];
        const int  up[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for(int k = 0; k < 4; ++k)
            if(up[k] >= 0)
            {
                w0 += mv.Z[3 * (int64_t)up[k]];
                w1 += mv.Z[3 * (int64_t)up[k] + 1];
                w2 += mv.Z[3 * (int64_t)up[k] + 2];
            }
        c0 += w0;
        c1 += w1;
        c2 += w2;
    }
    z[0] = (double)c0;
    z[1] = (double)c1;
    z[2] = (double)c2;
}

// z_i for block row i: MAS (partitioned vertices of its range), else 3x3
// block Jacobi (kind 1 / 2), else identity (kind 0); r_i is returned in rr.
// ORD: r and i are in PCG order (the slots, then the other rows)
template <typename VT, int NS, bool ORD>
__device__ __forceinline__ void precond_row(int kind, const MasView& mv, const double* dinv, const VT* r, int i,
                                            double z[3], double rr[3])
{
    load_r<VT, NS>(r, i, rr[0], rr[1], rr[2]);
    const double r0 = rr[0], r1 = rr[1], r2 = rr[2];
    int          row = i;  // the matrix's row
    if constexpr(ORD)
    {
        if(kind == B2S_PRECOND_MAS && i < mv.slots)
        {
            mas_value(mv, i, mv.T > 0 ? mv.slot_node1[i] : -1, z);
            return;
        }
        if(kind != B2S_PRECOND_NONE)
            row = mv.row_of[i];
    }
    else if(kind == B2S_PRECOND_MAS && mv.active)
    {
        const int v = i - mv.off;
        if(v >= 0 && v < mv.vn)
        {
            const int p = mv.r2p[v];
            if(p >= 0)
            {
                mas_value(mv, p, mv.T > 0 ? mv.node1[v] : -1, z);
                return;
            }
        }
    }
    if(kind == B2S_PRECOND_NONE)
    {
        z[0] = r0;
        z[1] = r1;
        z[2] = r2;
        return;
    }
    if(mv.abd_n > 0 && row >= mv.abd_off && row < mv.abd_off + 4 * mv.abd_n)
    {
        // row l of body b: z = (H_b^-1)[3l .. 3l+2][0 .. 11] r_b
        const int     b = (row - mv.abd_off) >> 2, l = (row - mv.abd_off) & 3;
        const double* Hi = mv.abd_inv + (size_t)b * 144 + 36 * l;
        double        a0 = 0.0, a1 = 0.0, a2 = 0.0;
        for(int j = 0; j < 12; ++j)
        {
            // in PCG order a body's rows need not follow one another: a caller
            // may have put some of them into the MAS partition
            const int64_t n  = ORD ? mv.pos[row - l + j / 3] : row - l + j / 3;
            const double  rj = r[NS * n + j % 3];
            a0 += Hi[j] * rj;
            a1 += Hi[12 + j] * rj;
            a2 += Hi[24 + j] * rj;
        }
        z[0] = a0;
        z[1] = a1;
        z[2] = a2;
        return;
    }
    const double* D = dinv + (size_t)row * 9;
    z[0] = D[0] * r0 + D[1] * r1 + D[2] * r2;
    z[1] = D[3] * r0 + D[4] * r1 + D[5] * r2;
    z[2] = D[6] * r0 + D[7] * r1 + D[8] * r2;
}

// z = P r for every block row; with `sc`, also r.z and r.r (FP64 sums) and
// the scalar update of the iteration (last block). VT: vector storage type.
// 32 registers, so the whole reduction grid (8 CTAs per SM) is resident at
// once (with 40 the last quarter of the grid ran as a second wave: the MAS
// apply with this finish measured 77.4 -> 73.8 us on 551 k vertices).
template <typename VT, int NS, bool ORD>
__global__ void __launch_bounds__(RED_BLOCK, 8) k_precond_finish(int32_t nb, int kind, MasView mv,
                                                              const double* __restrict__ dinv,
                                                              const VT* __restrict__ r, VT* __restrict__ z,
                                                              PcgScalars* sc, double* partials,
                                                              unsigned int* counter)
{
    if(frozen(sc))
        return;
    double rz = 0.0, rr = 0.0;
    for(int i = blockIdx.x * RED_BLOCK + threadIdx.x; i < nb; i += gridDim.x * RED_BLOCK)
    {
        double zi[3], ri[3];
        precond_row<VT, NS, ORD>(kind, mv, dinv, r, i, zi, ri);
        const VT z0 = (VT)zi[0], z1 = (VT)zi[1], z2 = (VT)zi[2];
        if constexpr(NS == 4)
            *reinterpret_cast<float4*>(z + 4 * (int64_t)i) = make_float4(z0, z1, z2, 0.0f);
        else
        {
            z[3 * (int64_t)i]     = z0;
            z[3 * (int64_t)i + 1] = z1;
            z[3 * (int64_t)i + 2] = z2;
        }
        if(sc)
        {
            rz += ri[0] * (double)z0 + ri[1] * (double)z1 + ri[2] * (double)z2;
            rr += ri[0] * ri[0] + ri[1] * ri[1] + ri[2] * ri[2];
        }
    }
    if(!sc)
        return;
    double v[2] = {rz, rr}, tot[2];
    if(!grid_sum<2>(v, partials, counter, tot))
        return;
    // scalar update of the iteration (one thread)
    const double rz_new = tot[0];
    sc->rz_new          = rz_new;
    sc->rr              = tot[1];
    sc->iter += 1;
    const bool hit = (sc->stop_rule == B2S_STOP_RZ) ? (fabs(rz_new) <= sc->rz_tol) : (tot[1] <= sc->rr_tol);
    if(!isfinite(rz_new))
        sc->converged = 3;
    else if(hit)
    {
        sc->converged = 1;
        sc->iter_conv = sc->iter;
    }
    else if(sc->iter >= sc->max_iter - 1)
        sc->converged = 2;
    else
    {
        sc->beta = rz_new / sc->rz;
        sc->rz   = rz_new;
    }
}

__global__ void k_update_xr(int64_t n, PcgScalars* sc, double* __restrict__ x, const double* __restrict__ p,
                            double* __restrict__ r, double* __restrict__ Ap)
{
    if(frozen(sc))
        return;
    const double alpha = sc->rz / sc->pAp;
    if(blockIdx.x == 0 && threadIdx.x == 0)
        sc->alpha = alpha;
    for(int64_t i = (int64_t)blockIdx.x * VEC_BLOCK + threadIdx.x; i < n; i += (int64_t)gridDim.x * VEC_BLOCK)
    {
        const double api = Ap[i];
        x[i] += alpha * p[i];
        r[i] -= alpha * api;
        Ap[i] = 0.0;
    }
}

__global__ void k_update_p(int64_t n, const PcgScalars* sc, const double* __restrict__ z, double* __restrict__ p)
{
    if(frozen(sc))
        return;
    const double beta = sc->beta;
    for(int64_t i = (int64_t)blockIdx.x * VEC_BLOCK + threadIdx.x; i < n; i += (int64_t)gridDim.x * VEC_BLOCK)
        p[i] = z[i] + beta * p[i];
}

// ---- mixed precision (FP32 vectors, FP64 solution and scalars) ----------------
// The FP32 vectors (r, z, p, Ap) hold 4 floats per node, the 4th zero
// (16-byte gathers and vector reductions in the SpMV and the MAS apply); the
// FP64 solution x holds 3. x += alpha p, r -= alpha Ap, Ap = 0, one node per
// thread and step.
__global__ void k_update_xr_mixed4(int32_t nb, PcgScalars* sc, double* __restrict__ x, const float* __restrict__ p,
                                   float* __restrict__ r, const float* __restrict__ Ap)
{
    if(frozen(sc))
        return;
    const double alpha = sc->rz / sc->pAp;
    if(blockIdx.x == 0 && threadIdx.x == 0)
        sc->alpha = alpha;
    const float af = (float)alpha;
    for(int64_t i = (int64_t)blockIdx.x * VEC_BLOCK + threadIdx.x; i < nb; i += (int64_t)gridDim.x * VEC_BLOCK)
    {
        const float4 ap = reinterpret_cast<const float4*>(Ap)[i];
        const float4 pp = reinterpret_cast<const float4*>(p)[i];
        float4       rr = reinterpret_cast<float4*>(r)[i];
        x[3 * i] += alpha * (double)pp.x;
        x[3 * i + 1] += alpha * (double)pp.y;
        x[3 * i + 2] += alpha * (double)pp.z;
        rr.x = __fmaf_rn(-af, ap.x, rr.x);
        rr.y = __fmaf_rn(-af, ap.y, rr.y);
        rr.z = __fmaf_rn(-af, ap.z, rr.z);
        reinterpret_cast<float4*>(r)[i] = rr;
    }
}

// The same update in PCG order with the MAS restriction in the pass: the
// first `slots` rows are the partition slots, 16 per bank, so the half-warp
// that updates a bank's residuals also writes them as R_0 (FP32), and the
// block their sums at the coarse levels (restrict_coarse). In the vertices'
// own order the restriction was a launch of its own that gathered r through
// the partition: 20.3 us for update and restriction of 551,368 vertices (mixed),
// 16.7 here with the sums of every coarse level. NS: entries per node (3: FP64
// vectors, Ap zeroed here; 4: padded FP32). UPDATE = false: only the restriction of r.
template <typename VT, int NS, bool UPDATE>
__global__ void __launch_bounds__(VEC_BLOCK)
    k_update_restrict(int32_t n, int32_t slots, PcgScalars* sc, double* __restrict__ x, const VT* __restrict__ p,
                      VT* __restrict__ r, VT* __restrict__ Ap, const uint16_t* __restrict__ comp_mask,
                      const int32_t* __restrict__ new_local, const int4* __restrict__ dst, int begin1, int push,
                      float* __restrict__ R, double* __restrict__ part)
{
    if(UPDATE && frozen(sc))
        return;
    __shared__ float s_r[VEC_BLOCK][3];
    __shared__ float s_p[VEC_BLOCK][3];  // p (NS = 4), then the components' sums
    __shared__ int4  s_dst[VEC_BLOCK];
    __shared__ int   s_n[VEC_BLOCK / 32];
    const int        t = threadIdx.x, i = blockIdx.x * VEC_BLOCK + t, sub = t & 15;
    const int64_t    e0 = 3 * (int64_t)blockIdx.x * VEC_BLOCK;  // the block's first entry of 3 per node
    uint32_t         cm = 0;
    int              nl = 0;
    int4             to = make_int4(-1, -1, -1, -1);
    if(i < slots && push)
    {
        cm = comp_mask[i];
        nl = new_local[i];
        if(cm != 0 && (cm & ((1u << sub) - 1u)) == 0)
            to = dst[nl];
    }
    double alpha = 0.0;
    if constexpr(UPDATE)
        alpha = sc->rz / sc->pAp;
    float* fr = &s_r[0][0];
    if constexpr(NS == 4)
    {
        if(i < n)
        {
            float4 rr = reinterpret_cast<const float4*>(r)[i];
            if constexpr(UPDATE)
            {
                const float  af = (float)alpha;
                const float4 ap = reinterpret_cast<const float4*>(Ap)[i];
                const float4 pp = reinterpret_cast<const float4*>(p)[i];
                rr.x = __fmaf_rn(-af, ap.x, rr.x);
                rr.y = __fmaf_rn(-af, ap.y, rr.y);
                rr.z = __fmaf_rn(-af, ap.z, rr.z);
                reinterpret_cast<float4*>(r)[i] = rr;
                s_p[t][0] = pp.x;
                s_p[t][1] = pp.y;
                s_p[t][2] = pp.z;
            }
            s_r[t][0] = rr.x;
            s_r[t][1] = rr.y;
            s_r[t][2] = rr.z;
        }
        __syncthreads();
    }
    // the arrays of 3 per node, entry by entry (consecutive lanes on
    // consecutive entries: thread by node, each access spread over 3 times the
    // lines)
#pragma unroll
    for(int j = 0; j < 3; ++j)
    {
        const int     f = t + j * VEC_BLOCK;
        const int64_t e = e0 + f;
        if(e >= 3 * (int64_t)n)
            continue;
        if constexpr(NS == 4)
        {
            if constexpr(UPDATE)
                x[e] += alpha * (double)(&s_p[0][0])[f];
        }
        else
        {
            double q = r[e];
            if constexpr(UPDATE)
            {
                x[e] += alpha * p[e];
                q -= alpha * Ap[e];
                r[e]  = q;
                Ap[e] = 0.0;
            }
            fr[f] = (float)q;
        }
        if(e < 3 * (int64_t)slots)
            R[e] = fr[f];
    }
    if(UPDATE && i == 0)
        sc->alpha = alpha;
    if(push)
    {
        __syncthreads();  // s_r is complete, s_p is free
        restrict_coarse<VEC_BLOCK>(s_r, cm, nl, to, begin1, R, part, s_p, s_dst, s_n);
    }
}

// p = z + beta p over the padded vectors (nb nodes), and Ap = 0 for the
// SpMV that follows: zeroed here rather than after its last reader, so the
// zero lines are still in L2 when the SpMV's reductions reach them
__global__ void k_update_p_mixed4(int32_t nb, const PcgScalars* sc, const float* __restrict__ z, float* __restrict__ p,
                                  float* __restrict__ Ap)
{
    if(frozen(sc))
        return;
    const float beta = (float)sc->beta;
    for(int64_t i = (int64_t)blockIdx.x * VEC_BLOCK + threadIdx.x; i < nb; i += (int64_t)gridDim.x * VEC_BLOCK)
    {
        const float4 zz = reinterpret_cast<const float4*>(z)[i];
        float4       pp = reinterpret_cast<float4*>(p)[i];
        pp.x = __fmaf_rn(beta, pp.x, zz.x);
        pp.y = __fmaf_rn(beta, pp.y, zz.y);
        pp.z = __fmaf_rn(beta, pp.z, zz.z);
        pp.w = __fmaf_rn(beta, pp.w, zz.w);
        reinterpret_cast<float4*>(p)[i]  = pp;
        reinterpret_cast<float4*>(Ap)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// r32 = b - Ax computed in FP64, stored FP32 (padded: 4 floats per node)
__global__ void k_residual_f32(int32_t nb, const double* __restrict__ b, const double* __restrict__ Ax,
                               float* __restrict__ r)
{
    for(int64_t i = (int64_t)blockIdx.x * VEC_BLOCK + threadIdx.x; i < nb; i += (int64_t)gridDim.x * VEC_BLOCK)
        reinterpret_cast<float4*>(r)[i] = make_float4((float)(b[3 * i] - Ax[3 * i]), (float)(b[3 * i + 1] - Ax[3 * i + 1]),
                                                      (float)(b[3 * i + 2] - Ax[3 * i + 2]), 0.0f);
}

// r = b - Ax in PCG order (b, Ax in the matrix's order; Ax null: r = b), zero in
// padding slots; NS = 4: FP32, padded
template <typename VT, int NS>
__global__ void k_residual_ord(int32_t n, const int32_t* __restrict__ row_of, const double* __restrict__ b,
                               const double* __restrict__ Ax, VT* __restrict__ r)
{
    for(int i = blockIdx.x * VEC_BLOCK + threadIdx.x; i < n; i += gridDim.x * VEC_BLOCK)
    {
        const int64_t o = 3 * (int64_t)row_of[i];
        double        v[3] = {0.0, 0.0, 0.0};
        if(o >= 0)
#pragma unroll
            for(int c = 0; c < 3; ++c)
                v[c] = Ax ? b[o + c] - Ax[o + c] : b[o + c];
        if constexpr(NS == 4)
            reinterpret_cast<float4*>(r)[i] = make_float4((float)v[0], (float)v[1], (float)v[2], 0.0f);
        else
#pragma unroll
            for(int c = 0; c < 3; ++c)
                r[3 * (int64_t)i + c] = v[c];
    }
}

// FP64 vector between the matrix's order and PCG order
__global__ void k_to_ord(int32_t n, const int32_t* __restrict__ row_of, const double* __restrict__ x,
                         double* __restrict__ xs)
{
    for(int i = blockIdx.x * VEC_BLOCK + threadIdx.x; i < n; i += gridDim.x * VEC_BLOCK)
    {
        const int64_t o = 3 * (int64_t)row_of[i];
#pragma unroll
        for(int c = 0; c < 3; ++c)
            xs[3 * (int64_t)i + c] = o >= 0 ? x[o + c] : 0.0;
    }
}
__global__ void k_from_ord(int32_t nb, const int32_t* __restrict__ pos, const double* __restrict__ xs,
                           double* __restrict__ x)
{
    for(int r = blockIdx.x * VEC_BLOCK + threadIdx.x; r < nb; r += gridDim.x * VEC_BLOCK)
    {
        const int64_t i = 3 * (int64_t)pos[r];
#pragma unroll
        for(int c = 0; c < 3; ++c)
            x[3 * (int64_t)r + c] = xs[i + c];
    }
}

// the order: 1 for the rows outside the MAS slots, then their places
__global__ void k_ord_other(int32_t nb, int off, int vn, const int32_t* __restrict__ r2p, int32_t* __restrict__ other)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i < nb)
        other[i] = (i < off || i >= off + vn || r2p[i - off] < 0) ? 1 : 0;
}
__global__ void k_ord_pos(int32_t nb, int off, int vn, int slots, const int32_t* __restrict__ r2p,
                          const int32_t* __restrict__ rank, int32_t* __restrict__ pos, int32_t* __restrict__ row_of)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= nb)
        return;
    const int p = (i >= off && i < off + vn) ? r2p[i - off] : -1;
    const int q = p >= 0 ? p : slots + rank[i];
    pos[i]      = q;
    row_of[q]   = i;
}
__global__ void k_ord_node1(int slots, int begin1, const int32_t* __restrict__ new_local, int32_t* __restrict__ node1)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if(p < slots)
        node1[p] = new_local[p] >= 0 ? begin1 + new_local[p] : -1;
}

// the matrix in that order: blocks per row (one at least), the rows' blocks
// moved together (columns renumbered, the order inside a row kept; row and
// column may swap sides, which a symmetric product does not mind), and the
// zero diagonal blocks of the empty rows
__global__ void k_ord_count(int32_t n, const int32_t* __restrict__ row_of, const int32_t* __restrict__ rowptr,
                            int32_t* __restrict__ cnt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n)
        return;
    const int r = row_of[i];
    cnt[i]      = r >= 0 ? max(rowptr[r + 1] - rowptr[r], 1) : 1;
}
template <typename VT>
__global__ void k_ord_fill(int64_t U, int64_t S, int64_t So, const int32_t* __restrict__ pos,
                           const int32_t* __restrict__ rowptr, const int32_t* __restrict__ rows,
                           const int32_t* __restrict__ cols, const double* __restrict__ vals,
                           const int32_t* __restrict__ rowptr_o, int32_t* __restrict__ rows_o,
                           int32_t* __restrict__ cols_o, VT* __restrict__ vals_o)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(k >= U)
        return;
    const int     r = rows[k], i = pos[r];
    const int64_t d = (int64_t)rowptr_o[i] + (k - rowptr[r]);
    rows_o[d]       = i;
    cols_o[d]       = pos[cols[k]];
#pragma unroll
    for(int q = 0; q < 9; ++q)
        vals_o[q * So + d] = (VT)vals[q * S + k];
}
template <typename VT>
__global__ void k_ord_empty(int32_t n, int64_t So, const int32_t* __restrict__ row_of,
                            const int32_t* __restrict__ rowptr, const int32_t* __restrict__ rowptr_o,
                            int32_t* __restrict__ rows_o, int32_t* __restrict__ cols_o, VT* __restrict__ vals_o)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n)
        return;
    const int     r = row_of[i];
    const int64_t d = rowptr_o[i];
    if(r < 0 || rowptr[r + 1] == rowptr[r])
    {
        rows_o[d] = i;
        cols_o[d] = i;
#pragma unroll
        for(int q = 0; q < 9; ++q)
            vals_o[q * So + d] = (VT)0;
    }
    if(i == n - 1)  // the padding of the stream
        for(int64_t e = rowptr_o[n]; e < So; ++e)
        {
            rows_o[e] = -1;
            cols_o[e] = 0;
#pragma unroll
            for(int q = 0; q < 9; ++q)
                vals_o[q * So + e] = (VT)0;
        }
}

// between the 3-per-node FP32 vectors of the ABI and the padded ones
// (with `zero`, that padded vector is cleared in the same pass)
__global__ void k_pad4(int32_t nb, const float* __restrict__ a, float* __restrict__ b, float* __restrict__ zero)
{
    for(int64_t i = (int64_t)blockIdx.x * VEC_BLOCK + threadIdx.x; i < nb; i += (int64_t)gridDim.x * VEC_BLOCK)
    {
        reinterpret_cast<float4*>(b)[i] = make_float4(a[3 * i], a[3 * i + 1], a[3 * i + 2], 0.0f);
        if(zero)
            reinterpret_cast<float4*>(zero)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__global__ void k_unpad4(int32_t nb, const float* __restrict__ a, float* __restrict__ b)
{
    for(int64_t i = (int64_t)blockIdx.x * VEC_BLOCK + threadIdx.x; i < nb; i += (int64_t)gridDim.x * VEC_BLOCK)
    {
        const float4 q = reinterpret_cast<const float4*>(a)[i];
        b[3 * i]       = q.x;
        b[3 * i + 1]   = q.y;
        b[3 * i + 2]   = q.z;
    }
}

// FP32 vectors, FP64 sums: out[0] = a.b, out[1] = a.a
__global__ void __launch_bounds__(RED_BLOCK) k_dot2_f32(int64_t n, const float* __restrict__ a,
                                                        const float* __restrict__ b, double* partials,
                                                        unsigned int* counter, double* out)
{
    double ab = 0.0, aa = 0.0;
    for(int64_t i = (int64_t)blockIdx.x * RED_BLOCK + threadIdx.x; i < n; i += (int64_t)gridDim.x * RED_BLOCK)
    {
        const double ai = a[i];
        ab += ai * (double)b[i];
        aa += ai * ai;
    }
    double v[2] = {ab, aa}, tot[2];
    if(grid_sum<2>(v, partials, counter, tot))
    {
        out[0] = tot[0];
        out[1] = tot[1];
    }
}

// scalars and error bits (cleared) into pinned host memory
__global__ void k_scalars_out(const PcgScalars* sc, int* err, PcgScalars* out, ReadBack* back)
{
    *out      = *sc;
    back->err = atomicExch(err, 0);
}

// FP32 copy of the value planes (mixed-precision SpMV)
__global__ void k_planes_f32(int64_t count, const double* __restrict__ src, float* __restrict__ dst)
{
    for(int64_t i = (int64_t)blockIdx.x * VEC_BLOCK + threadIdx.x; i < count; i += (int64_t)gridDim.x * VEC_BLOCK)
        dst[i] = (float)src[i];
}

__global__ void k_residual(int64_t n, const double* __restrict__ b, const double* __restrict__ Ax,
                           double* __restrict__ r)
{
    for(int64_t i = (int64_t)blockIdx.x * VEC_BLOCK + threadIdx.x; i < n; i += (int64_t)gridDim.x * VEC_BLOCK)
        r[i] = b[i] - Ax[i];
}

// sum (b - Ax)^2 and b.b
__global__ void __launch_bounds__(RED_BLOCK) k_res_norms(int64_t n, const double* __restrict__ b,
                                                         const double* __restrict__ Ax, double* partials,
                                                         unsigned int* counter, double* out)
{
    double rr = 0.0, bb = 0.0;
    for(int64_t i = (int64_t)blockIdx.x * RED_BLOCK + threadIdx.x; i < n; i += (int64_t)gridDim.x * RED_BLOCK)
    {
        const double d = b[i] - Ax[i];
        rr += d * d;
        bb += b[i] * b[i];
    }
    double v[2] = {rr, bb}, tot[2];
    if(grid_sum<2>(v, partials, counter, tot))
    {
        out[0] = tot[0];
        out[1] = tot[1];
    }
}

}  // namespace

// ---------------------------------------------------------------------------
void precond_assemble(b2s_solver* s, int kind, int invert_mode)
{
    B2S_REQUIRE(s->A.valid, B2S_ERR_STATE, "precond_assemble before b2s_assemble");
    B2S_REQUIRE(kind >= B2S_PRECOND_NONE && kind <= B2S_PRECOND_MAS, B2S_ERR_ARGUMENT, "unknown preconditioner");
    B2S_REQUIRE(invert_mode == B2S_INVERT_F32 || invert_mode == B2S_INVERT_F64 || invert_mode == B2S_INVERT_F32_ONLY,
                B2S_ERR_ARGUMENT,
                "unknown inversion mode");
    cudaStream_t st = s->stream;
    const Matrix& A = s->A;
    s->dinv.resize((size_t)std::max(A.nb, 1) * 9);
    const bool mas = kind == B2S_PRECOND_MAS;
    B2S_REQUIRE(!mas || s->mas.initialized, B2S_ERR_STATE, "MAS preconditioner requested before b2s_mas_init");
    if(A.nb > 0)
    {
        k_diag_inverse<<<grid_for(A.nb, 256), 256, 0, st>>>(A.nb, A.diag_index.data(), A.vals.data(), A.stride,
                                                            s->dinv.data(), mas ? s->mas.r2p.data() : nullptr,
                                                            s->mas.offset, s->mas.vn);
        B2S_CHECK_LAUNCH();
    }
    if(mas)
        mas_assemble(s, invert_mode);
    if(s->abd_n > 0)
    {
        B2S_REQUIRE(s->abd_offset + 4 * (int64_t)s->abd_n <= A.nb, B2S_ERR_ARGUMENT,
                    "affine-body range exceeds the matrix");
        s->abd_inv.resize((size_t)s->abd_n * 144);
        k_abd_inverse<<<grid_for(s->abd_n, ABD_WARPS), ABD_WARPS * 32, 0, st>>>(s->abd_n, s->abd_offset, A.rowptr.data(),
                                                               A.cols.data(), A.vals.data(), A.stride,
                                                               s->abd_inv.data());
        B2S_CHECK_LAUNCH();
    }
    s->precond_kind = kind;
    s->precond_generation += 1;
    s->invert_mode  = invert_mode;
    B2S_CUDA(cudaStreamSynchronize(st));
}

MasView mas_view(b2s_solver* s)
{
    MasView mv{};
    const MasState& M = s->mas;
    mv.active = (s->precond_kind == B2S_PRECOND_MAS && M.initialized) ? 1 : 0;
    mv.abd_n   = s->abd_n;
    mv.abd_off = s->abd_offset;
    mv.abd_inv = s->abd_inv.data();
    mv.off    = M.offset;
    mv.vn     = M.vn;
    mv.r2p    = M.r2p.data();
    mv.node1  = M.node1.data();
    mv.anc    = M.anc.data();
    mv.begin1 = M.L > 1 ? M.level_begin[1] : 0;
    mv.T      = M.L <= 1 ? 0 : M.L - 1;
    mv.Z      = M.Z.data();
    mv.row_of     = s->pcg.ord.row_of.data();
    mv.pos        = s->pcg.ord.pos.data();
    mv.slot_node1 = s->pcg.ord.node1.data();
    mv.slots      = s->pcg.ord.slots;
    return mv;
}

// the PCG order of the current MAS and matrix, and the matrix in it
static void ensure_order(b2s_solver* s, bool f32)
{
    PcgOrder&       O  = s->pcg.ord;
    const MasState& M  = s->mas;
    const Matrix&   A  = s->A;
    cudaStream_t    st = s->stream;
    const int       TB = 256;
    AssemblyScratch& w = s->asmb;
    if(O.mas_generation != M.generation || O.nb != A.nb)
    {
        O.mas_generation = -1;
        O.f64_generation = O.f32_generation = -1;
        w.row_count.resize((size_t)A.nb + 1, 1.25);
        w.row_start.resize((size_t)A.nb + 1, 1.25);
        k_ord_other<<<grid_for(A.nb, TB), TB, 0, st>>>(A.nb, M.offset, M.vn, M.r2p.data(), w.row_count.data());
        B2S_CHECK_LAUNCH();
        exclusive_scan(s, w.row_count.data(), w.row_start.data(), A.nb, w.scan_tmp);
        int32_t others = 0;
        B2S_CUDA(cudaMemcpyAsync(&others, w.row_start.data() + A.nb, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        B2S_CUDA(cudaStreamSynchronize(st));
        O.slots = M.N;
        O.nb    = A.nb;
        O.n     = M.N + others;
        O.row_of.resize(O.n);
        O.pos.resize(A.nb);
        B2S_CUDA(cudaMemsetAsync(O.row_of.data(), 0xff, O.row_of.bytes(), st));
        k_ord_pos<<<grid_for(A.nb, TB), TB, 0, st>>>(A.nb, M.offset, M.vn, M.N, M.r2p.data(), w.row_start.data(),
                                                     O.pos.data(), O.row_of.data());
        B2S_CHECK_LAUNCH();
        O.node1.resize(M.N);
        k_ord_node1<<<grid_for(M.N, TB), TB, 0, st>>>(M.N, M.L > 1 ? M.level_begin[1] : 0, M.new_local[0].data(),
                                                      O.node1.data());
        B2S_CHECK_LAUNCH();
        O.mas_generation = M.generation;
    }
    if((f32 ? O.f32_generation : O.f64_generation) == A.generation)
        return;
    Matrix& P = O.A;
    if(O.f32_generation != A.generation && O.f64_generation != A.generation)
    {
        w.row_count.resize((size_t)O.n + 1, 1.25);
        P.rowptr.resize((size_t)O.n + 1, 1.25);
        k_ord_count<<<grid_for(O.n, TB), TB, 0, st>>>(O.n, O.row_of.data(), A.rowptr.data(), w.row_count.data());
        B2S_CHECK_LAUNCH();
        exclusive_scan(s, w.row_count.data(), P.rowptr.data(), O.n, w.scan_tmp);
        int32_t nnz = 0;
        B2S_CUDA(cudaMemcpyAsync(&nnz, P.rowptr.data() + O.n, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        B2S_CUDA(cudaStreamSynchronize(st));
        P.nb     = O.n;
        P.nnz    = nnz;
        P.stride = (P.nnz + 15) / 16 * 16;
        P.rows.resize(P.stride, 1.2);
        P.cols.resize(P.stride, 1.2);
        P.has_trank = P.has_groups = false;
    }
    auto fill = [&](auto* vals)
    {
        using VT = std::remove_pointer_t<decltype(vals)>;
        if(A.nnz > 0)
        {
            k_ord_fill<VT><<<grid_for(A.nnz, TB), TB, 0, st>>>(A.nnz, A.stride, P.stride, O.pos.data(),
                                                               A.rowptr.data(), A.rows.data(), A.cols.data(),
                                                               A.vals.data(), P.rowptr.data(), P.rows.data(),
                                                               P.cols.data(), vals);
            B2S_CHECK_LAUNCH();
        }
        k_ord_empty<VT><<<grid_for(O.n, TB), TB, 0, st>>>(O.n, P.stride, O.row_of.data(), A.rowptr.data(),
                                                          P.rowptr.data(), P.rows.data(), P.cols.data(), vals);
        B2S_CHECK_LAUNCH();
    };
    if(f32)
    {
        P.vals32.resize((size_t)9 * P.stride, 1.2);
        fill(P.vals32.data());
        if(!P.has_groups)
            build_row_groups_full(s, P);
        O.f32_generation = A.generation;
    }
    else
    {
        P.vals.resize((size_t)9 * P.stride, 1.2);
        fill(P.vals.data());
        O.f64_generation = A.generation;
    }
}

// ensure_order and room(true), which allocates what the solve needs in that
// order; false when the device has no room for the second copy of the matrix and
// the longer vectors. They are given back then, and the recursion runs in the
// matrix's own order.
template <typename Room>
static bool try_order(b2s_solver* s, bool f32, const Room& room)
{
    try
    {
        ensure_order(s, f32);
        room(true);
        return true;
    }
    catch(const OutOfMemory&)
    {
        PcgState& P = s->pcg;
        PcgOrder& O = P.ord;
        for(DBuf<double>* d : {&O.A.vals, &P.xs, &P.r, &P.z, &P.p, &P.Ap})
            d->release();
        for(DBuf<float>* d : {&O.A.vals32, &P.r32, &P.z32, &P.p32, &P.Ap32})
            d->release();
        O.A.rows.release();
        O.A.cols.release();
        O.A.trank.release();
        O.A.has_trank    = false;
        O.f64_generation = O.f32_generation = -1;
        return false;
    }
}

// the restriction in PCG order, with the x, r update of the iteration
// (UPDATE). Without an apply to follow (kind other than MAS) nothing is
// restricted.
template <typename VT, int NS, bool UPDATE>
static void update_restrict_launch(b2s_solver* s, int kind, PcgScalars* sc, double* xs, const VT* p, VT* r, VT* Ap)
{
    const PcgOrder& O = s->pcg.ord;
    MasState&       M = s->mas;
    k_update_restrict<VT, NS, UPDATE><<<grid_for(O.n, VEC_BLOCK), VEC_BLOCK, 0, s->stream>>>(
        O.n, O.slots, sc, xs, p, r, Ap, M.comp_mask[0].data(), M.new_local[0].data(), M.part_dst.data(),
        M.L > 1 ? M.level_begin[1] : 0, kind == B2S_PRECOND_MAS && M.L > 1 ? 1 : 0, M.R.data(), M.part.data());
    B2S_CHECK_LAUNCH();
}

// z = P r in PCG order from R_0 and R_1 (update_restrict_launch first), with
// the dots and the scalar update of the iteration when `sc` is given
template <typename VT, int NS>
static void precond_launch_ord(b2s_solver* s, int kind, bool bf16, const VT* r, VT* z, PcgScalars* sc, Reduction& red)
{
    const int32_t n = s->pcg.ord.n;
    if(kind == B2S_PRECOND_MAS)
        mas_apply_all(s, sc ? &sc->converged : nullptr, bf16);
    const int grid = reduction_grid(n);
    ensure_reduction(s, red, grid, 2);
    k_precond_finish<VT, NS, true><<<grid, RED_BLOCK, 0, s->stream>>>(n, kind, mas_view(s), s->dinv.data(), r, z, sc,
                                                                     red.partials.data(), red.counter.data());
    B2S_CHECK_LAUNCH();
}

// z = P r, optionally fused with the dots + scalar update of a PCG iteration
static void precond_launch(b2s_solver* s, int kind, const double* r, double* z, PcgScalars* sc, Reduction& red)
{
    cudaStream_t st = s->stream;
    const int32_t nb = s->A.nb;
    if(nb == 0)
        return;
    if(kind == B2S_PRECOND_MAS)
        mas_apply_levels(s, r, sc ? &sc->converged : nullptr);
    const int grid = reduction_grid(nb);
    ensure_reduction(s, red, grid, 2);
    k_precond_finish<double, 3, false><<<grid, RED_BLOCK, 0, st>>>(nb, kind, mas_view(s), s->dinv.data(), r, z, sc,
                                                 red.partials.data(), red.counter.data());
    B2S_CHECK_LAUNCH();
}

void precond_apply(b2s_solver* s, const double* r, double* z)
{
    B2S_REQUIRE(s->precond_kind >= 0, B2S_ERR_STATE, "precond_apply before b2s_precond_assemble");
    precond_launch(s, s->precond_kind, r, z, nullptr, s->red);
    read_back(s, nullptr, 0, nullptr);
}

// z = P r queued on the solver's stream (no synchronisation, no error check)
void precond_launch(b2s_solver* s, const double* r, double* z)
{
    B2S_REQUIRE(s->precond_kind >= 0, B2S_ERR_STATE, "precond_apply before b2s_precond_assemble");
    precond_launch(s, s->precond_kind, r, z, nullptr, s->red);
}

// ---------------------------------------------------------------------------
// PCG
// ---------------------------------------------------------------------------
namespace
{
// iterations per launch of the one-launch loop at most (bounds its duration)
constexpr long long SMALL_LOOP = 1 << 14;

struct GraphKey
{
    const void* ptrs[14];
    int64_t     ints[6];
    bool operator==(const GraphKey& o) const { return std::memcmp(this, &o, sizeof(GraphKey)) == 0; }
};
}  // namespace

// a stage-timing event: an external event node when the stream is being
// captured into the PCG graph, a plain stream event otherwise
static cudaError_t record_timing_event(cudaEvent_t ev, cudaStream_t st)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaError_t             e  = cudaStreamIsCapturing(st, &cs);
    if(e != cudaSuccess)
        return e;
    return cs == cudaStreamCaptureStatusActive ? cudaEventRecordWithFlags(ev, st, cudaEventRecordExternal)
                                               : cudaEventRecord(ev, st);
}

// one PCG iteration; with timing on, `slot` selects the 4 events that
// bracket its SpMV and its preconditioner apply. ord: in PCG order (MAS)
static void pcg_iteration(b2s_solver* s, int kind, bool ord, double* x, int slot)
{
    PcgState&     P  = s->pcg;
    const Matrix& A  = ord ? P.ord.A : s->A;
    cudaStream_t  st = s->stream;
    const int64_t n  = 3 * (int64_t)A.nb;
    cudaEvent_t*  ev = s->timing ? &s->iter_events[(size_t)slot * 4] : nullptr;
    if(ev)
        B2S_CUDA(record_timing_event(ev[0], st));
    spmv_f64_launch(s, A, P.p.data(), P.Ap.data(), P.red, &P.sc.data()->pAp, &P.sc.data()->converged);
    if(ev)
        B2S_CUDA(record_timing_event(ev[1], st));
    if(ord)
        update_restrict_launch<double, 3, true>(s, kind, P.sc.data(), x, P.p.data(), P.r.data(), P.Ap.data());
    else
    {
        k_update_xr<<<vec_grid(n), VEC_BLOCK, 0, st>>>(n, P.sc.data(), x, P.p.data(), P.r.data(), P.Ap.data());
        B2S_CHECK_LAUNCH();
    }
    if(ev)
        B2S_CUDA(record_timing_event(ev[2], st));
    if(ord)
        precond_launch_ord<double, 3>(s, kind, false, P.r.data(), P.z.data(), P.sc.data(), P.red);
    else
        precond_launch(s, kind, P.r.data(), P.z.data(), P.sc.data(), P.red);
    if(ev)
        B2S_CUDA(record_timing_event(ev[3], st));
    k_update_p<<<vec_grid(n), VEC_BLOCK, 0, st>>>(n, P.sc.data(), P.z.data(), P.p.data());
    B2S_CHECK_LAUNCH();
}

// The loop's scalars and the device's error bits to the host, in one wait.
// Throws when a wait on the device has run out (the one-launch loop then leaves
// the scalars as they were) or when the iterations launched since `iter_before`
// did nothing: the host's loop ends with every launch that does not advance.
static void read_scalars(b2s_solver* s, long long iter_before)
{
    PcgState& P = s->pcg;
    k_scalars_out<<<1, 1, 0, s->stream>>>(P.sc.data(), s->dev_err.data(), &s->host->sc, &s->host->back);
    B2S_CHECK_LAUNCH();
    B2S_CUDA(cudaStreamSynchronize(s->stream));
    raise_device_errors(s->host->back.err);
    B2S_REQUIRE(s->host->sc.converged != 0 || s->host->sc.iter > iter_before, B2S_ERR_CUDA, "the PCG made no progress");
}

static void ensure_iter_events(b2s_solver* s, int ci)
{
    while((int)s->iter_events.size() < 4 * ci)
    {
        cudaEvent_t e;
        B2S_CUDA(cudaEventCreate(&e));
        s->iter_events.push_back(e);
    }
}

void pcg_solve(b2s_solver* s, const double* b, double* x, const b2s_pcg_options& o, b2s_pcg_stats& st_out)
{
    B2S_REQUIRE(s->A.valid, B2S_ERR_STATE, "b2s_pcg before b2s_assemble");
    B2S_REQUIRE(s->precond_kind >= 0, B2S_ERR_STATE, "b2s_pcg before b2s_precond_assemble");
    B2S_REQUIRE(o.precision == B2S_PRECISION_FP64 || o.precision == B2S_PRECISION_MIXED, B2S_ERR_ARGUMENT,
                "unknown precision");
    if(o.precision == B2S_PRECISION_MIXED)
    {
        pcg_solve_mixed(s, b, x, o, st_out);
        return;
    }
    B2S_REQUIRE(o.tol > 0.0 && std::isfinite(o.tol), B2S_ERR_ARGUMENT, "tolerance must be positive");
    B2S_REQUIRE(o.stop_rule == B2S_STOP_RZ || o.stop_rule == B2S_STOP_RELRES, B2S_ERR_ARGUMENT, "unknown stop rule");
    cudaStream_t  st = s->stream;
    PcgState&     P  = s->pcg;
    const int64_t n0 = 3 * (int64_t)s->A.nb;  // b and x
    std::memset(&st_out, 0, sizeof(st_out));
    if(n0 == 0)
    {
        st_out.converged = 1;
        return;
    }
    // with the MAS the recursion runs in its slot order (see PcgOrder)
    int  kind      = s->precond_kind;
    bool use_graph = o.use_graph && st != nullptr;
    auto room      = [&](bool in_order)
    {
        Matrix&       M = in_order ? P.ord.A : s->A;
        const int64_t m = 3 * (int64_t)M.nb;
        for(DBuf<double>* d : {&P.r, &P.z, &P.p, &P.Ap})
            d->resize(m, 1.1);
        P.tmp.resize(n0, 1.1);
        if(in_order)
            P.xs.resize(m, 1.1);
        P.sc.resize(1);
        ensure_reduction(s, P.red, std::max(spmv_grid(M.nnz), reduction_grid()), 2);
        ensure_reduction(s, s->red, reduction_grid(), 2);  // the largest grid: the sums below run over rows and over entries
        device_error_flag(s);  // allocated before any graph capture
        s->dot_out.resize(4);
        if(!use_graph || s->timing || !pcg_small_fits(s, M, kind, in_order, false))
            M.trank.resize(M.stride, 1.2);  // filled when the steps are prepared
    };
    const bool ord = kind == B2S_PRECOND_MAS && s->mas.initialized && try_order(s, false, room);
    if(!ord)
        room(false);
    const PcgOrder& O  = P.ord;
    const Matrix&   A  = ord ? O.A : s->A;
    const int64_t   n  = 3 * (int64_t)A.nb;         // the recursion's vectors
    double*         xi = ord ? P.xs.data() : x;  // the iterate
    const int ci = o.check_interval > 0 ? o.check_interval : 1;
    const int64_t max_iter = o.max_iter > 0 ? o.max_iter : std::max<int64_t>(2 * n0, 1);

    // r = b - A x (x0 = 0: r = b), z = P r
    auto residual = [&](bool zero)
    {
        if(!zero)
            spmv_f64(s, s->A, x, P.tmp.data(), nullptr);
        if(ord)
            k_residual_ord<double, 3><<<vec_grid(A.nb), VEC_BLOCK, 0, st>>>(A.nb, O.row_of.data(), b,
                                                                            zero ? nullptr : P.tmp.data(), P.r.data());
        else if(!zero)
            k_residual<<<vec_grid(n), VEC_BLOCK, 0, st>>>(n, b, P.tmp.data(), P.r.data());
        else
        {
            B2S_CUDA(cudaMemcpyAsync(P.r.data(), b, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
            return;
        }
        B2S_CHECK_LAUNCH();
    };
    auto apply = [&](int k)
    {
        if(!ord)
        {
            precond_launch(s, k, P.r.data(), P.z.data(), nullptr, s->red);
            return;
        }
        if(k == B2S_PRECOND_MAS)
            update_restrict_launch<double, 3, false>(s, k, nullptr, nullptr, nullptr, P.r.data(), nullptr);
        precond_launch_ord<double, 3>(s, k, false, P.r.data(), P.z.data(), nullptr, s->red);
    };
    if(!o.x0_given)
        B2S_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * n0, st));
    residual(!o.x0_given);
    if(ord)
    {
        if(o.x0_given)
        {
            k_to_ord<<<vec_grid(A.nb), VEC_BLOCK, 0, st>>>(A.nb, O.row_of.data(), x, xi);
            B2S_CHECK_LAUNCH();
        }
        else
            B2S_CUDA(cudaMemsetAsync(xi, 0, sizeof(double) * n, st));
    }
    apply(kind);
    launch_dot(s, P.r.data(), P.z.data(), n, s->dot_out.data());
    launch_dot(s, P.r.data(), P.r.data(), n, s->dot_out.data() + 1);
    launch_dot(s, b, b, n0, s->dot_out.data() + 2);
    double h3[3];
    read_back(s, s->dot_out.data(), 3, h3);
    double rz0 = h3[0];
    const double rr0 = h3[1], bb = h3[2];
    B2S_REQUIRE(std::isfinite(rr0) && std::isfinite(bb), B2S_ERR_NUMERIC,
                "non-finite right-hand side or initial residual");
    bool bypass = false;
    if(kind != B2S_PRECOND_NONE && (rz0 < 0.0 || !std::isfinite(rz0)))
    {
        // PSD guard: the preconditioner's action is not SPD/finite -> plain CG
        bypass = true;
        kind   = B2S_PRECOND_NONE;
        B2S_CUDA(cudaMemcpyAsync(P.z.data(), P.r.data(), sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
        rz0 = rr0;
    }
    st_out.rz0      = rz0;
    st_out.bypassed = bypass ? 1 : 0;
    const double bnorm = std::sqrt(bb);

    auto true_residual = [&]() -> double
    {
        spmv_f64(s, s->A, x, P.tmp.data(), nullptr);
        k_res_norms<<<reduction_grid(n0), RED_BLOCK, 0, st>>>(n0, b, P.tmp.data(), s->red.partials.data(),
                                                            s->red.counter.data(), s->dot_out.data());
        B2S_CHECK_LAUNCH();
        double h2[2];
        read_back(s, s->dot_out.data(), 2, h2);
        return h2[1] > 0 ? std::sqrt(h2[0] / h2[1]) : 0.0;
    };

    if(rz0 == 0.0 || bb == 0.0)
    {
        st_out.converged = 1;
        st_out.rel_res   = true_residual();
        return;
    }

    // device scalars
    PcgScalars h{};
    h.rz        = rz0;
    h.rz_tol    = o.tol * std::fabs(rz0);
    h.rr_tol    = (o.tol * bnorm) * (o.tol * bnorm);
    h.stop_rule = o.stop_rule;
    h.max_iter  = max_iter;
    int64_t iter_total = 0, replacements = 0;
    bool    done = false;
    while(!done)
    {
        h.converged = 0;
        h.iter      = iter_total;
        h.iter_conv = 0;
        B2S_CUDA(cudaMemcpyAsync(P.sc.data(), &h, sizeof(h), cudaMemcpyHostToDevice, st));
        B2S_CUDA(cudaMemcpyAsync(P.p.data(), P.z.data(), sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
        B2S_CUDA(cudaMemsetAsync(P.Ap.data(), 0, sizeof(double) * n, st));

        // small systems: the whole loop in one launch
        bool small = use_graph && !s->timing && pcg_small_fits(s, A, kind, ord, false);
        if(s->timing)
            ensure_iter_events(s, ci);
        // else launch by launch, from a CUDA graph of `ci` iterations
        // (re-captured when anything it bakes in changes)
        auto prepare_steps = [&]()
        {
            ensure_tile_ranks(s, ord ? P.ord.A : s->A);
            if(!use_graph)
                return;
            GraphKey key{};
            key.ptrs[0] = xi;
            key.ptrs[1] = A.vals.data();
            key.ptrs[2] = A.rows.data();
            key.ptrs[3] = P.r.data();
            key.ptrs[4] = s->mas.inv.data();
            key.ptrs[5] = s->dinv.data();
            key.ptrs[6] = P.red.partials.data();
            key.ptrs[7] = s->mas.Z.data();
            key.ptrs[8] = A.cols.data();
            key.ptrs[9] = P.z.data();
            key.ptrs[10] = P.p.data();
            key.ptrs[11] = P.Ap.data();
            key.ptrs[12] = A.trank.data();
            key.ptrs[13] = O.row_of.data();
            key.ints[0] = A.nnz;
            key.ints[1] = A.nb;
            key.ints[2] = kind;
            key.ints[3] = ci;
            key.ints[4] = s->mas.initialized ? s->mas.total : -1;
            key.ints[5] = s->mas.generation * 2 + (s->timing ? 1 : 0);
            size_t hk = 1469598103934665603ull;
            const unsigned char* kb = reinterpret_cast<const unsigned char*>(&key);
            for(size_t q = 0; q < sizeof(key); ++q)
                hk = (hk ^ kb[q]) * 1099511628211ull;
            if(!P.graph || P.graph_key != hk)
            {
                if(P.graph)
                {
                    cudaGraphExecDestroy(P.graph);
                    P.graph = nullptr;
                }
                cudaGraph_t g = nullptr;
                const long long before = g_kernel_launches;
                B2S_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
                for(int it = 0; it < ci; ++it)
                    pcg_iteration(s, kind, ord, xi, it);
                B2S_CUDA(cudaStreamEndCapture(st, &g));
                P.graph_kernels = g_kernel_launches - before;
                g_kernel_launches = before;
                cudaError_t e = cudaGraphInstantiate(&P.graph, g, 0);
                cudaGraphDestroy(g);
                if(e != cudaSuccess)
                {
                    P.graph   = nullptr;
                    use_graph = false;
                    cudaGetLastError();
                }
                else
                    P.graph_key = hk;
            }
        };
        if(!small)
            prepare_steps();
        long long iter_before = h.iter;
        while(true)
        {
            if(small && !pcg_small_launch(s, A, kind, SMALL_LOOP, xi))
            {
                small = false;
                prepare_steps();
            }
            if(!small && use_graph)
            {
                B2S_CUDA(cudaGraphLaunch(P.graph, st));
                g_kernel_launches += P.graph_kernels;
            }
            else if(!small)
                for(int it = 0; it < ci; ++it)
                    pcg_iteration(s, kind, ord, xi, it);
            read_scalars(s, iter_before);
            if(s->timing)
            {
                // the iterations of this block that did work (the rest were frozen)
                const long long live = std::min<long long>(s->host->sc.iter - iter_before, ci);
                for(long long it = 0; it < live; ++it)
                {
                    float a = 0.f, c = 0.f;
                    B2S_CUDA(cudaEventElapsedTime(&a, s->iter_events[it * 4 + 0], s->iter_events[it * 4 + 1]));
                    B2S_CUDA(cudaEventElapsedTime(&c, s->iter_events[it * 4 + 2], s->iter_events[it * 4 + 3]));
                    s->timers.spmv_ms += a;
                    s->timers.spmv_launches += 1;
                    s->timers.precond_apply_ms += c;
                    s->timers.precond_apply_launches += 1;
                }
            }
            iter_before = s->host->sc.iter;
            if(s->host->sc.converged != 0)
                break;
        }
        const PcgScalars r = s->host->sc;
        iter_total         = r.iter;
        if(ord)
        {
            k_from_ord<<<vec_grid(O.nb), VEC_BLOCK, 0, st>>>(O.nb, O.pos.data(), xi, x);
            B2S_CHECK_LAUNCH();
        }
        if(r.converged == 3)
            throw Error(B2S_ERR_NUMERIC, "PCG breakdown: r.z became non-finite at iteration " + std::to_string(r.iter));
        st_out.iterations_exact = r.converged == 1 ? r.iter_conv : r.iter;
        st_out.converged        = r.converged == 1 ? 1 : 0;
        st_out.rel_res          = true_residual();
        done = true;
        if(r.converged == 1 && o.stop_rule == B2S_STOP_RELRES && st_out.rel_res > o.tol && replacements < 8
           && iter_total < max_iter - 1)
        {
            // the recursive residual drifted from b - A x: replace it and continue
            ++replacements;
            residual(false);
            apply(kind);
            launch_dot(s, P.r.data(), P.z.data(), n, s->dot_out.data());
            read_back(s, s->dot_out.data(), 1, &h.rz);
            done = false;
        }
    }
    st_out.replacements = replacements;
    check_device_errors(s);
    if(st_out.converged)
        st_out.iterations = ci > 1 ? std::min<int64_t>(((st_out.iterations_exact + ci - 1) / ci) * ci, max_iter)
                                   : st_out.iterations_exact;
    else
        st_out.iterations = max_iter;
}

// ---------------------------------------------------------------------------
// mixed precision PCG
// ---------------------------------------------------------------------------
void drop_graphs(b2s_solver* s)
{
    if(s->pcg.graph)
        cudaGraphExecDestroy(s->pcg.graph);
    if(s->pcg.graph_mixed)
        cudaGraphExecDestroy(s->pcg.graph_mixed);
    s->pcg.graph       = nullptr;
    s->pcg.graph_mixed = nullptr;
}

// storage of the MAS inverses in the mixed path: BF16 diagonal-scaled
// (default) or FP32, from B2S_MIXED_MAS_INVERSE=bf16|fp32, read once
static bool mixed_inverse_bf16()
{
    static const bool v = []
    {
        const char* e = std::getenv("B2S_MIXED_MAS_INVERSE");
        return !(e && std::string(e) == "fp32");
    }();
    return v;
}

// z = P r on FP32 vectors (MAS with BF16 inverses), optionally fused with the
// iteration's dots and scalar update
static void precond_launch_f32(b2s_solver* s, int kind, const float* r, float* z, PcgScalars* sc, Reduction& red)
{
    const int32_t nb = s->A.nb;
    if(nb == 0)
        return;
    if(kind == B2S_PRECOND_MAS)
        mas_apply_levels_f32(s, r, sc ? &sc->converged : nullptr, mixed_inverse_bf16());
    const int grid = reduction_grid(nb);
    ensure_reduction(s, red, grid, 2);
    k_precond_finish<float, 4, false><<<grid, RED_BLOCK, 0, s->stream>>>(nb, kind, mas_view(s), s->dinv.data(), r, z, sc,
                                                               red.partials.data(), red.counter.data());
    B2S_CHECK_LAUNCH();
}

static void ensure_bf16_inverses(b2s_solver* s)
{
    if(s->precond_kind == B2S_PRECOND_MAS && s->mas.inv16_generation != s->precond_generation)
    {
        mas_pack_bf16(s);
        s->mas.inv16_generation = s->precond_generation;
    }
}

// the FP32 copy of the value planes the mixed PCG's SpMV reads (once per assembly)
static void ensure_f32_planes(b2s_solver* s)
{
    Matrix& A = s->A;
    if(A.vals32_generation == A.generation)
        return;
    A.vals32.resize((size_t)9 * A.stride, 1.2);
    k_planes_f32<<<vec_grid(9 * A.stride), VEC_BLOCK, 0, s->stream>>>(9 * A.stride, A.vals.data(), A.vals32.data());
    B2S_CHECK_LAUNCH();
    build_row_groups(s, A);
    A.vals32_generation = A.generation;
}

// y = A x as the mixed PCG computes it (FP32 planes and products, x.(A x) in
// FP64 into d_dot, device); x, y: 3 floats per node, padded around the product
void spmv_mixed(b2s_solver* s, const float* x, float* y, double* d_dot)
{
    Matrix&       A  = s->A;
    PcgState&     P  = s->pcg;
    const int32_t nb = A.nb;
    cudaStream_t  st = s->stream;
    ensure_f32_planes(s);
    ensure_reduction(s, P.red, std::max(spmv_grid(A.nnz), reduction_grid()), 2);
    P.p32.resize(4 * (size_t)nb, 1.1);
    P.Ap32.resize(4 * (size_t)nb, 1.1);
    k_pad4<<<vec_grid(nb), VEC_BLOCK, 0, st>>>(nb, x, P.p32.data(), P.Ap32.data());
    B2S_CHECK_LAUNCH();
    if(A.nnz == 0)
        B2S_CUDA(cudaMemsetAsync(d_dot, 0, sizeof(double), st));
    spmv_f32_launch(s, A, P.p32.data(), P.Ap32.data(), P.red, d_dot, nullptr);
    k_unpad4<<<vec_grid(nb), VEC_BLOCK, 0, st>>>(nb, P.Ap32.data(), y);
    B2S_CHECK_LAUNCH();
}

// the FP32 SpMV (with its fused dot) launched back to back on the solver's
// stream, events around the batch: the kernel's average launch duration on
// the assembled matrix (the padded vectors' values do not change its work)
double spmv_mixed_timing(b2s_solver* s, int launches)
{
    Matrix&       A  = s->A;
    PcgState&     P  = s->pcg;
    const int32_t nb = A.nb;
    cudaStream_t  st = s->stream;
    B2S_REQUIRE(launches > 0, B2S_ERR_ARGUMENT, "launch count must be positive");
    ensure_f32_planes(s);
    ensure_reduction(s, P.red, std::max(spmv_grid(A.nnz), reduction_grid()), 2);
    P.p32.resize(4 * (size_t)nb, 1.1);
    P.Ap32.resize(4 * (size_t)nb, 1.1);
    s->dot_out.resize(4);
    B2S_CUDA(cudaMemsetAsync(P.p32.data(), 0, sizeof(float) * 4 * (size_t)nb, st));
    B2S_CUDA(cudaMemsetAsync(P.Ap32.data(), 0, sizeof(float) * 4 * (size_t)nb, st));
    spmv_f32_launch(s, A, P.p32.data(), P.Ap32.data(), P.red, s->dot_out.data(), nullptr);  // warm-up
    cudaEvent_t e0, e1;
    B2S_CUDA(cudaEventCreate(&e0));
    B2S_CUDA(cudaEventCreate(&e1));
    B2S_CUDA(cudaEventRecord(e0, st));
    for(int i = 0; i < launches; ++i)
        spmv_f32_launch(s, A, P.p32.data(), P.Ap32.data(), P.red, s->dot_out.data(), nullptr);
    B2S_CUDA(cudaEventRecord(e1, st));
    B2S_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    B2S_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    B2S_CUDA(cudaEventDestroy(e0));
    B2S_CUDA(cudaEventDestroy(e1));
    return (double)ms / launches;
}

// r, z: 3 floats per node (the ABI's layout), padded around the apply
void precond_apply_mixed(b2s_solver* s, const float* r, float* z)
{
    B2S_REQUIRE(s->precond_kind >= 0, B2S_ERR_STATE, "precond_apply before b2s_precond_assemble");
    ensure_bf16_inverses(s);
    ensure_reduction(s, s->red, reduction_grid(), 2);
    const int32_t nb = s->A.nb;
    PcgState&     P  = s->pcg;
    P.r32.resize(4 * (size_t)nb, 1.1);
    P.z32.resize(4 * (size_t)nb, 1.1);
    k_pad4<<<vec_grid(nb), VEC_BLOCK, 0, s->stream>>>(nb, r, P.r32.data(), nullptr);
    B2S_CHECK_LAUNCH();
    precond_launch_f32(s, s->precond_kind, P.r32.data(), P.z32.data(), nullptr, s->red);
    k_unpad4<<<vec_grid(nb), VEC_BLOCK, 0, s->stream>>>(nb, P.z32.data(), z);
    B2S_CHECK_LAUNCH();
    read_back(s, nullptr, 0, nullptr);
}

static void pcg_iteration_mixed(b2s_solver* s, int kind, bool ord, double* x, int slot)
{
    PcgState&     P  = s->pcg;
    const Matrix& A  = ord ? P.ord.A : s->A;
    cudaStream_t  st = s->stream;
    const int32_t nb = A.nb;
    cudaEvent_t*  ev = s->timing ? &s->iter_events[(size_t)slot * 4] : nullptr;
    if(ev)
        B2S_CUDA(record_timing_event(ev[0], st));
    spmv_f32_launch(s, A, P.p32.data(), P.Ap32.data(), P.red, &P.sc.data()->pAp, &P.sc.data()->converged);
    if(ev)
        B2S_CUDA(record_timing_event(ev[1], st));
    if(ord)
        update_restrict_launch<float, 4, true>(s, kind, P.sc.data(), x, P.p32.data(), P.r32.data(), P.Ap32.data());
    else
    {
        k_update_xr_mixed4<<<vec_grid(nb), VEC_BLOCK, 0, st>>>(nb, P.sc.data(), x, P.p32.data(), P.r32.data(),
                                                               P.Ap32.data());
        B2S_CHECK_LAUNCH();
    }
    if(ev)
        B2S_CUDA(record_timing_event(ev[2], st));
    if(ord)
        precond_launch_ord<float, 4>(s, kind, mixed_inverse_bf16(), P.r32.data(), P.z32.data(), P.sc.data(), P.red);
    else
        precond_launch_f32(s, kind, P.r32.data(), P.z32.data(), P.sc.data(), P.red);
    if(ev)
        B2S_CUDA(record_timing_event(ev[3], st));
    k_update_p_mixed4<<<vec_grid(nb), VEC_BLOCK, 0, st>>>(nb, P.sc.data(), P.z32.data(), P.p32.data(),
                                                         P.Ap32.data());
    B2S_CHECK_LAUNCH();
}

// Mixed precision: the matrix in FP32 (planes converted once per assembly),
// r, z, p, Ap in FP32, the solution x and every scalar (alpha, beta, r.z,
// p.Ap, r.r) in FP64, MAS inverses as BF16 of the diagonal-scaled inverse
// with FP32 accumulation. Every `replace_every` iterations the recursive
// residual is replaced by b - A x computed in FP64 with the FP64 matrix
// (p, z and r.z are kept: a reliable update); the stop is always confirmed
// by the FP64 residual, and a stop the FP64 residual does not confirm
// continues from the true residual (with p = z).
void pcg_solve_mixed(b2s_solver* s, const double* b, double* x, const b2s_pcg_options& o, b2s_pcg_stats& st_out)
{
    cudaStream_t st = s->stream;
    PcgState&    P  = s->pcg;
    const int64_t n = 3 * (int64_t)s->A.nb;  // b and x
    std::memset(&st_out, 0, sizeof(st_out));
    if(n == 0)
    {
        st_out.converged = 1;
        return;
    }
    // FP32 matrix planes (in the MAS slot order with the MAS, see PcgOrder) and
    // BF16 inverses: once per assembly / build
    auto room = [&](bool in_order)
    {
        if(!in_order)
            ensure_f32_planes(s);
        ensure_bf16_inverses(s);
        const Matrix& M = in_order ? P.ord.A : s->A;
        for(DBuf<float>* d : {&P.r32, &P.z32, &P.p32, &P.Ap32})
            d->resize(4 * (size_t)M.nb, 1.1);
        P.tmp.resize(n, 1.1);
        if(in_order)
            P.xs.resize(3 * (size_t)M.nb, 1.1);
        P.sc.resize(1);
        ensure_reduction(s, P.red, std::max(spmv_grid(M.nnz), reduction_grid()), 2);
        ensure_reduction(s, s->red, reduction_grid(), 2);
        device_error_flag(s);
        s->dot_out.resize(4);
    };
    const bool ord = s->precond_kind == B2S_PRECOND_MAS && s->mas.initialized && try_order(s, true, room);
    if(!ord)
        room(false);
    const PcgOrder& O  = P.ord;
    const Matrix&   A  = ord ? O.A : s->A;
    const int32_t   nb = A.nb;                      // the recursion's rows
    const int64_t   n4 = 4 * (int64_t)nb;           // padded FP32 vectors
    double*         xi = ord ? P.xs.data() : x;  // the iterate
    const int     ci       = o.check_interval > 0 ? o.check_interval : 1;
    const int64_t max_iter = o.max_iter > 0 ? o.max_iter : std::max<int64_t>(2 * n, 1);
    int           kind     = s->precond_kind;

    // r = b - A x (FP64; x0 = 0: r = b), stored FP32
    auto residual = [&](bool zero)
    {
        if(!zero)
            spmv_f64(s, s->A, x, P.tmp.data(), nullptr);
        if(ord)
            k_residual_ord<float, 4><<<vec_grid(nb), VEC_BLOCK, 0, st>>>(nb, O.row_of.data(), b,
                                                                         zero ? nullptr : P.tmp.data(), P.r32.data());
        else
        {
            if(zero)
                B2S_CUDA(cudaMemsetAsync(P.tmp.data(), 0, sizeof(double) * n, st));
            k_residual_f32<<<vec_grid(nb), VEC_BLOCK, 0, st>>>(nb, b, P.tmp.data(), P.r32.data());
        }
        B2S_CHECK_LAUNCH();
    };
    auto store_x = [&]()
    {
        if(!ord)
            return;
        k_from_ord<<<vec_grid(O.nb), VEC_BLOCK, 0, st>>>(O.nb, O.pos.data(), xi, x);
        B2S_CHECK_LAUNCH();
    };
    if(!o.x0_given)
        B2S_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * n, st));
    residual(!o.x0_given);
    if(ord)
    {
        if(o.x0_given)
        {
            k_to_ord<<<vec_grid(nb), VEC_BLOCK, 0, st>>>(nb, O.row_of.data(), x, xi);
            B2S_CHECK_LAUNCH();
        }
        else
            B2S_CUDA(cudaMemsetAsync(xi, 0, sizeof(double) * 3 * (size_t)nb, st));
    }

    double bb = 0.0;  // b.b (dot_out[2])
    auto restart_from_r = [&](int k) -> double
    {
        // z = P r, p = z; returns r.z (FP64 sum); also leaves r.r in dot_out[1]
        if(ord)
        {
            if(k == B2S_PRECOND_MAS)
                update_restrict_launch<float, 4, false>(s, k, nullptr, nullptr, nullptr, P.r32.data(), nullptr);
            precond_launch_ord<float, 4>(s, k, mixed_inverse_bf16(), P.r32.data(), P.z32.data(), nullptr, s->red);
        }
        else
            precond_launch_f32(s, k, P.r32.data(), P.z32.data(), nullptr, s->red);
        k_dot2_f32<<<reduction_grid(n4), RED_BLOCK, 0, st>>>(n4, P.r32.data(), P.z32.data(), s->red.partials.data(),
                                                            s->red.counter.data(), s->dot_out.data());
        B2S_CHECK_LAUNCH();
        B2S_CUDA(cudaMemcpyAsync(P.p32.data(), P.z32.data(), sizeof(float) * n4, cudaMemcpyDeviceToDevice, st));
        double h3[3];
        read_back(s, s->dot_out.data(), 3, h3);
        bb = h3[2];
        return h3[0];
    };
    launch_dot(s, b, b, n, s->dot_out.data() + 2);
    double rz0 = restart_from_r(kind);
    B2S_REQUIRE(std::isfinite(bb), B2S_ERR_NUMERIC, "non-finite right-hand side");
    bool bypass = false;
    if(kind != B2S_PRECOND_NONE && (rz0 < 0.0 || !std::isfinite(rz0)))
    {
        bypass = true;  // PSD guard: plain CG
        kind   = B2S_PRECOND_NONE;
        rz0    = restart_from_r(kind);
    }
    st_out.rz0      = rz0;
    st_out.bypassed = bypass ? 1 : 0;
    const double bnorm = std::sqrt(bb);
    auto true_residual = [&]() -> double
    {
        spmv_f64(s, s->A, x, P.tmp.data(), nullptr);
        k_res_norms<<<reduction_grid(n), RED_BLOCK, 0, st>>>(n, b, P.tmp.data(), s->red.partials.data(),
                                                            s->red.counter.data(), s->dot_out.data());
        B2S_CHECK_LAUNCH();
        double h2[2];
        read_back(s, s->dot_out.data(), 2, h2);
        return h2[1] > 0 ? std::sqrt(h2[0] / h2[1]) : 0.0;
    };
    if(rz0 == 0.0 || bb == 0.0)
    {
        st_out.converged = 1;
        st_out.rel_res   = true_residual();
        return;
    }

    PcgScalars h{};
    h.rz        = rz0;
    h.rz_tol    = o.tol * std::fabs(rz0);
    h.rr_tol    = (o.tol * bnorm) * (o.tol * bnorm);
    h.stop_rule = o.stop_rule;
    h.max_iter  = max_iter;
    int64_t iter_total = 0, replacements = 0, last_replace = 0;
    bool    done = false;
    while(!done)
    {
        h.converged = 0;
        h.iter      = iter_total;
        h.iter_conv = 0;
        B2S_CUDA(cudaMemcpyAsync(P.sc.data(), &h, sizeof(h), cudaMemcpyHostToDevice, st));
        B2S_CUDA(cudaMemsetAsync(P.Ap32.data(), 0, sizeof(float) * n4, st));
        bool use_graph = o.use_graph && st != nullptr;
        // small systems: the loop in one launch, up to the next replacement
        bool small = use_graph && !s->timing && (kind != B2S_PRECOND_MAS || mixed_inverse_bf16())
                     && pcg_small_fits(s, A, kind, ord, true);
        if(s->timing)
            ensure_iter_events(s, ci);
        // else launch by launch (graph as in pcg_solve)
        auto prepare_steps = [&]()
        {
            if(!use_graph)
                return;
            const void*   ptrs[15] = {xi,         A.vals32.data(), A.rows.data(),     P.r32.data(),
                                      s->mas.inv16.data(), s->dinv.data(), P.red.partials.data(), s->mas.Z.data(),
                                      A.cols.data(), P.p32.data(), P.Ap32.data(), P.z32.data(),
                                      A.grp_row.data(), A.grp_mask.data(), O.row_of.data()};
            const int64_t ints[6]  = {A.nnz, A.nb, kind, ci, s->mas.initialized ? s->mas.total : -1,
                                      s->mas.generation * 2 + (s->timing ? 1 : 0)};
            size_t hk = 1469598103934665603ull;
            for(const void* q : ptrs)
                hk = (hk ^ (size_t)q) * 1099511628211ull;
            for(int64_t q : ints)
                hk = (hk ^ (size_t)q) * 1099511628211ull;
            if(!P.graph_mixed || P.graph_mixed_key != hk)
            {
                if(P.graph_mixed)
                {
                    cudaGraphExecDestroy(P.graph_mixed);
                    P.graph_mixed = nullptr;
                }
                cudaGraph_t     g      = nullptr;
                const long long before = g_kernel_launches;
                B2S_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
                for(int it = 0; it < ci; ++it)
                    pcg_iteration_mixed(s, kind, ord, xi, it);
                B2S_CUDA(cudaStreamEndCapture(st, &g));
                P.graph_mixed_kernels = g_kernel_launches - before;
                g_kernel_launches     = before;
                cudaError_t e         = cudaGraphInstantiate(&P.graph_mixed, g, 0);
                cudaGraphDestroy(g);
                if(e != cudaSuccess)
                {
                    P.graph_mixed = nullptr;
                    use_graph     = false;
                    cudaGetLastError();
                }
                else
                    P.graph_mixed_key = hk;
            }
        };
        if(!small)
            prepare_steps();
        long long iter_before = h.iter;
        while(true)
        {
            if(small)
            {
                // whole blocks of check_interval, as the replacements are counted
                const long long due = o.replace_every > 0 ? std::max<long long>(last_replace + o.replace_every - iter_before, 1) :
                                                            SMALL_LOOP;
                if(!pcg_small_launch_f32(s, A, kind, std::min<long long>((due + ci - 1) / ci * ci, SMALL_LOOP), xi))
                {
                    small = false;
                    prepare_steps();
                }
            }
            if(!small && use_graph)
            {
                B2S_CUDA(cudaGraphLaunch(P.graph_mixed, st));
                g_kernel_launches += P.graph_mixed_kernels;
            }
            else if(!small)
                for(int it = 0; it < ci; ++it)
                    pcg_iteration_mixed(s, kind, ord, xi, it);
            read_scalars(s, iter_before);
            if(s->timing)
            {
                const long long live = std::min<long long>(s->host->sc.iter - iter_before, ci);
                for(long long it = 0; it < live; ++it)
                {
                    float a = 0.f, c = 0.f;
                    B2S_CUDA(cudaEventElapsedTime(&a, s->iter_events[it * 4 + 0], s->iter_events[it * 4 + 1]));
                    B2S_CUDA(cudaEventElapsedTime(&c, s->iter_events[it * 4 + 2], s->iter_events[it * 4 + 3]));
                    s->timers.spmv_ms += a;
                    s->timers.spmv_launches += 1;
                    s->timers.precond_apply_ms += c;
                    s->timers.precond_apply_launches += 1;
                }
            }
            iter_before = s->host->sc.iter;
            if(s->host->sc.converged != 0)
                break;
            if(o.replace_every > 0 && s->host->sc.iter - last_replace >= o.replace_every)
            {
                // reliable update: FP64 residual of the FP64 iterate, p and r.z kept
                store_x();
                residual(false);
                ++replacements;
                last_replace = s->host->sc.iter;
            }
        }
        const PcgScalars r = s->host->sc;
        iter_total         = r.iter;
        store_x();
        if(r.converged == 3)
            throw Error(B2S_ERR_NUMERIC, "mixed PCG breakdown: r.z non-finite at iteration " + std::to_string(r.iter));
        st_out.iterations_exact = r.converged == 1 ? r.iter_conv : r.iter;
        st_out.converged        = r.converged == 1 ? 1 : 0;
        st_out.rel_res          = true_residual();
        done                    = true;
        const bool verified = o.stop_rule != B2S_STOP_RELRES || st_out.rel_res <= o.tol;
        if(r.converged == 1 && !verified && replacements < 64 && iter_total < max_iter - 1)
        {
            // the FP32 recursion claimed a stop the FP64 residual does not
            // confirm: continue from the true residual
            residual(false);
            ++replacements;
            last_replace = iter_total;
            h.rz         = restart_from_r(kind);
            done         = false;
        }
        else if(r.converged == 1 && !verified)
            st_out.converged = 0;
    }
    st_out.replacements = replacements;
    check_device_errors(s);
    if(st_out.converged)
        st_out.iterations = ci > 1 ? std::min<int64_t>(((st_out.iterations_exact + ci - 1) / ci) * ci, max_iter)
                                   : st_out.iterations_exact;
    else
        st_out.iterations = max_iter;
}
}  // namespace b2s
