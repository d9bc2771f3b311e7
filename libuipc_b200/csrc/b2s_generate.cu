// Newton systems of tet meshes generated on the GPU (include/b200gen.h):
// kinetic + stable Neo-Hookean (PSD-projected) + ground barrier + Dirichlet
// vertices, straight into device triplet buffers. The arithmetic restates the
// host generator (csrc/scene/scene_gen.cpp: snh_derivatives, the kinetic /
// elastic / ground / fixed passes) per element, with the closed-form PSD
// projection of b2s_snh.cuh in place of its 9x9 Jacobi; results agree with it
// to rounding.
#include "b2s_fixed_reduce.cuh"
#include "b2s_internal.cuh"
#include "b2s_snh.cuh"

#include "../../include/b200gen.h"

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

namespace
{
thread_local std::string g_gen_err;

constexpr int GEN_BLOCK = 128;

struct DevMesh
{
    int32_t nv = 0, nt = 0, ng = 0;
    b2s::DBuf<int32_t> tets;      // [nt*4]
    b2s::DBuf<double>  vol;       // [nt]
    b2s::DBuf<double>  grad;      // [nt*12] shape gradients g_q[b]
    b2s::DBuf<double>  mass;      // [nv]
    b2s::DBuf<uint8_t> fixed;     // [nv] (empty: none)
    b2s::DBuf<int32_t> vt_start;  // [nv+1] incident (tet, corner) pairs by tet index
    b2s::DBuf<int32_t> vt_list;   // [4 nt]: t * 4 + q
    b2s::DBuf<int32_t> ground;    // [ng]
    b2s::DBuf<double>  tet_g;     // [nt*12] per-tet gradient scratch
    b2gen_material     mat{};
    int                device = 0;
};

// a row-major 3x3 block of the pair (ra, rb) into slot k, upper orientation
__device__ __forceinline__ void write_block(int64_t k, int32_t ra, int32_t rb, const double* Hab, int32_t* rows,
                                            int32_t* cols, double* vals)
{
    const bool tp = ra > rb;
    rows[k]       = tp ? rb : ra;
    cols[k]       = tp ? ra : rb;
    double* V     = vals + k * 9;
    for(int p = 0; p < 3; ++p)
        for(int q = 0; q < 3; ++q)
            V[q * 3 + p] = tp ? Hab[q * 3 + p] : Hab[p * 3 + q];  // column-major
}

// ---- kernels -----------------------------------------------------------------
__global__ void k_rest(int nt, const double* __restrict__ X, const int32_t* __restrict__ tets, double rho,
                       double* __restrict__ vol, double* __restrict__ G)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if(t >= nt)
        return;
    const int32_t* T = tets + (int64_t)t * 4;
    double         e[3][3];
    for(int q = 0; q < 3; ++q)
        for(int a = 0; a < 3; ++a)
            e[q][a] = X[T[q + 1] * 3 + a] - X[T[0] * 3 + a];
    auto cross = [](const double* a, const double* b, double* c) {
        c[0] = a[1] * b[2] - a[2] * b[1];
        c[1] = a[2] * b[0] - a[0] * b[2];
        c[2] = a[0] * b[1] - a[1] * b[0];
    };
    double c12[3], c20[3], c01[3];
    cross(e[1], e[2], c12);
    cross(e[2], e[0], c20);
    cross(e[0], e[1], c01);
    const double det = e[0][0] * c12[0] + e[0][1] * c12[1] + e[0][2] * c12[2];
    vol[t]           = det / 6.0;
    double* g        = G + (int64_t)t * 12;
    for(int b = 0; b < 3; ++b)
    {
        const double r0 = c12[b] / det, r1 = c20[b] / det, r2 = c01[b] / det;
        g[3 + b] = r0;
        g[6 + b] = r1;
        g[9 + b] = r2;
        g[b]     = -(r0 + r1 + r2);
    }
}

// lumped masses, in tet order per vertex (the host generator's sum order)
__global__ void k_mass(int nv, const int32_t* __restrict__ vt_start, const int32_t* __restrict__ vt_list,
                       const double* __restrict__ vol, double rho, double* __restrict__ mass)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if(v >= nv)
        return;
    double m = 0.0;
    for(int e = vt_start[v]; e < vt_start[v + 1]; ++e)
        m += rho * vol[vt_list[e] >> 2] * 0.25;
    mass[v] = m;
}

// the block of vertex pair (i, j) after the Dirichlet rule: rows and columns
// of fixed vertices zero, the identity on their diagonal blocks
__device__ __forceinline__ void apply_fixed(bool fix, bool diag, double* H)
{
    if(!fix)
        return;
#pragma unroll
    for(int e = 0; e < 9; ++e)
        H[e] = (diag && e % 4 == 0) ? 1.0 : 0.0;
}

// slot k of a tet's ten upper blocks -> its vertex pair (q, r), q <= r
__device__ __forceinline__ int slot_q(int k) { return (0x3221110000ull >> (4 * k)) & 0xF; }
__device__ __forceinline__ int slot_r(int k) { return (0x3323213210ull >> (4 * k)) & 0xF; }

// One thread per tet: F, the stress for the gradient and the ten projected
// Hessian blocks (b2s_snh.cuh: closed form, everything in registers). Bound by
// the FP64 pipe and the 800 B of triplets written per tet. A 9x9 Jacobi per
// tet, its two 648-byte arrays in local memory, took the whole system of
// 480,000 tets 11.1 ms; with this kernel it takes 0.19 ms (2.1 TB/s). The
// blocks go through shared memory, five slots at a time, so that a warp's
// stores cover whole 360-byte runs: written thread by thread every 8-byte
// store of a warp would touch 32 sectors. 46 KB and at most 128 registers:
// four CTAs per SM. The Dirichlet rule is applied as the blocks are made, not
// in a pass over the written triplets.
constexpr int GEN_HALF = 5;             // slots staged together
constexpr int GEN_RUN  = 9 * GEN_HALF;  // their doubles per tet (odd: no bank conflicts)
__global__ void __launch_bounds__(GEN_BLOCK, 4) k_elastic(int nv, int nt, const int32_t* __restrict__ tets,
                                                          const double* __restrict__ vol,
                                                          const double* __restrict__ G, const double* __restrict__ x,
                                                          const uint8_t* __restrict__ fixed, double mu, double lambda,
                                                          double dt2, int32_t* rows, int32_t* cols, double* vals,
                                                          double* __restrict__ tet_g)
{
    __shared__ double s_val[GEN_BLOCK / 32][32 * GEN_RUN];
    __shared__ int4   s_tet[GEN_BLOCK];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int t0 = blockIdx.x * GEN_BLOCK + 32 * w;  // the warp's first tet
    if(t0 >= nt)
        return;
    const int     n    = min(32, nt - t0);  // its tets; the lanes past them repeat the last one
    const int     t    = t0 + min(lane, n - 1);
    const int4    T4   = reinterpret_cast<const int4*>(tets)[t];
    const int32_t T[4] = {T4.x, T4.y, T4.z, T4.w};
    s_tet[threadIdx.x] = T4;
    unsigned fx = 0;
    if(fixed)
#pragma unroll
        for(int q = 0; q < 4; ++q)
            fx |= fixed[T[q]] ? 1u << q : 0u;
    double g[4][3];
#pragma unroll
    for(int i = 0; i < 6; ++i)
    {
        const double2 d = reinterpret_cast<const double2*>(G + (int64_t)t * 12)[i];
        g[(2 * i) / 3][(2 * i) % 3]         = d.x;
        g[(2 * i + 1) / 3][(2 * i + 1) % 3] = d.y;
    }
    double F[9] = {0};
#pragma unroll
    for(int q = 0; q < 4; ++q)
#pragma unroll
        for(int a = 0; a < 3; ++a)
        {
            const double xa = x[(int64_t)T[q] * 3 + a];
#pragma unroll
            for(int b = 0; b < 3; ++b)
                F[a + 3 * b] += xa * g[q][b];
        }
    double               P[9];
    b2s::snh::Projected h;
    b2s::snh::derivatives(F, mu, lambda, vol[t] * dt2, P, h);
    if(lane < n)
    {
        double f[12];
#pragma unroll
        for(int i = 0; i < 12; ++i)
            f[i] = P[i % 3] * g[i / 3][0] + P[i % 3 + 3] * g[i / 3][1] + P[i % 3 + 6] * g[i / 3][2];
#pragma unroll
        for(int i = 0; i < 6; ++i)
            reinterpret_cast<double2*>(tet_g + (int64_t)t * 12)[i] = make_double2(f[2 * i], f[2 * i + 1]);
    }
    // the shape gradients in the V frame
#pragma unroll
    for(int q = 0; q < 4; ++q)
    {
        const double a = g[q][0], b = g[q][1], c = g[q][2];
#pragma unroll
        for(int i = 0; i < 3; ++i)
            g[q][i] = h.v[i][0] * a + h.v[i][1] * b + h.v[i][2] * c;
    }
    const int64_t slot0 = (int64_t)nv + (int64_t)t0 * 10;
#pragma unroll
    for(int half = 0; half < 2; ++half)
    {
        double* mine = s_val[w] + lane * GEN_RUN;
#pragma unroll
        for(int k = 0; k < GEN_HALF; ++k)
        {
            const int q = slot_q(GEN_HALF * half + k), r = slot_r(GEN_HALF * half + k);
            double    Hb[9];
            b2s::snh::block(h, g[q], g[r], Hb);
            if(q == r)  // exact symmetry of diagonal blocks
            {
#pragma unroll
                for(int a = 0; a < 3; ++a)
#pragma unroll
                    for(int c = a + 1; c < 3; ++c)
                        Hb[a * 3 + c] = Hb[c * 3 + a] = 0.5 * (Hb[a * 3 + c] + Hb[c * 3 + a]);
            }
            apply_fixed((fx >> q & 1u) || (fx >> r & 1u), T[q] == T[r], Hb);
            const bool tp = T[q] > T[r];
#pragma unroll
            for(int a = 0; a < 3; ++a)
#pragma unroll
                for(int c = 0; c < 3; ++c)
                    mine[9 * k + c * 3 + a] = tp ? Hb[c * 3 + a] : Hb[a * 3 + c];  // column-major, upper orientation
        }
        __syncwarp();
        double* V = vals + slot0 * 9 + half * GEN_RUN;
#pragma unroll 5
        for(int i = 0; i < GEN_RUN; ++i)
        {
            const int e = i * 32 + lane, tt = e / GEN_RUN;
            if(tt < n)
                V[(int64_t)tt * (2 * GEN_RUN) + (e - tt * GEN_RUN)] = s_val[w][e];
        }
        __syncwarp();
    }
    const int32_t* ids = reinterpret_cast<const int32_t*>(s_tet + 32 * w);
#pragma unroll
    for(int i = 0; i < 10; ++i)
    {
        const int e = i * 32 + lane, tt = e / 10, k = e - tt * 10;
        if(tt < n)
        {
            const int32_t va = ids[4 * tt + slot_q(k)], vb = ids[4 * tt + slot_r(k)];
            rows[slot0 + e]  = min(va, vb);
            cols[slot0 + e]  = max(va, vb);
        }
    }
}

// kinetic block and the gradient (kinetic, tets by index, ground) per vertex
__global__ void k_vertex(int nv, int nt, const double* __restrict__ mass, const double* __restrict__ x,
                         const double* __restrict__ xt, const int32_t* __restrict__ vt_start,
                         const int32_t* __restrict__ vt_list, const double* __restrict__ tet_g,
                         const uint8_t* __restrict__ fixed, int32_t* rows, int32_t* cols, double* vals,
                         double* __restrict__ grad)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if(v >= nv)
        return;
    const bool   fix  = fixed && fixed[v];
    const double m    = mass[v];
    double       H[9] = {m, 0, 0, 0, m, 0, 0, 0, m};
    apply_fixed(fix, true, H);
    write_block(v, v, v, H, rows, cols, vals);
    double g[3];
    for(int a = 0; a < 3; ++a)
        g[a] = m * (x[(int64_t)v * 3 + a] - xt[(int64_t)v * 3 + a]);
    for(int e = vt_start[v]; e < vt_start[v + 1]; ++e)
    {
        const int tq = vt_list[e];  // t * 4 + q
        for(int a = 0; a < 3; ++a)
            g[a] += tet_g[(int64_t)(tq >> 2) * 12 + (tq & 3) * 3 + a];
    }
    for(int a = 0; a < 3; ++a)
        grad[(int64_t)v * 3 + a] = fix ? 0.0 : g[a];
}

// ground barrier (normal +y) on the candidates: one diagonal block each
__global__ void k_ground(int nv, int nt, int ng, const int32_t* __restrict__ ground, const double* __restrict__ x,
                         const uint8_t* __restrict__ fixed, double ground_y, double dhat, double kappa, double dt2,
                         int32_t* rows, int32_t* cols, double* vals, double* __restrict__ grad)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= ng)
        return;
    const int32_t g   = ground[i];
    const bool    fix = fixed && fixed[g];
    const double  d   = x[(int64_t)g * 3 + 1] - ground_y;
    double        k   = 0.0, gy = 0.0;
    if(d < dhat)
    {
        const double D = d * d, Dh = dhat * dhat, tt = D - Dh, l = log(D / Dh);
        const double b1 = -2.0 * tt * l - tt * tt / D;
        const double b2 = -2.0 * l - 4.0 * tt / D + tt * tt / (D * D);
        k               = fmax(0.0, dt2 * kappa * (b2 * 4.0 * D + 2.0 * b1));
        gy              = dt2 * kappa * b1 * 2.0 * d;
    }
    double H[9] = {0, 0, 0, 0, k, 0, 0, 0, 0};
    apply_fixed(fix, true, H);
    write_block((int64_t)nv + (int64_t)nt * 10 + i, g, g, H, rows, cols, vals);
    // one candidate per vertex: the add keeps the order kinetic, tets, ground
    if(!fix)
        grad[(int64_t)g * 3 + 1] += gy;
}

int grid_of(int64_t n) { return (int)((n + GEN_BLOCK - 1) / GEN_BLOCK); }

// ---- energy and the ground's time of impact (the line search after the solve) ----
// per-term energies: kinetic 1/2 m |x - x_tilde|^2 per vertex, dt^2 vol Psi(F)
// per tet with Psi = mu/2 (|F|^2 - 3) - mu (J - 1) + lambda/2 (J - 1)^2 (the
// potential whose derivatives k_elastic writes), dt^2 kappa b(d^2) per ground
// candidate (infinite at or below the plane)
__global__ void k_energy_terms(int nv, int nt, int ng, const int32_t* __restrict__ tets, const double* __restrict__ vol,
                               const double* __restrict__ G, const double* __restrict__ mass,
                               const int32_t* __restrict__ ground, const double* __restrict__ x,
                               const double* __restrict__ xt, double mu, double lambda, double dt2, double ground_y,
                               double dhat, double kappa, double* __restrict__ e)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i < nv)
    {
        double d2 = 0.0;
        for(int a = 0; a < 3; ++a)
        {
            const double d = x[i * 3 + a] - xt[i * 3 + a];
            d2 += d * d;
        }
        e[i] = 0.5 * mass[i] * d2;
    }
    else if(i < (int64_t)nv + nt)
    {
        const int64_t  t  = i - nv;
        const int32_t* T  = tets + t * 4;
        const double*  Gs = G + t * 12;
        double         F[9] = {0};
        for(int q = 0; q < 4; ++q)
            for(int a = 0; a < 3; ++a)
                for(int b = 0; b < 3; ++b)
                    F[a + 3 * b] += x[T[q] * 3 + a] * Gs[q * 3 + b];
        const double J = F[0] * (F[4] * F[8] - F[7] * F[5]) - F[3] * (F[1] * F[8] - F[7] * F[2]) +
                         F[6] * (F[1] * F[5] - F[4] * F[2]);
        double f2 = 0.0;
        for(int k = 0; k < 9; ++k)
            f2 += F[k] * F[k];
        const double psi = 0.5 * mu * (f2 - 3.0) - mu * (J - 1.0) + 0.5 * lambda * (J - 1.0) * (J - 1.0);
        e[i]             = dt2 * vol[t] * psi;
    }
    else if(i < (int64_t)nv + nt + ng)
    {
        const int32_t g = ground[i - nv - nt];
        const double  d = x[(int64_t)g * 3 + 1] - ground_y;
        double        v = 0.0;
        if(!(d > 0.0))
            v = INFINITY;
        else if(d < dhat)
        {
            const double D = d * d, Dh = dhat * dhat, tt = D - Dh;
            v              = -dt2 * kappa * tt * tt * log(D / Dh);
        }
        e[i] = v;
    }
}

// time of impact with the ground plane (normal +y) of every candidate moving
// along d: (1 - eta) (y - ground_y) / (-d_y) when it moves down, else 1.1
__global__ void k_ground_toi(int ng, const int32_t* __restrict__ ground, const double* __restrict__ x,
                             const double* __restrict__ dx, double ground_y, double eta, double* __restrict__ toi)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= ng)
        return;
    const int32_t g = ground[i];
    const double  t = -dx[(int64_t)g * 3 + 1];  // approach speed along -normal
    double        v = 1.1;
    if(t > 0.0)
        v = (x[(int64_t)g * 3 + 1] - ground_y) / t * (1.0 - eta);
    toi[i] = v;
}
}  // namespace

struct b2gen_mesh : DevMesh
{
    b2s::DBuf<double> terms;  // per-term energies / times of impact
    b2s::DBuf<double> result;
};

extern "C" {

const char* b2gen_last_error(void) { return g_gen_err.c_str(); }

int b2gen_mesh_create(int device, int32_t n_verts, int32_t n_tets, const double* rest, const int32_t* tets,
                      const uint8_t* fixed, int32_t n_ground, const int32_t* ground, const b2gen_material* mat,
                      b2gen_mesh** out)
{
    try
    {
        if(!out || !rest || !tets || !mat || n_verts <= 0 || n_tets <= 0 || n_ground < 0 ||
           (n_ground > 0 && !ground))
            throw b2s::Error(B2S_ERR_ARGUMENT, "b2gen_mesh_create: bad arguments");
        if((int64_t)n_verts + 10ll * n_tets + n_ground > (int64_t)INT32_MAX)
            throw b2s::Error(B2S_ERR_ARGUMENT, "b2gen_mesh_create: too many triplets for 32-bit slots");
        for(int64_t i = 0; i < 4ll * n_tets; ++i)
            if(tets[i] < 0 || tets[i] >= n_verts)
                throw b2s::Error(B2S_ERR_ARGUMENT, "b2gen_mesh_create: tet vertex out of range");
        for(int32_t i = 0; i < n_ground; ++i)
            if(ground[i] < 0 || ground[i] >= n_verts)
                throw b2s::Error(B2S_ERR_ARGUMENT, "b2gen_mesh_create: ground vertex out of range");
        B2S_CUDA(cudaSetDevice(device));
        auto M    = new b2gen_mesh();
        M->device = device;
        M->nv     = n_verts;
        M->nt     = n_tets;
        M->ng     = n_ground;
        M->mat    = *mat;
        // vertex -> (tet, corner) incidence, by tet index
        std::vector<int32_t> start(n_verts + 1, 0), list(4 * (size_t)n_tets);
        for(int64_t i = 0; i < 4ll * n_tets; ++i)
            ++start[tets[i] + 1];
        for(int32_t v = 0; v < n_verts; ++v)
            start[v + 1] += start[v];
        std::vector<int32_t> fill(start.begin(), start.end() - 1);
        for(int32_t t = 0; t < n_tets; ++t)
            for(int q = 0; q < 4; ++q)
                list[fill[tets[4 * t + q]]++] = 4 * t + q;
        b2s::DBuf<double> X;
        X.resize((size_t)n_verts * 3);
        M->tets.resize(4 * (size_t)n_tets);
        M->vol.resize(n_tets);
        M->grad.resize(12 * (size_t)n_tets);
        M->mass.resize(n_verts);
        M->vt_start.resize(n_verts + 1);
        M->vt_list.resize(list.size());
        M->tet_g.resize(12 * (size_t)n_tets);
        B2S_CUDA(cudaMemcpy(X.data(), rest, X.bytes(), cudaMemcpyHostToDevice));
        B2S_CUDA(cudaMemcpy(M->tets.data(), tets, M->tets.bytes(), cudaMemcpyHostToDevice));
        B2S_CUDA(cudaMemcpy(M->vt_start.data(), start.data(), M->vt_start.bytes(), cudaMemcpyHostToDevice));
        B2S_CUDA(cudaMemcpy(M->vt_list.data(), list.data(), M->vt_list.bytes(), cudaMemcpyHostToDevice));
        if(fixed)
        {
            M->fixed.resize(n_verts);
            B2S_CUDA(cudaMemcpy(M->fixed.data(), fixed, n_verts, cudaMemcpyHostToDevice));
        }
        if(n_ground > 0)
        {
            M->ground.resize(n_ground);
            B2S_CUDA(cudaMemcpy(M->ground.data(), ground, sizeof(int32_t) * n_ground, cudaMemcpyHostToDevice));
        }
        k_rest<<<grid_of(n_tets), GEN_BLOCK>>>(n_tets, X.data(), M->tets.data(), mat->rho, M->vol.data(),
                                               M->grad.data());
        B2S_CHECK_LAUNCH();
        k_mass<<<grid_of(n_verts), GEN_BLOCK>>>(n_verts, M->vt_start.data(), M->vt_list.data(), M->vol.data(),
                                                mat->rho, M->mass.data());
        B2S_CHECK_LAUNCH();
        B2S_CUDA(cudaDeviceSynchronize());
        *out = M;
        return 0;
    }
    catch(const b2s::Error& e)
    {
        g_gen_err = e.what();
        return e.code;
    }
    catch(const std::exception& e)
    {
        g_gen_err = e.what();
        return B2S_ERR_CUDA;
    }
}

int b2gen_mesh_destroy(b2gen_mesh* m)
{
    delete m;
    return 0;
}

int64_t b2gen_num_triplets(const b2gen_mesh* m)
{
    return m ? (int64_t)m->nv + 10ll * m->nt + m->ng : -1;
}

int b2gen_system(b2gen_mesh* m, const double* d_x, const double* d_xtilde, int32_t* d_rows, int32_t* d_cols,
                 double* d_vals, double* d_grad, void* stream)
{
    try
    {
        if(!m || !d_x || !d_xtilde || !d_rows || !d_cols || !d_vals || !d_grad)
            throw b2s::Error(B2S_ERR_ARGUMENT, "b2gen_system: null argument");
        B2S_CUDA(cudaSetDevice(m->device));
        cudaStream_t      st  = static_cast<cudaStream_t>(stream);
        const b2gen_material& c = m->mat;
        const double      dt2 = c.dt * c.dt;
        const uint8_t*    fixed = m->fixed.size() > 0 ? m->fixed.data() : nullptr;  // Dirichlet rule in every pass
        k_elastic<<<grid_of(m->nt), GEN_BLOCK, 0, st>>>(m->nv, m->nt, m->tets.data(), m->vol.data(), m->grad.data(),
                                                        d_x, fixed, c.mu, c.lambda, dt2, d_rows, d_cols,
                                                        d_vals, m->tet_g.data());
        B2S_CHECK_LAUNCH();
        k_vertex<<<grid_of(m->nv), GEN_BLOCK, 0, st>>>(m->nv, m->nt, m->mass.data(), d_x, d_xtilde,
                                                       m->vt_start.data(), m->vt_list.data(), m->tet_g.data(), fixed,
                                                       d_rows, d_cols, d_vals, d_grad);
        B2S_CHECK_LAUNCH();
        if(m->ng > 0)
        {
            k_ground<<<grid_of(m->ng), GEN_BLOCK, 0, st>>>(m->nv, m->nt, m->ng, m->ground.data(), d_x, fixed,
                                                           c.ground_y, c.dhat, c.kappa, dt2, d_rows, d_cols, d_vals,
                                                           d_grad);
            B2S_CHECK_LAUNCH();
        }
        B2S_CUDA(cudaStreamSynchronize(st));
        return 0;
    }
    catch(const b2s::Error& e)
    {
        g_gen_err = e.what();
        return e.code;
    }
    catch(const std::exception& e)
    {
        g_gen_err = e.what();
        return B2S_ERR_CUDA;
    }
}

int b2gen_energy(b2gen_mesh* m, const double* d_x, const double* d_xtilde, double* h_energy, void* stream)
{
    try
    {
        if(!m || !d_x || !d_xtilde || !h_energy)
            throw b2s::Error(B2S_ERR_ARGUMENT, "b2gen_energy: null argument");
        B2S_CUDA(cudaSetDevice(m->device));
        cudaStream_t          st = static_cast<cudaStream_t>(stream);
        const b2gen_material& c  = m->mat;
        const int64_t         n  = (int64_t)m->nv + m->nt + m->ng;
        m->terms.resize(n);
        m->result.resize(1);
        k_energy_terms<<<grid_of(n), GEN_BLOCK, 0, st>>>(m->nv, m->nt, m->ng, m->tets.data(), m->vol.data(),
                                                         m->grad.data(), m->mass.data(),
                                                         m->ng ? m->ground.data() : nullptr, d_x, d_xtilde, c.mu,
                                                         c.lambda, c.dt * c.dt, c.ground_y, c.dhat, c.kappa,
                                                         m->terms.data());
        B2S_CHECK_LAUNCH();
        b2s::k_fixed_reduce<<<1, b2s::SUM_THREADS, 0, st>>>(n, m->terms.data(), 0, m->result.data());
        B2S_CHECK_LAUNCH();
        B2S_CUDA(cudaMemcpyAsync(h_energy, m->result.data(), sizeof(double), cudaMemcpyDeviceToHost, st));
        B2S_CUDA(cudaStreamSynchronize(st));
        return 0;
    }
    catch(const b2s::Error& e)
    {
        g_gen_err = e.what();
        return e.code;
    }
    catch(const std::exception& e)
    {
        g_gen_err = e.what();
        return B2S_ERR_CUDA;
    }
}

int b2gen_ground_toi(b2gen_mesh* m, const double* d_x, const double* d_dx, double* h_alpha, void* stream)
{
    try
    {
        if(!m || !d_x || !d_dx || !h_alpha)
            throw b2s::Error(B2S_ERR_ARGUMENT, "b2gen_ground_toi: null argument");
        *h_alpha = 1.0;
        if(m->ng == 0)
            return 0;
        B2S_CUDA(cudaSetDevice(m->device));
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        m->terms.resize(m->ng);
        m->result.resize(1);
        k_ground_toi<<<grid_of(m->ng), GEN_BLOCK, 0, st>>>(m->ng, m->ground.data(), d_x, d_dx, m->mat.ground_y, 0.1,
                                                           m->terms.data());
        B2S_CHECK_LAUNCH();
        b2s::k_fixed_reduce<<<1, b2s::SUM_THREADS, 0, st>>>(m->ng, m->terms.data(), 1, m->result.data());
        B2S_CHECK_LAUNCH();
        double toi = 1.1;
        B2S_CUDA(cudaMemcpyAsync(&toi, m->result.data(), sizeof(double), cudaMemcpyDeviceToHost, st));
        B2S_CUDA(cudaStreamSynchronize(st));
        *h_alpha = toi < 1.0 ? toi : 1.0;
        return 0;
    }
    catch(const b2s::Error& e)
    {
        g_gen_err = e.what();
        return e.code;
    }
    catch(const std::exception& e)
    {
        g_gen_err = e.what();
        return B2S_ERR_CUDA;
    }
}

}  // extern "C"
