// MAS (multi-level additive Schwarz) preconditioner: hierarchy, Galerkin
// cluster matrices, cluster inversion and apply.
//
// Algorithm of libuipc's MASPreconditionerEngine (StiffGIPC MAS, 16-node
// banks), src/backends/cuda/finite_element/mas_preconditioner_engine.cu:
//  * hierarchy (:57-460, host :1958-2280): partition slots form 16-lane banks;
//    connected components of the mesh graph inside a bank become one node of
//    the next level, numbered by bank then by lowest lane; coarser levels
//    repeat on the remaining cross-bank edges; levels capped at 6.
//  * Galerkin matrices (:530-953): the 48x48 matrix of every bank at every
//    level is R_l A R_l^T restricted to the bank, R_l summing the fine
//    vertices of each level-l node.
//  * inversion (:1077-1175): the inverse of every cluster matrix, no pivoting,
//    zero diagonal -> 1 (b2s_mas_invert.cu).
//  * apply (:1604-1955, :2887-2960): z = sum_l P_l^T A_l^{-1} P_l r with
//    summation restriction and injection prolongation, FP32 inside.
//
// Design here: the hierarchy is built by bank-parallel kernels; the coarse
// Galerkin matrices are built level by level as sparse matrices with the same
// deterministic triplet assembly as the global matrix (A_{l+1} from A_l), so
// no FP64 atomics pile onto the few clusters of the top levels; the apply
// restricts to every coarse level in one launch (above level 1 as partial sums
// per block of slots) and does every level in a second one (one warp per bank);
// every sum has a fixed order, so an apply is bit-reproducible.
#include "b2s_internal.cuh"
#include "b2s_reduce.cuh"
#include "b2s_mas_apply.cuh"

#include <algorithm>

namespace b2s
{
void mas_invert_clusters(b2s_solver* s, int mode);

namespace
{
inline int bank_align(int n) { return (n + BANK - 1) / BANK * BANK; }

int compute_num_levels(int vert_num)
{
    int n_level = 1, sz = bank_align(vert_num);
    while(sz > BANK)
    {
        sz /= BANK;
        n_level++;
        sz = bank_align(sz);
    }
    n_level++;
    return std::min(n_level, MAX_LEVELS);
}

// ---------------------------------------------------------------------------
// hierarchy kernels
// ---------------------------------------------------------------------------

// level 0: direct in-bank adjacency mask of every partition slot; cross-bank
// neighbours stay in the (compacted) list, unpartitioned ones are dropped
__global__ void k_h_mask_l0(int N, const int32_t* p2r, const int32_t* r2p, const int32_t* nbr_start,
                            int32_t* nbr_num, int32_t* nbr_list, uint32_t* mask)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if(p >= N)
        return;
    const int v = p2r[p];
    if(v < 0)
    {
        mask[p] = 0;
        return;
    }
    uint32_t m = 1u << (p % BANK);
    const int s = nbr_start[v], n = nbr_num[v];
    int       keep = 0;
    for(int e = 0; e < n; ++e)
    {
        const int u  = nbr_list[s + e];
        const int pu = r2p[u];
        if(pu < 0)
            continue;
        if(pu / BANK == p / BANK)
            m |= 1u << (pu % BANK);
        else
            nbr_list[s + keep++] = u;
    }
    nbr_num[v] = keep;
    mask[p]    = m;
}

// level l >= 1: OR the in-bank adjacency of every level-l node from its fine
// vertices' remaining neighbours
__global__ void k_h_mask_lx(int N, int vn, const int32_t* p2r, const int32_t* cst_prev, const int32_t* nbr_start,
                            int32_t* nbr_num, int32_t* nbr_list, uint32_t* next_mask, int cnt)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if(p >= N)
        return;
    const int v = p2r[p];
    if(v < 0)
        return;
    const int c = cst_prev[v];
    if(c < 0 || c >= cnt)
        return;
    uint32_t  conn = 0;
    const int s = nbr_start[v], n = nbr_num[v];
    int       keep = 0;
    for(int e = 0; e < n; ++e)
    {
        const int u  = nbr_list[s + e];
        const int cu = cst_prev[u];
        if(cu < 0 || cu >= cnt)
        {
            nbr_list[s + keep++] = u;
            continue;
        }
        if(cu / BANK == c / BANK)
            conn |= 1u << (cu % BANK);
        else
            nbr_list[s + keep++] = u;
    }
    nbr_num[v] = keep;
    if(conn)
        atomicOr(&next_mask[c], conn);
}

// one thread per bank: components (transitive closure of the lane masks),
// numbered by lowest lane; writes the component count, each node's rank and
// each node's component mask
__global__ void k_h_components(int n_nodes, int n_banks, const uint32_t* mask, const int32_t* valid_p2r,
                               int level0, int32_t* comp_count, int32_t* rank, uint16_t* comp_mask)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if(b >= n_banks)
        return;
    uint32_t m[BANK];
    bool     valid[BANK];
    for(int l = 0; l < BANK; ++l)
    {
        const int node = b * BANK + l;
        valid[l]       = node < n_nodes && (!level0 || valid_p2r[node] >= 0);
        m[l]           = valid[l] ? (mask[node] | (1u << l)) : 0u;
    }
    uint32_t closure[BANK];
    uint32_t elected = 0;
    for(int l = 0; l < BANK; ++l)
    {
        if(!valid[l])
        {
            closure[l] = 0;
            continue;
        }
        uint32_t c = m[l], visited = 1u << l;
        for(int guard = 0; guard < BANK; ++guard)
        {
            const uint32_t todo = visited ^ c;
            if(!todo)
                break;
            const int nv = __ffs(todo) - 1;
            visited |= 1u << nv;
            c |= m[nv];
        }
        closure[l] = c;
        if((c & ((1u << l) - 1u)) == 0)
            elected |= 1u << l;
    }
    for(int l = 0; l < BANK; ++l)
    {
        const int node = b * BANK + l;
        if(node >= n_nodes)
            break;
        if(valid[l])
        {
            const int el = __ffs(closure[l]) - 1;
            rank[node]      = __popc(elected & ((1u << el) - 1u));
            comp_mask[node] = (uint16_t)closure[l];
        }
        else
        {
            rank[node]      = -1;
            comp_mask[node] = 0;
        }
    }
    comp_count[b] = __popc(elected);
}

// next-level local id of every node (bank offset + component rank)
__global__ void k_h_assign(int n_nodes, const int32_t* rank, const int32_t* bank_offset, int32_t* new_local)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if(c >= n_nodes)
        return;
    const int rk = rank[c];
    new_local[c] = rk >= 0 ? bank_offset[c / BANK] + rk : -1;
}

// per vertex: local id at level 1 from its partition slot
__global__ void k_h_cst_l1(int vn, const int32_t* r2p, const int32_t* new_local0, int32_t* cst0)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if(v >= vn)
        return;
    const int p = r2p[v];
    cst0[v]     = p >= 0 ? new_local0[p] : -1;
}

__global__ void k_h_cst_next(int vn, const int32_t* cst_prev, const int32_t* new_local, int cnt, int32_t* cst_next)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if(v >= vn)
        return;
    const int c = cst_prev[v];
    cst_next[v] = (c >= 0 && c < cnt) ? new_local[c] : -1;
}

__global__ void k_h_ctable(int vn, int L, const int32_t* cst, const int32_t* level_begin_dev, int32_t* ctable)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if(v >= vn)
        return;
    for(int l = 1; l < L; ++l)
    {
        const int c = cst[(size_t)(l - 1) * vn + v];
        ctable[(size_t)v * (L - 1) + (l - 1)] = c >= 0 ? level_begin_dev[l] + c : -1;
    }
}

__global__ void k_h_node1(int vn, int L, const int32_t* ctable, int32_t* node1)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if(v < vn)
        node1[v] = ctable[(size_t)v * (L - 1)];
}

// ---------------------------------------------------------------------------
// Galerkin matrices
// ---------------------------------------------------------------------------

// One pass over a block-upper matrix, GAL_BLOCKS blocks per CTA, their values
// read once into shared memory in block order:
//  * EXTRACT (the global matrix): blocks inside one partition bank go to the
//    level-0 clusters, oriented by slot;
//  * the restriction to the next level as raw triplets: (a, b, B) -> (P a, P b)
//    with B, B^T or (a != b) B + B^T when both map to one node. Entries that
//    leave the MAS range get row -1 (their values are not written).
// Both outputs leave shared memory with consecutive lanes on consecutive
// doubles. (Two passes with 72-byte stores per thread took 406 us for 4.3 M
// blocks; this takes 184, of which 0.7 GB at the copy rate are 107.)
constexpr int GAL_BLOCKS = 256;
template <bool EXTRACT>
__global__ void __launch_bounds__(GAL_BLOCKS)
    k_g_restrict(int64_t U, const int32_t* __restrict__ rows, const int32_t* __restrict__ cols,
                 const double* __restrict__ vals, int64_t S, int off, int n_in, const int32_t* __restrict__ r2p,
                 const int32_t* __restrict__ map, int32_t* __restrict__ out_rows, int32_t* __restrict__ out_cols,
                 double* __restrict__ out_vals, double* __restrict__ hess)
{
    __shared__ double  s_b[GAL_BLOCKS * 9];
    __shared__ int32_t s_dst[GAL_BLOCKS];           // level-0 block (sign of swap in s_mode), -1: none
    __shared__ unsigned char s_mode[GAL_BLOCKS];  // bits 0-1: 0 drop, 1 B, 2 B^T, 3 B + B^T; bit 2: swap for level 0
    const int64_t base = (int64_t)blockIdx.x * GAL_BLOCKS;
    const int     m    = (int)(U - base < GAL_BLOCKS ? U - base : GAL_BLOCKS);
    const int     t    = threadIdx.x;
    if(t < m)
    {
        const int64_t k = base + t;
#pragma unroll
        for(int q = 0; q < 9; ++q)
            s_b[9 * t + q] = vals[(int64_t)q * S + k];
        const int a = rows[k] - off, b = cols[k] - off;
        int       ca = -1, cb = -1, mode = 0, dst = -1;
        if(a >= 0 && a < n_in && b >= 0 && b < n_in)
        {
            ca = map[a];
            cb = map[b];
            if constexpr(EXTRACT)
            {
                const int pa = r2p[a], pb = r2p[b];
                if(pa >= 0 && pb >= 0 && pa / BANK == pb / BANK)
                {
                    const int lo = pa < pb ? pa : pb, hi = pa < pb ? pb : pa;
                    dst = (lo / BANK) * SYM + sym_index(lo % BANK, hi % BANK);
                    mode |= pb < pa ? 4 : 0;
                }
            }
        }
        if(ca >= 0 && cb >= 0)
            mode |= ca < cb ? 1 : (ca > cb ? 2 : (a == b ? 1 : 3));
        else
            ca = cb = -1;
        out_rows[k] = ca < cb ? ca : cb;
        out_cols[k] = ca < cb ? cb : ca;
        s_mode[t] = (unsigned char)mode;
        if constexpr(EXTRACT)
            s_dst[t] = dst;
    }
    __syncthreads();
    for(int e = t; e < 9 * m; e += GAL_BLOCKS)
    {
        const int    blk = e / 9, q = e - 9 * blk, qt = (q % 3) * 3 + q / 3;  // qt: the transposed entry
        const int    mode = s_mode[blk];
        const double v = s_b[e], vt = s_b[9 * blk + qt];
        if((mode & 3) != 0)
            out_vals[base * 9 + e] = (mode & 3) == 1 ? v : ((mode & 3) == 2 ? vt : v + vt);
        if constexpr(EXTRACT)
            if(s_dst[blk] >= 0)
                hess[(size_t)s_dst[blk] * 9 + q] = (mode & 4) ? vt : v;
    }
}

// level l >= 1: in-bank blocks of the level-l Galerkin matrix into clusters
__global__ void k_g_extract(int64_t U, const int32_t* rows, const int32_t* cols, const double* vals, int64_t S,
                            int level_begin, double* hess)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(k >= U)
        return;
    const int a = rows[k], b = cols[k];
    if(a / BANK != b / BANK)
        return;
    const int ga = level_begin + a, gb = level_begin + b;
    double*   dst = hess + ((size_t)(ga / BANK) * SYM + sym_index(ga % BANK, gb % BANK)) * 9;
#pragma unroll
    for(int q = 0; q < 9; ++q)
        dst[q] = vals[(int64_t)q * S + k];
}

// The last coarse levels in one CTA: while a level's matrix has at most
// TAIL_BLOCKS blocks, every further level -- restriction, sort by (row, column,
// source), sums in source order, extraction of the clusters -- is a few
// microseconds of work that the general assembly spreads over a dozen launches
// and a wait of the host (about 50 us per level whatever its size). Same order
// of the sums as there.
constexpr int TAIL_BLOCKS  = 2048;
constexpr int TAIL_THREADS = 1024;
struct TailLevel
{
    int            begin;  // first node slot
    const int32_t* map;    // node of the level below -> node of this level
    int32_t*       rows;
    int32_t*       cols;
    double*        vals;  // planes of TAIL_BLOCKS
};
struct TailArgs
{
    int            first, L;
    int            U;  // blocks of level first - 1
    const int32_t* rows;
    const int32_t* cols;
    const double*  vals;
    int64_t        S;
    TailLevel      lv[MAX_LEVELS];
    double*        hess;
};
constexpr size_t TAIL_SMEM = (size_t)TAIL_BLOCKS * (9 * sizeof(double) + sizeof(uint64_t));

__global__ void __launch_bounds__(TAIL_THREADS) k_coarse_tail(TailArgs A)
{
    extern __shared__ double s_val[];  // [TAIL_BLOCKS][9], then the keys
    uint64_t*      s_key = reinterpret_cast<uint64_t*>(s_val + 9 * TAIL_BLOCKS);
    __shared__ int s_start[TAIL_BLOCKS + 1], s_warp[TAIL_THREADS / 32];
    const int      tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int            n = A.U;
    const int32_t* rows = A.rows;
    const int32_t* cols = A.cols;
    const double*  vals = A.vals;
    int64_t        S    = A.S;
    for(int l = A.first; l < A.L; ++l)
    {
        const TailLevel& T = A.lv[l];
        int              n2 = 32;
        while(n2 < n)
            n2 <<= 1;
        // keys (row << 38 | column << 12 | source) and values as restricted
        for(int k = tid; k < n2; k += TAIL_THREADS)
        {
            uint64_t key = ~0ull;
            if(k < n)
            {
                const int a = rows[k], b = cols[k], ca = T.map[a], cb = T.map[b];
                if(ca >= 0 && cb >= 0)
                {
                    const int lo = ca < cb ? ca : cb, hi = ca < cb ? cb : ca;
                    key = ((uint64_t)lo << 38) | ((uint64_t)hi << 12) | (uint64_t)k;
                    double B[9];
#pragma unroll
                    for(int q = 0; q < 9; ++q)
                        B[q] = vals[q * S + k];
#pragma unroll
                    for(int q = 0; q < 9; ++q)
                    {
                        const double t = B[(q % 3) * 3 + q / 3];
                        s_val[9 * k + q] = ca < cb || a == b ? B[q] : (ca > cb ? t : B[q] + t);
                    }
                }
            }
            s_key[k] = key;
        }
        __syncthreads();
        for(int size = 2; size <= n2; size <<= 1)
            for(int stride = size >> 1; stride > 0; stride >>= 1)
            {
                for(int i = tid; i < n2 / 2; i += TAIL_THREADS)
                {
                    const int      lo = 2 * i - (i & (stride - 1));
                    const int      hi = lo + stride;
                    const bool     up = (lo & size) == 0;
                    const uint64_t x = s_key[lo], y = s_key[hi];
                    if((x > y) == up)
                    {
                        s_key[lo] = y;
                        s_key[hi] = x;
                    }
                }
                __syncthreads();
            }
        // run starts: two consecutive positions per thread
        bool head[2], end[2];
#pragma unroll
        for(int j = 0; j < 2; ++j)
        {
            const int p = 2 * tid + j;
            const bool in = p < n2 && s_key[p] != ~0ull;
            head[j] = in && (p == 0 || (s_key[p - 1] >> 12) != (s_key[p] >> 12));
            end[j]  = in && (p + 1 == n2 || s_key[p + 1] == ~0ull);
        }
        int v = (int)head[0] + (int)head[1], incl = v;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            incl += lane >= o ? t : 0;
        }
        if(lane == 31)
            s_warp[w] = incl;
        __syncthreads();
        int slot = incl - v, U = 0;
#pragma unroll
        for(int q = 0; q < TAIL_THREADS / 32; ++q)
        {
            slot += q < w ? s_warp[q] : 0;
            U += s_warp[q];
        }
#pragma unroll
        for(int j = 0; j < 2; ++j)
        {
            if(head[j])
                s_start[slot++] = 2 * tid + j;
            if(end[j])
                s_start[U] = 2 * tid + j + 1;
        }
        __syncthreads();
        for(int e = tid; e < 9 * U; e += TAIL_THREADS)
        {
            const int      o = e / 9, q = e - 9 * o, b = s_start[o], f = s_start[o + 1];
            const uint64_t key = s_key[b];
            const int      r = (int)(key >> 38), c = (int)((key >> 12) & 0x3FFFFFFu);
            double         acc = s_val[9 * (int)(key & 0xFFFu) + q];
            for(int k = b + 1; k < f; ++k)
                acc += s_val[9 * (int)(s_key[k] & 0xFFFu) + q];
            T.vals[(int64_t)q * TAIL_BLOCKS + o] = acc;
            if(r / BANK == c / BANK)
            {
                const int gr = T.begin + r, gc = T.begin + c;
                A.hess[((size_t)(gr / BANK) * SYM + sym_index(gr % BANK, gc % BANK)) * 9 + q] = acc;
            }
            if(q == 0)
            {
                T.rows[o] = r;
                T.cols[o] = c;
            }
        }
        __syncthreads();  // the level's matrix is visible to the CTA, the shared arrays are free
        n    = U;
        rows = T.rows;
        cols = T.cols;
        vals = T.vals;
        S    = TAIL_BLOCKS;
    }
}

// pack the FP32 inverse M of every cluster as D (FP32) + the BF16 tiles of
// D^-1 M D^-1, D = diag(M)^1/2: the stored matrix has a unit diagonal, so BF16
// rounds every entry relative to O(1), and M = D (D^-1 M D^-1) D is recovered
// in the apply. Entry (a, b) comes from the stored upper 3x3 block of nodes
// (min, max) and is scaled as stored row times stored column.
// One CTA per cluster: the FP32 inverse staged in shared memory by 16-byte
// loads, then each thread writes 8 consecutive BF16 entries of one tile row
// (one 16-byte store): 6 tiles x 16 rows x 2 halves = 192 threads.
constexpr int PACK_THREADS = 192;
__global__ void __launch_bounds__(PACK_THREADS) k_pack_inverse_bf16(int clusters, const float* __restrict__ inv,
                                                                    unsigned char* __restrict__ out)
{
    const int c = blockIdx.x;
    if(c >= clusters)
        return;
    __shared__ float4 Ms4[SYM * 9 / 4];
    __shared__ float  S[BANK * 3];  // 1 / D
    const float4*  src = reinterpret_cast<const float4*>(inv + (size_t)c * SYM * 9);
    unsigned char* o   = out + (size_t)c * INV16_BYTES;
    for(int i = threadIdx.x; i < SYM * 9 / 4; i += PACK_THREADS)
        Ms4[i] = src[i];
    __syncthreads();
    const float* M = reinterpret_cast<const float*>(Ms4);
    if(threadIdx.x < BANK * 3)
    {
        const int   nd = threadIdx.x / 3, a = threadIdx.x % 3;
        const float d  = M[sym_index(nd, nd) * 9 + a * 3 + a];
        const float Dv = d > 0.f ? sqrtf(d) : 1.0f;
        S[threadIdx.x] = 1.0f / Dv;
        reinterpret_cast<float*>(o)[threadIdx.x] = Dv;
    }
    __syncthreads();
    const int t = threadIdx.x >> 5, row = (threadIdx.x >> 1) & 15, half = threadIdx.x & 1;
    const int I = t < 3 ? 0 : (t < 5 ? 1 : 2);
    const int J = t - (I * 3 - I * (I + 1) / 2);
    const int a = I * 16 + row, na = a / 3, pa = a % 3;
    uint32_t  w[4];
#pragma unroll
    for(int k = 0; k < 8; k += 2)
    {
        float v2[2];
#pragma unroll
        for(int u = 0; u < 2; ++u)
        {
            const int b = J * 16 + half * 8 + k + u, nb = b / 3, pb = b % 3;
            v2[u] = na <= nb ? M[sym_index(na, nb) * 9 + pb * 3 + pa] * S[a] * S[b]
                             : M[sym_index(nb, na) * 9 + pa * 3 + pb] * S[b] * S[a];
        }
        const __nv_bfloat162 h = __floats2bfloat162_rn(v2[0], v2[1]);
        w[k >> 1]              = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(o + INV16_SCALE_BYTES + t * INV16_TILE_BYTES + tile_off(row, half)) =
        make_uint4(w[0], w[1], w[2], w[3]);
}

// Every level in one launch: the restriction has left R_0, R_1 and the FP64
// partial sums of the levels above, so no bank waits for another. One launch per level
// (level 1 on the whole GPU, the others on a side stream beside the fine level,
// then a fold of the prolongation) left systems below ~100,000 vertices
// waiting for a chain of six 4-5 us launches: the level launches and the fold
// of an apply took 36 us for 88,641 vertices (FP32 inverses) and 54 for 551,368
// (BF16), launch by launch; this takes 8.8 and 26.8.
template <bool BF, int NST>
__global__ void __launch_bounds__(APPLY_WARPS * 32, BF ? 7 : 5) k_apply_all(ApplyArgs A, const int* converged)
{
    constexpr uint32_t SB = stage_bytes<BF>();
    __shared__ __align__(128) unsigned char s_stage[APPLY_WARPS][NST][SB];
    __shared__ uint64_t s_bar[APPLY_WARPS][NST];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if(lane == 0)
    {
        for(int q = 0; q < NST; ++q)
            mbar_init(&s_bar[w][q], 1);
        mbar_fence_init();
    }
    __syncwarp();
    __shared__ double s_sum[BANK * APPLY_WARPS * 3];
    const int         rest = (int)gridDim.x - A.heavy;
    int               gw = ((int)blockIdx.x - A.heavy) * APPLY_WARPS + w, W = rest * APPLY_WARPS;
    if(A.join)
        W += A.heavy * (APPLY_WARPS - 1);
    if((int)blockIdx.x < A.heavy)
    {
        static_assert(NST >= 2 && SB % 16 == 0, "a barrier and room for the entries");
        heavy_bank<BF, APPLY_WARPS>(A, (int64_t)A.g3 + blockIdx.x, converged, &s_stage[0][0][0], &s_stage[0][1][0],
                                    (APPLY_WARPS * NST - 1) * SB, s_bar[0], s_sum);
        if(w == 0 || !A.join)
            return;
        gw = rest * APPLY_WARPS + (int)blockIdx.x * (APPLY_WARPS - 1) + w - 1;  // last in the order
    }
    apply_banks<BF, NST>(gw, W, lane, A, converged, &s_stage[w][0][0], s_bar[w]);
}

// The fine residual in partition order and the sums of every coarse level, a
// thread per slot: R_0 (FP32, zero in padding slots) is the only gather of r
// through part_to_real, so the fine level streams its banks' residuals with
// their inverses.
template <typename VT>
__global__ void __launch_bounds__(RESTRICT_THREADS)
    k_restrict_fine(int n_slots, const int32_t* __restrict__ p2r, const VT* __restrict__ r, int roff,
                    const uint16_t* __restrict__ comp_mask, const int32_t* __restrict__ new_local,
                    const int4* __restrict__ dst, int begin1, int push, float* __restrict__ R,
                    double* __restrict__ part, const int* converged)
{
    if(converged && *converged)
        return;
    __shared__ float s_r[RESTRICT_THREADS][3], s_lead[RESTRICT_THREADS][3];
    __shared__ int4  s_dst[RESTRICT_THREADS];
    __shared__ int   s_n[RESTRICT_THREADS / 32];
    const int t = threadIdx.x, p = blockIdx.x * RESTRICT_THREADS + t, sub = t & 15;
    float     n0 = 0.f, n1 = 0.f, n2 = 0.f;
    uint32_t  cm = 0;
    int       nl = 0;
    int4      to = make_int4(-1, -1, -1, -1);
    if(p < n_slots)
    {
        const int v = p2r[p];
        if(v >= 0)
        {
            if(push)
            {
                cm = comp_mask[p];
                nl = new_local[p];
                if(cm != 0 && (cm & ((1u << sub) - 1u)) == 0)
                    to = dst[nl];
            }
            if constexpr(sizeof(VT) == 4)
            {
                const float4 q = *reinterpret_cast<const float4*>(r + roff + 4 * (int64_t)v);
                n0 = q.x;
                n1 = q.y;
                n2 = q.z;
            }
            else
            {
                n0 = (float)r[roff + 3 * (int64_t)v];
                n1 = (float)r[roff + 3 * (int64_t)v + 1];
                n2 = (float)r[roff + 3 * (int64_t)v + 2];
            }
        }
        R[3 * (int64_t)p]     = n0;
        R[3 * (int64_t)p + 1] = n1;
        R[3 * (int64_t)p + 2] = n2;
    }
    s_r[t][0] = n0;
    s_r[t][1] = n1;
    s_r[t][2] = n2;
    __syncthreads();
    if(push)
        restrict_coarse<RESTRICT_THREADS>(s_r, cm, nl, to, begin1, R, part, s_lead, s_dst, s_n);
}

// the ancestors of the level-1 nodes, four per node (levels 2-5; -1: none):
// the finish adds Z of a vertex's slot, its level-1 node and these
static_assert(MAX_LEVELS == 6, "four ancestors above level 1");
struct LevelIds
{
    const int32_t* new_local[MAX_LEVELS];
    int32_t        begin[MAX_LEVELS + 1];
};
__global__ void k_h_ancestors(int cnt1, int L, LevelIds ids, int4* anc)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if(c >= cnt1)
        return;
    int loc = c, a[4] = {-1, -1, -1, -1};
    for(int l = 2; l < L; ++l)
    {
        loc      = loc >= 0 ? ids.new_local[l - 1][loc] : -1;
        a[l - 2] = loc >= 0 ? ids.begin[l] + loc : -1;
    }
    anc[c] = make_int4(a[0], a[1], a[2], a[3]);
}

// the block of slots of every level-1 node
__global__ void k_h_block(int n_slots, const int32_t* __restrict__ new_local, int32_t* __restrict__ block)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if(p < n_slots && new_local[p] >= 0)
        block[new_local[p]] = p / RESTRICT_THREADS;  // the same from every slot of the node
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

// The entries of the partial sums above level 1 (MasState::part): for every
// node there, one per block of RESTRICT_THREADS slots with a level-1 node under
// it, in block order; every level-1 node learns its entries. Level-1 nodes are
// numbered bank by bank, so their blocks ascend.
static void place_partials(b2s_solver* s)
{
    MasState&     M    = s->mas;
    const int     cnt1 = M.level_count[1], begin2 = M.level_begin[2], nodes = M.total - begin2;
    cudaStream_t  st   = s->stream;
    DBuf<int32_t> d_block;
    d_block.resize(std::max(cnt1, 1));
    std::vector<int32_t> block(cnt1), start(nodes + 1, 0), last(nodes, -1);
    std::vector<int4>    dst(cnt1);
    if(cnt1 > 0)
    {
        k_h_block<<<grid_for(M.N, 256), 256, 0, st>>>(M.N, M.new_local[0].data(), d_block.data());
        B2S_CHECK_LAUNCH();
        B2S_CUDA(cudaMemcpyAsync(block.data(), d_block.data(), sizeof(int32_t) * cnt1, cudaMemcpyDeviceToHost, st));
        B2S_CUDA(cudaMemcpyAsync(dst.data(), M.anc.data(), sizeof(int4) * cnt1, cudaMemcpyDeviceToHost, st));
        B2S_CUDA(cudaStreamSynchronize(st));
    }
    // dst: the ancestors, then 2 (place among the node's entries) + (not the
    // entry's first); start[m + 1]: the node's entries
    for(int c = 0; c < cnt1; ++c)
        for(int32_t* a : {&dst[c].x, &dst[c].y, &dst[c].z, &dst[c].w})
            if(*a >= 0)
            {
                const int  m     = *a - begin2;
                const bool first = last[m] != block[c];
                last[m]          = block[c];
                start[m + 1] += first ? 1 : 0;
            }
    int64_t entries = 0;
    for(int m = 0; m < nodes; ++m)
    {
        entries += start[m + 1];
        B2S_REQUIRE(entries < INT32_MAX / 2, B2S_ERR_ARGUMENT, "MAS hierarchy too large");
        start[m + 1] = (int32_t)entries;
        last[m]      = -1;
    }
    std::vector<int32_t> next(start.begin(), start.end() - 1);  // the entry after the node's current one
    for(int c = 0; c < cnt1; ++c)
        for(int32_t* a : {&dst[c].x, &dst[c].y, &dst[c].z, &dst[c].w})
            if(*a >= 0)
            {
                const int  m     = *a - begin2;
                const bool first = last[m] != block[c];
                last[m]          = block[c];
                next[m] += first ? 1 : 0;
                *a = 2 * (next[m] - 1) + (first ? 0 : 1);
            }
    M.tail_idx.resize((size_t)2 * TAIL_BLOCKS * (M.L - 2));
    M.tail_vals.resize((size_t)9 * TAIL_BLOCKS * (M.L - 2));
    M.part.resize(3 * (size_t)entries + 3);  // one more: copies end at even entries
    M.part_start.resize(nodes + 1);
    M.part_dst.resize(std::max(cnt1, 1));
    B2S_CUDA(cudaMemcpyAsync(M.part_start.data(), start.data(), sizeof(int32_t) * (nodes + 1), cudaMemcpyHostToDevice,
                             st));
    if(cnt1 > 0)
        B2S_CUDA(cudaMemcpyAsync(M.part_dst.data(), dst.data(), sizeof(int4) * cnt1, cudaMemcpyHostToDevice, st));
    B2S_CUDA(cudaStreamSynchronize(st));
}

void mas_init(b2s_solver* s, int32_t offset, int32_t vn, const int32_t* adj_start, const int32_t* adj_list, int32_t N,
              const int32_t* p2r, const int32_t* r2p)
{
    B2S_REQUIRE(vn > 0 && N > 0 && offset >= 0, B2S_ERR_ARGUMENT, "MAS range must be non-empty");
    B2S_REQUIRE(N % BANK == 0, B2S_ERR_ARGUMENT, "part_map_size must be a multiple of 16");
    // validate the maps on the host (the reference asserts the same, fem_mas_preconditioner.cu:331-360)
    for(int p = 0; p < N; ++p)
    {
        B2S_REQUIRE(p2r[p] >= -1 && p2r[p] < vn, B2S_ERR_ARGUMENT, "part_to_real entry out of range");
        if(p2r[p] >= 0)
            B2S_REQUIRE(r2p[p2r[p]] == p, B2S_ERR_ARGUMENT, "part_to_real / real_to_part are not inverse");
    }
    for(int v = 0; v < vn; ++v)
    {
        B2S_REQUIRE(r2p[v] >= -1 && r2p[v] < N, B2S_ERR_ARGUMENT, "real_to_part entry out of range");
        if(r2p[v] >= 0)
            B2S_REQUIRE(p2r[r2p[v]] == v, B2S_ERR_ARGUMENT, "part_to_real / real_to_part are not inverse");
        B2S_REQUIRE(adj_start[v + 1] >= adj_start[v], B2S_ERR_ARGUMENT, "adjacency start not monotone");
    }
    const int64_t nnz_adj = adj_start[vn];
    for(int64_t e = 0; e < nnz_adj; ++e)
        B2S_REQUIRE(adj_list[e] >= 0 && adj_list[e] < vn, B2S_ERR_ARGUMENT, "adjacency entry out of range");

    cudaStream_t st = s->stream;
    MasState&    M  = s->mas;
    MasState&    X  = s->mas;
    M.initialized   = false;
    M.generation += 1;
    M.offset        = offset;
    M.vn            = vn;
    M.N             = N;
    M.L             = compute_num_levels(std::max(N, vn));
    const int L     = M.L;
    M.level_begin.assign(L + 1, 0);
    M.level_count.assign(L + 1, 0);

    DBuf<int32_t> d_start, d_num, d_list;
    std::vector<int32_t> h_num(vn);
    for(int v = 0; v < vn; ++v)
        h_num[v] = adj_start[v + 1] - adj_start[v];
    d_start.resize(vn + 1);
    d_num.resize(vn);
    d_list.resize(std::max<int64_t>(nnz_adj, 1));
    M.p2r.resize(N);
    M.r2p.resize(vn);
    B2S_CUDA(cudaMemcpyAsync(d_start.data(), adj_start, sizeof(int32_t) * (vn + 1), cudaMemcpyHostToDevice, st));
    B2S_CUDA(cudaMemcpyAsync(d_num.data(), h_num.data(), sizeof(int32_t) * vn, cudaMemcpyHostToDevice, st));
    if(nnz_adj > 0)
        B2S_CUDA(cudaMemcpyAsync(d_list.data(), adj_list, sizeof(int32_t) * nnz_adj, cudaMemcpyHostToDevice, st));
    B2S_CUDA(cudaMemcpyAsync(M.p2r.data(), p2r, sizeof(int32_t) * N, cudaMemcpyHostToDevice, st));
    B2S_CUDA(cudaMemcpyAsync(M.r2p.data(), r2p, sizeof(int32_t) * vn, cudaMemcpyHostToDevice, st));

    // level-1 node slots start after every level-0 slot and every vertex id
    // (mas_preconditioner_engine.cu:2162-2184 numbers them the same way)
    const int level1_begin = bank_align(std::max(bank_align(N), vn));
    X.cst.resize((size_t)L * vn);
    B2S_CUDA(cudaMemsetAsync(X.cst.data(), 0xff, sizeof(int32_t) * (size_t)L * vn, st));

    DBuf<uint32_t> mask;
    DBuf<int32_t>  comp_count, bank_off, rank, scan_tmp;
    mask.resize(std::max(N, vn) + BANK);
    rank.resize(std::max(N, vn) + BANK);
    const int TB = 256;

    // level 0
    {
        const int n_banks = N / BANK;
        comp_count.resize(n_banks + 1);
        bank_off.resize(n_banks + 1);
        X.comp_mask[0].resize(N);
        X.new_local[0].resize(N);
        k_h_mask_l0<<<grid_for(N, TB), TB, 0, st>>>(N, M.p2r.data(), M.r2p.data(), d_start.data(), d_num.data(),
                                                    d_list.data(), mask.data());
        B2S_CHECK_LAUNCH();
        k_h_components<<<grid_for(n_banks, 128), 128, 0, st>>>(N, n_banks, mask.data(), M.p2r.data(), 1,
                                                                comp_count.data(), rank.data(),
                                                                X.comp_mask[0].data());
        B2S_CHECK_LAUNCH();
        exclusive_scan(s, comp_count.data(), bank_off.data(), n_banks, scan_tmp);
        k_h_assign<<<grid_for(N, TB), TB, 0, st>>>(N, rank.data(), bank_off.data(), X.new_local[0].data());
        B2S_CHECK_LAUNCH();
        k_h_cst_l1<<<grid_for(vn, TB), TB, 0, st>>>(vn, M.r2p.data(), X.new_local[0].data(), X.cst.data());
        B2S_CHECK_LAUNCH();
        int32_t cnt1 = 0;
        B2S_CUDA(cudaMemcpyAsync(&cnt1, bank_off.data() + n_banks, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        B2S_CUDA(cudaStreamSynchronize(st));
        M.level_begin[0] = 0;
        M.level_count[0] = N;
        M.level_begin[1] = level1_begin;
        M.level_count[1] = cnt1;
    }
    // levels 1 .. L-1
    for(int level = 1; level < L; ++level)
    {
        const int cnt = M.level_count[level], beg = M.level_begin[level];
        const int n_banks = (cnt + BANK - 1) / BANK;
        const int next_begin = beg + bank_align(cnt);
        B2S_CUDA(cudaMemsetAsync(mask.data(), 0, sizeof(uint32_t) * (cnt + BANK), st));
        const int32_t* cst_prev = X.cst.data() + (size_t)(level - 1) * vn;
        k_h_mask_lx<<<grid_for(N, TB), TB, 0, st>>>(N, vn, M.p2r.data(), cst_prev, d_start.data(), d_num.data(),
                                                    d_list.data(), mask.data(), cnt);
        B2S_CHECK_LAUNCH();
        comp_count.resize(n_banks + 1);
        bank_off.resize(n_banks + 1);
        X.comp_mask[level].resize(std::max(cnt, 1));
        X.new_local[level].resize(std::max(cnt, 1));
        k_h_components<<<grid_for(n_banks, 128), 128, 0, st>>>(cnt, n_banks, mask.data(), nullptr, 0,
                                                                comp_count.data(), rank.data(),
                                                                X.comp_mask[level].data());
        B2S_CHECK_LAUNCH();
        exclusive_scan(s, comp_count.data(), bank_off.data(), n_banks, scan_tmp);
        k_h_assign<<<grid_for(cnt, TB), TB, 0, st>>>(cnt, rank.data(), bank_off.data(), X.new_local[level].data());
        B2S_CHECK_LAUNCH();
        k_h_cst_next<<<grid_for(vn, TB), TB, 0, st>>>(vn, cst_prev, X.new_local[level].data(), cnt,
                                                      X.cst.data() + (size_t)level * vn);
        B2S_CHECK_LAUNCH();
        int32_t cnt_next = 0;
        B2S_CUDA(cudaMemcpyAsync(&cnt_next, bank_off.data() + n_banks, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        B2S_CUDA(cudaStreamSynchronize(st));
        if(level + 1 <= L)
        {
            if(level + 1 < (int)M.level_begin.size())
            {
                M.level_begin[level + 1] = next_begin;
                M.level_count[level + 1] = cnt_next;
            }
        }
    }
    M.total    = M.level_begin[L];
    M.clusters = M.total / BANK;
    // coarse table
    X.level_begin_dev.resize(L + 1);
    B2S_CUDA(cudaMemcpyAsync(X.level_begin_dev.data(), M.level_begin.data(), sizeof(int32_t) * (L + 1),
                             cudaMemcpyHostToDevice, st));
    M.ctable.resize((size_t)vn * std::max(L - 1, 1));
    if(L > 1)
    {
        k_h_ctable<<<grid_for(vn, TB), TB, 0, st>>>(vn, L, X.cst.data(), X.level_begin_dev.data(), M.ctable.data());
        B2S_CHECK_LAUNCH();
    }
    M.hess.resize((size_t)M.clusters * SYM * 9);
    M.inv.resize((size_t)M.clusters * SYM * 9);
    M.R.resize((size_t)M.total * 3 + 3);
    M.Z.resize((size_t)M.total * 3 + 3);
    B2S_CUDA(cudaMemsetAsync(M.R.data(), 0, M.R.bytes(), st));
    B2S_CUDA(cudaMemsetAsync(M.Z.data(), 0, M.Z.bytes(), st));
    // the coarse ancestors of every level-1 node (the prolongation)
    if(L > 1 && M.level_count[1] > 0)
    {
        LevelIds ids{};
        for(int l = 0; l < L; ++l)
        {
            ids.new_local[l] = X.new_local[l].data();
            ids.begin[l]     = M.level_begin[l];
        }
        M.anc.resize(M.level_count[1]);
        k_h_ancestors<<<grid_for(M.level_count[1], TB), TB, 0, st>>>(M.level_count[1], L, ids, M.anc.data());
        B2S_CHECK_LAUNCH();
    }
    if(L > 1)
        place_partials(s);
    // level-1 node of every vertex, contiguous (the finish reads it per vertex)
    M.node1.resize(std::max(vn, 1));
    if(L > 1)
    {
        k_h_node1<<<grid_for(vn, TB), TB, 0, st>>>(vn, L, M.ctable.data(), M.node1.data());
        B2S_CHECK_LAUNCH();
    }
    M.h_ctable.resize((size_t)vn * std::max(L - 1, 1));
    if(L > 1)
        B2S_CUDA(cudaMemcpyAsync(M.h_ctable.data(), M.ctable.data(), sizeof(int32_t) * M.h_ctable.size(),
                                 cudaMemcpyDeviceToHost, st));
    B2S_CUDA(cudaStreamSynchronize(st));
    M.initialized = true;
}

void mas_assemble(b2s_solver* s, int invert_mode)
{
    MasState& M = s->mas;
    MasState& X = s->mas;
    B2S_REQUIRE(M.initialized, B2S_ERR_STATE, "MAS not initialised");
    B2S_REQUIRE(s->A.valid, B2S_ERR_STATE, "no assembled matrix");
    B2S_REQUIRE(M.offset + M.vn <= s->A.nb, B2S_ERR_ARGUMENT, "MAS range exceeds the matrix");
    cudaStream_t st = s->stream;
    const int    TB = 256;
    const Matrix& A = s->A;
    B2S_CUDA(cudaMemsetAsync(M.hess.data(), 0, M.hess.bytes(), st));
    // coarse levels: A_1 from A (vertex ids -> level-1 ids), A_{l+1} from A_l
    const Matrix* prev     = &A;
    int           prev_off = M.offset;
    int           prev_n   = M.vn;
    const int32_t* map     = X.cst.data();  // vertex -> level-1 local id
    for(int level = 1; level < M.L; ++level)
    {
        const int64_t T = prev->nnz;
        Matrix&       C = M.coarse[level];
        if(level > 1 && T <= TAIL_BLOCKS)
        {
            if(T == 0)
                break;
            TailArgs a{};
            a.first = level;
            a.L     = M.L;
            a.U     = (int)T;
            a.rows  = prev->rows.data();
            a.cols  = prev->cols.data();
            a.vals  = prev->vals.data();
            a.S     = prev->stride;
            a.hess  = M.hess.data();
            for(int l = level; l < M.L; ++l)
            {
                int32_t* idx = M.tail_idx.data() + (size_t)2 * TAIL_BLOCKS * (l - 2);
                a.lv[l] = TailLevel{M.level_begin[l], X.new_local[l - 1].data(), idx, idx + TAIL_BLOCKS,
                                    M.tail_vals.data() + (size_t)9 * TAIL_BLOCKS * (l - 2)};
            }
            B2S_CUDA(cudaFuncSetAttribute(k_coarse_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_SMEM));
            k_coarse_tail<<<1, TAIL_THREADS, TAIL_SMEM, st>>>(a);
            B2S_CHECK_LAUNCH();
            break;
        }
        M.trip_rows.resize(std::max<int64_t>(T, 1), 1.2);
        M.trip_cols.resize(std::max<int64_t>(T, 1), 1.2);
        M.trip_vals.resize((size_t)9 * std::max<int64_t>(T, 1), 1.2);
        if(T > 0)
        {
            auto k = level == 1 ? k_g_restrict<true> : k_g_restrict<false>;  // level 1: and the level-0 clusters
            k<<<grid_for(T, GAL_BLOCKS), GAL_BLOCKS, 0, st>>>(
                T, prev->rows.data(), prev->cols.data(), prev->vals.data(), prev->stride, prev_off, prev_n,
                M.r2p.data(), map, M.trip_rows.data(), M.trip_cols.data(), M.trip_vals.data(), M.hess.data());
            B2S_CHECK_LAUNCH();
        }
        assemble_triplets(s, C, M.level_count[level], T, M.trip_rows.data(), M.trip_cols.data(), M.trip_vals.data());
        if(C.nnz > 0)
        {
            k_g_extract<<<grid_for(C.nnz, TB), TB, 0, st>>>(C.nnz, C.rows.data(), C.cols.data(), C.vals.data(),
                                                            C.stride, M.level_begin[level], M.hess.data());
            B2S_CHECK_LAUNCH();
        }
        prev     = &C;
        prev_off = 0;
        prev_n   = M.level_count[level];
        map      = X.new_local[level].data();
    }
    mas_invert_clusters(s, invert_mode);
}

ApplyArgs mas_apply_args(b2s_solver* s, bool bf16)
{
    MasState& M = s->mas;
    ApplyArgs A{};
    A.inv   = bf16 ? M.inv16.data() : reinterpret_cast<const unsigned char*>(M.inv.data());
    A.inv32 = M.inv.data();
    A.stiff = bf16 ? M.stiff.data() : nullptr;
    A.R     = M.R.data();
    A.Z     = M.Z.data();
    A.part       = M.part.data();
    A.part_start = M.part_start.data();
    A.err   = device_error_flag(s);
    A.n0    = M.N / BANK;
    A.n1    = M.L > 1 ? (M.level_count[1] + BANK - 1) / BANK : 0;
    A.g1    = M.L > 1 ? M.level_begin[1] / BANK : 0;
    A.g2    = M.L > 2 ? M.level_begin[2] / BANK : M.clusters;
    A.g3    = M.L > 3 ? M.level_begin[3] / BANK : M.clusters;
    A.n2    = M.clusters - A.g2;
    A.n3    = M.clusters - A.g3;
    A.heavy = A.join = 0;
    return A;
}

// Z of every node from R_0, R_1 and the partial sums of the levels above
void mas_apply_all(b2s_solver* s, const int* converged, bool bf16)
{
    ApplyArgs A = mas_apply_args(s, bf16);
    const int n = A.n0 + A.n1 + A.n2;
    if(n == 0)
        return;
    auto k   = bf16 ? k_apply_all<true, APPLY_STAGES_BF16> : k_apply_all<false, APPLY_STAGES_F32>;
    int  occ = 0;
    if(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, APPLY_WARPS * 32, 0) != cudaSuccess || occ < 1)
        occ = 1;
    // persistent: the CTAs that fit at once, at most one warp per bank; the banks
    // of level 3 up have a CTA each, while those are an eighth at most. Its other
    // warps are late for the rest: they join it when it takes four banks a warp
    const int most = NUM_SMS_HINT * occ;
    if(8 * A.n3 <= std::min((n + APPLY_WARPS - 1) / APPLY_WARPS, most))
        A.heavy = A.n3;
    const int grid = std::min(A.heavy + (n - A.heavy + APPLY_WARPS - 1) / APPLY_WARPS, most);
    A.join         = n >= 4 * APPLY_WARPS * grid;
    k<<<grid, APPLY_WARPS * 32, 0, s->stream>>>(A, converged);
    B2S_CHECK_LAUNCH();
}

// z[off..off+vn) gets the MAS part of z = P r; Jacobi/identity elsewhere is
// handled by the caller (collect kernel in the PCG, or precond_apply).
// bf16: use the packed D + BF16 tiles of D^-1 M D^-1 (mas_pack_bf16 first).
template <typename VT>
static void apply_levels_t(b2s_solver* s, const VT* r, const int* converged, bool bf16)
{
    MasState&    M        = s->mas;
    cudaStream_t st       = s->stream;
    // element offset of the range's first vertex in r (FP32: 4 per node)
    const int off = (sizeof(VT) == 4 ? 4 : 3) * M.offset;
    k_restrict_fine<VT><<<grid_for(M.N, RESTRICT_THREADS), RESTRICT_THREADS, 0, st>>>(
        M.N, M.p2r.data(), r, off, M.comp_mask[0].data(), M.new_local[0].data(), M.part_dst.data(),
        M.L > 1 ? M.level_begin[1] : 0, M.L > 1 ? 1 : 0, M.R.data(), M.part.data(), converged);
    B2S_CHECK_LAUNCH();
    mas_apply_all(s, converged, bf16);
}

void mas_apply_levels(b2s_solver* s, const double* r, const int* converged)
{
    apply_levels_t<double>(s, r, converged, false);
}

void mas_apply_levels_f32(b2s_solver* s, const float* r, const int* converged, bool bf16)
{
    apply_levels_t<float>(s, r, converged, bf16);
}

// BF16 diagonal-scaled copy of the current FP32 inverses
void mas_pack_bf16(b2s_solver* s)
{
    MasState& M = s->mas;
    M.inv16.resize((size_t)M.clusters * INV16_BYTES);
    if(M.clusters > 0)
    {
        k_pack_inverse_bf16<<<M.clusters, PACK_THREADS, 0, s->stream>>>(M.clusters, M.inv.data(), M.inv16.data());
        B2S_CHECK_LAUNCH();
    }
}
}  // namespace b2s
