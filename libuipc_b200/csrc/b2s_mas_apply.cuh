// Device code of the MAS apply: the restriction to the coarse levels, products
// of one bank's inverse with its residuals, and the streams of banks.
#pragma once
#include "b2s_internal.cuh"
#include "b2s_tma.cuh"

#include <cuda_bf16.h>

namespace b2s
{
__host__ __device__ __forceinline__ int sym_index(int row, int col)
{
    return BANK * row - row * (row + 1) / 2 + col;
}

// ---------------------------------------------------------------------------
// apply: one warp per bank, persistent over banks. The bank's inverse is
// brought into shared memory by bulk asynchronous copies (TMA), NST deep per
// warp, so later banks' copies are in flight while this one computes.
//
// FP32 inverses (4,896 B: the 136 upper 3x3 blocks, column-major) are applied
// on the CUDA cores: lanes 0-15 own the bank's nodes and the 48x48 product is
// split over the two half-warps (columns 0-7 / 8-15).
//
// BF16 inverses (mixed precision) are applied on the tensor cores. Per cluster:
// the FP32 factor D = diag(M)^1/2 (48 floats, 192 B), then the six upper 16x16
// tiles (I <= J) of the 48x48 matrix D^-1 M D^-1 in BF16 (6 x 512 B), 3,264 B
// in all. Tile rows are 32 B; the two 16-B halves of row R are swapped when
// bit 2 of R is set, so each 8-row ldmatrix phase touches all 32 banks once.
// z = D (M_s (D r)) by mma.m16n8k16 (BF16 operands, FP32 accumulation): A is
// tile (I, J), for J < I the stored tile (J, I) loaded transposed; B column 0
// is BF16(D r) and column 1 its BF16 rounding remainder, so the FP32 residual
// enters with ~16 significant bits and the stored inverse is the only 8-bit
// rounding. (A 48x48 matrix times one vector is an HBM-bound GEMV; the tensor
// cores are used to cut the instruction count per byte, not for FLOPs.)
// ---------------------------------------------------------------------------
constexpr int APPLY_WARPS = 4;
constexpr uint32_t INV_BYTES = SYM * 9 * sizeof(float);  // 4896, a multiple of 16
constexpr uint32_t INV16_SCALE_BYTES = BANK * 3 * sizeof(float);                    // 192
constexpr uint32_t INV16_TILE_BYTES  = 16 * 16 * 2;                                 // 512
constexpr uint32_t INV16_BYTES       = INV16_SCALE_BYTES + 6 * INV16_TILE_BYTES;  // 3264
constexpr int APPLY_STAGES_F32  = 2;
constexpr int APPLY_STAGES_BF16 = 2;

// index of the upper tile (I, J), I <= J: (0,0) (0,1) (0,2) (1,1) (1,2) (2,2)
__host__ __device__ __forceinline__ int tile_id(int I, int J) { return I * 3 - I * (I + 1) / 2 + J; }
// byte offset of 16-B half `half` of row `row` inside a tile
__host__ __device__ __forceinline__ uint32_t tile_off(int row, int half)
{
    return (uint32_t)row * 32u + ((uint32_t)(half ^ ((row >> 2) & 1)) << 4);
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t& a0, uint32_t& a1, uint32_t& a2, uint32_t& a3)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3)
                 : "r"(addr));
}
// c += A (16x16, row) * B (16x8, col), BF16 in, FP32 accumulate
__device__ __forceinline__ void mma_bf16_16816(float& c0, float& c1, float& c2, float& c3, uint32_t a0, uint32_t a1,
                                               uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c0), "+f"(c1), "+f"(c2), "+f"(c3)
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16x2(__nv_bfloat16 lo, __nv_bfloat16 hi)
{
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// Zb[0..48) = D M_s D r for one cluster; r48: the bank's residual (node-major)
__device__ __forceinline__ void cluster_product_mma(const unsigned char* slot, const float* r48, int lane,
                                                    float* __restrict__ Zb)
{
    const float*   D     = reinterpret_cast<const float*>(slot);
    const uint32_t tiles = smem_addr(slot + INV16_SCALE_BYTES);
    const int      g = lane >> 2, t = lane & 3;
    uint32_t       b[3][2];
#pragma unroll
    for(int J = 0; J < 3; ++J)
    {
#pragma unroll
        for(int h = 0; h < 2; ++h)
        {
            const int           k  = J * 16 + 2 * t + 8 * h;
            const float         x0 = r48[k] * D[k], x1 = r48[k + 1] * D[k + 1];
            const __nv_bfloat16 h0 = __float2bfloat16_rn(x0), h1 = __float2bfloat16_rn(x1);
            uint32_t            v  = 0;
            if(g == 0)
                v = pack_bf16x2(h0, h1);
            else if(g == 1)
                v = pack_bf16x2(__float2bfloat16_rn(x0 - __bfloat162float(h0)),
                                __float2bfloat16_rn(x1 - __bfloat162float(h1)));
            b[J][h] = v;
        }
    }
    // row address this lane gives ldmatrix: matrix q = lane / 8 of the four
    // 8x8 quarters, row lane % 8 of it
    const int      q = lane >> 3, rr = lane & 7;
    const uint32_t offN = tile_off(rr + ((q & 1) << 3), q >> 1);
    const uint32_t offT = tile_off(rr + ((q >> 1) << 3), q & 1);
#pragma unroll
    for(int I = 0; I < 3; ++I)
    {
        float c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f;
#pragma unroll
        for(int J = 0; J < 3; ++J)
        {
            uint32_t a0, a1, a2, a3;
            if(J >= I)
                ldsm_x4(tiles + tile_id(I, J) * INV16_TILE_BYTES + offN, a0, a1, a2, a3);
            else
                ldsm_x4_trans(tiles + tile_id(J, I) * INV16_TILE_BYTES + offT, a0, a1, a2, a3);
            mma_bf16_16816(c0, c1, c2, c3, a0, a1, a2, a3, b[J][0], b[J][1]);
        }
        if(t == 0)
        {
            const int k0 = I * 16 + g, k1 = k0 + 8;
            Zb[k0] = (c0 + c1) * D[k0];
            Zb[k1] = (c2 + c3) * D[k1];
        }
    }
}

__device__ __forceinline__ void cluster_product(const float* M, const float (*r)[3], int lane, float out[3])
{
    // lanes 0..15: row node `lane`, columns 0..7; lanes 16..31: row node lane-16, columns 8..15
    const int rn = lane & 15, c0 = (lane >> 4) * 8;
    float acc0 = 0.f, acc1 = 0.f, acc2 = 0.f;
#pragma unroll
    for(int cc = 0; cc < 8; ++cc)
    {
        const int cn = c0 + cc;
        const float x0 = r[cn][0], x1 = r[cn][1], x2 = r[cn][2];
        if(cn >= rn)
        {
            const float* B = M + sym_index(rn, cn) * 9;  // column-major
            acc0 = __fmaf_rn(B[0], x0, acc0); acc0 = __fmaf_rn(B[3], x1, acc0); acc0 = __fmaf_rn(B[6], x2, acc0);
            acc1 = __fmaf_rn(B[1], x0, acc1); acc1 = __fmaf_rn(B[4], x1, acc1); acc1 = __fmaf_rn(B[7], x2, acc1);
            acc2 = __fmaf_rn(B[2], x0, acc2); acc2 = __fmaf_rn(B[5], x1, acc2); acc2 = __fmaf_rn(B[8], x2, acc2);
        }
        else
        {
            const float* B = M + sym_index(cn, rn) * 9;  // use B^T
            acc0 = __fmaf_rn(B[0], x0, acc0); acc0 = __fmaf_rn(B[1], x1, acc0); acc0 = __fmaf_rn(B[2], x2, acc0);
            acc1 = __fmaf_rn(B[3], x0, acc1); acc1 = __fmaf_rn(B[4], x1, acc1); acc1 = __fmaf_rn(B[5], x2, acc1);
            acc2 = __fmaf_rn(B[6], x0, acc2); acc2 = __fmaf_rn(B[7], x1, acc2); acc2 = __fmaf_rn(B[8], x2, acc2);
        }
    }
    acc0 += __shfl_down_sync(0xffffffffu, acc0, 16);
    acc1 += __shfl_down_sync(0xffffffffu, acc1, 16);
    acc2 += __shfl_down_sync(0xffffffffu, acc2, 16);
    out[0] = acc0;
    out[1] = acc1;
    out[2] = acc2;
}

// Every bank's residual slice (16 nodes x 3 floats, 192 B, contiguous) and its
// inverse come into shared memory by bulk copies (TMA) on one barrier, NST
// banks ahead per warp, so a warp never waits on a dependent gather. BF: BF16
// tiles on the tensor cores (INV16_BYTES per cluster), otherwise FP32
// (INV_BYTES); a stiff cluster (inverted in FP64) is applied from its FP32
// inverse in HBM in the BF16 path.
constexpr uint32_t R_BYTES = BANK * 3 * sizeof(float);  // 192

template <bool BF>
__host__ __device__ constexpr uint32_t stage_bytes()
{
    return (BF ? INV16_BYTES : INV_BYTES) + R_BYTES;
}

// what the apply reads and writes
struct ApplyArgs
{
    const unsigned char* inv;    // packed inverses of all clusters (FP32 or BF16)
    const float*         inv32;  // FP32 inverses (stiff clusters of the BF16 path)
    const uint8_t*       stiff;  // [clusters], null in the FP32 path
    float*               R;
    float*               Z;
    const double*        part;        // partial sums of the levels above 1 (MasState::part)
    const int32_t*       part_start;  // [node from slot 16 g2 on] its first entry
    int*                 err;
    int                  n0, n1, n2, n3;  // banks of level 0, of level 1, of all levels from 2, 3 up
    int                  g1, g2, g3;      // first bank of level 1, 2 and 3
    int                  heavy;  // n3 when the first n3 CTAs take those banks, else 0
    int                  join;   // 1: their other warps then join the rest
};

// the bank's inverse and, with `with_r`, its residual slice, on one barrier
template <bool BF>
__device__ __forceinline__ void issue_bank_copy(unsigned char* stage, uint64_t* bar, const ApplyArgs& A, int64_t gbank,
                                                bool with_r)
{
    constexpr uint32_t CB = BF ? INV16_BYTES : INV_BYTES;
    mbar_arrive_expect_tx(bar, CB + (with_r ? R_BYTES : 0u));
    bulk_copy_g2s(stage, A.inv + (size_t)gbank * CB, CB, bar);
    if(with_r)
        bulk_copy_g2s(stage + CB, A.R + (size_t)gbank * (BANK * 3), R_BYTES, bar);
}

// Z of one bank from its staged inverse and residual (the whole warp)
template <bool BF>
__device__ __forceinline__ void bank_product(const ApplyArgs& A, unsigned char* stage, int64_t gbank, bool use32, int lane)
{
    constexpr uint32_t CB = BF ? INV16_BYTES : INV_BYTES;
    const float(*s_r)[3] = reinterpret_cast<const float(*)[3]>(stage + CB);
    float* Zb            = A.Z + gbank * (BANK * 3);
    if(BF && !use32)
        cluster_product_mma(stage, &s_r[0][0], lane, Zb);
    else
    {
        float        out[3];
        const float* Mc = use32 ? A.inv32 + (size_t)gbank * SYM * 9 : reinterpret_cast<const float*>(stage);
        cluster_product(Mc, s_r, lane, out);
        if(lane < 16)
        {
            Zb[3 * lane]     = out[0];
            Zb[3 * lane + 1] = out[1];
            Zb[3 * lane + 2] = out[2];
        }
    }
}

// a[c] = the sum of the entries b, b + step, .. < e, in that order, AHEAD of
// them fetched together
__device__ __forceinline__ void sum_entries(const double* part, int b, int e, int step, double a[3])
{
    constexpr int AHEAD = 4;
    a[0] = a[1] = a[2] = 0.0;
    for(int k = b; k < e; k += AHEAD * step)
    {
        double v[AHEAD][3];
#pragma unroll
        for(int j = 0; j < AHEAD; ++j)
#pragma unroll
            for(int c = 0; c < 3; ++c)
                v[j][c] = k + j * step < e ? __ldcg(part + 3 * (int64_t)(k + j * step) + c) : 0.0;
#pragma unroll
        for(int j = 0; j < AHEAD; ++j)
#pragma unroll
            for(int c = 0; c < 3; ++c)
                a[c] += v[j][c];
    }
}

// the entries of a coarse bank's nodes: lanes 2n and 2n + 1 get node n's
__device__ __forceinline__ int2 bank_entries(const ApplyArgs& A, int64_t gbank, int lane)
{
    const int32_t* st = A.part_start + (gbank - A.g2) * BANK + (lane >> 1);
    return make_int2(__ldg(st), __ldg(st + 1));
}

// The residual of a coarse bank (level 2 up) from the blocks' partial sums, in
// a fixed order, to R and the staged slice in FP32. A node has one entry per
// 256 slots under it: about 1 at level 2, 16 at level 3, 256 at level 4. All
// nodes at once, two lanes each in a full bank, up to the whole warp for a single
// node (upper levels have few, with many entries). be: bank_entries
__device__ __forceinline__ void take_coarse(const ApplyArgs& A, int64_t gbank, int2 be, float* s_r, int lane)
{
    const int nodes = __popc(__ballot_sync(0xffffffffu, be.x < be.y)) / 2;  // the level's last bank may not be full
    const int lanes = nodes > 8 ? 2 : (nodes > 4 ? 4 : (nodes > 2 ? 8 : (nodes > 1 ? 16 : 32)));
    const int node  = lane / lanes;
    const int b = __shfl_sync(0xffffffffu, be.x, 2 * node), e = __shfl_sync(0xffffffffu, be.y, 2 * node);
    double    a[3];
    sum_entries(A.part, b + lane % lanes, e, lanes, a);
    for(int o = lanes / 2; o > 0; o >>= 1)
#pragma unroll
        for(int c = 0; c < 3; ++c)
            a[c] += __shfl_xor_sync(0xffffffffu, a[c], o);
    for(int i = 3 * nodes + lane; i < BANK * 3; i += 32)
        s_r[i] = 0.0f;
    if(node < nodes && lane % lanes == 0)
#pragma unroll
        for(int c = 0; c < 3; ++c)
        {
            const float v       = (float)a[c];
            s_r[3 * node + c] = v;
            A.R[gbank * (BANK * 3) + 3 * node + c] = v;
        }
    __syncwarp();
}

// A bank of level 3 up with its sums by a whole CTA: its entries, one per 256
// slots under each node, come into shared memory by bulk copies of `room` bytes
// at most and are added by 8 (16 nodes) to 128 threads (one node) per node. Beside
// the fine level's copies, which fill the memory system from the first
// microsecond, every dependent round of loads takes 2-4 us: with plain loads, 4 or
// 9 ahead per lane of one warp, an iteration took 1.4 us (88,641 vertices) to 2.8
// us (551,368) longer; with these the apply takes what it took with reductions
// (10.6 us against 10.5, 88,641 vertices, caches flushed). The product is warp 0's; the others return at the end.
// copies: two free barriers (the bank's inverse, the entries); stage: the bank's;
// s_sum: [16][WARPS][3] doubles.
template <bool BF, int WARPS>
__device__ __forceinline__ void heavy_bank(const ApplyArgs& A, int64_t gbank, const int* stop, unsigned char* stage,
                                           unsigned char* entries, uint32_t room, uint64_t* copies, double* s_sum)
{
    constexpr uint32_t CB = BF ? INV16_BYTES : INV_BYTES;
    constexpr uint32_t ENTRY = 3 * sizeof(double);
    const int          t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int2         be = bank_entries(A, gbank, lane);  // on its way with the flag
    if(stop && *stop)
        return;
    const int nodes = __popc(__ballot_sync(0xffffffffu, be.x < be.y)) / 2;
    int       pow2 = 1;
    while(pow2 < nodes)
        pow2 <<= 1;
    const int G = WARPS * 32 / pow2, node = t / G, sub = t % G;  // threads of a node
    const int b = __shfl_sync(0xffffffffu, be.x, 2 * node), e = __shfl_sync(0xffffffffu, be.y, 2 * node);
    const int first = __shfl_sync(0xffffffffu, be.x, 0) & ~1;  // (copies start and end at even entries: 16 bytes)
    const int last  = __shfl_sync(0xffffffffu, be.y, 2 * max(nodes - 1, 0));
    const int step  = (int)(room / ENTRY) & ~1;
    auto      issue = [&](int c)
    {
        const uint32_t bytes = ENTRY * (uint32_t)min(step, (last - c + 1) & ~1);
        mbar_arrive_expect_tx(&copies[1], bytes);
        bulk_copy_g2s(entries, A.part + 3 * (int64_t)c, bytes, &copies[1]);
    };
    if(t == 0)
    {
        if(first < last)
            issue(first);
        issue_bank_copy<BF>(stage, &copies[0], A, gbank, false);
    }
    double a[3] = {0.0, 0.0, 0.0};
    bool     ok   = true;
    uint32_t phase = 0;
    __syncthreads();  // the barriers of warp 0, initialised by its lane 0
    for(int c = first; c < last; c += step, phase ^= 1u)
    {
        ok = __syncthreads_and(mbar_wait(&copies[1], phase, A.err, DERR_TMA_TIMEOUT));
        if(!ok)  // once more, for the copy to end before the block goes on
        {
            mbar_wait(&copies[1], phase, nullptr, 0);
            break;
        }
        const double* p  = reinterpret_cast<const double*>(entries);
        const int     to = min(e, c + step);
        for(int k = b + sub + (c > b + sub ? (c - b - sub + G - 1) / G * G : 0); k < to; k += G)
#pragma unroll
            for(int q = 0; q < 3; ++q)
                a[q] += p[3 * (k - c) + q];
        __syncthreads();  // the entries are read
        if(t == 0 && c + step < last)
        {
            fence_proxy_async_smem();
            issue(c + step);
        }
    }
    const int part = min(G, 32);
    for(int o = part / 2; o > 0; o >>= 1)
#pragma unroll
        for(int q = 0; q < 3; ++q)
            a[q] += __shfl_xor_sync(0xffffffffu, a[q], o);
    if(node < nodes && lane % part == 0)
#pragma unroll
        for(int q = 0; q < 3; ++q)
            s_sum[(node * WARPS + sub / 32) * 3 + q] = a[q];
    fence_proxy_async_smem();  // the entries are read: the warps' own copies may follow
    __syncthreads();
    if(w != 0)
        return;
    float* s_r = reinterpret_cast<float*>(stage + CB);
    for(int i = lane; i < BANK * 3; i += 32)
    {
        const int m = i / 3, c = i - 3 * m;
        double    v = 0.0;
        if(m < nodes)
            for(int q = 0; q < (G + 31) / 32; ++q)
                v += s_sum[(m * WARPS + q) * 3 + c];
        s_r[i]                      = (float)v;
        A.R[gbank * (BANK * 3) + i] = (float)v;
    }
    const bool here = mbar_wait(&copies[0], 0, A.err, DERR_TMA_TIMEOUT);
    if(!here)
        mbar_wait(&copies[0], 0, nullptr, 0);
    if(!__all_sync(0xffffffffu, here && ok))
        return;
    __syncwarp();  // every lane's residuals, for the others in the product
    bank_product<BF>(A, stage, gbank, BF && A.stiff != nullptr && A.stiff[gbank] != 0, lane);
}

// The banks handled by one warp (warp gw of W). The list: the banks from level
// 3 up (global banks g3 ..; skipped when CTAs of their own have them), of level
// 2, of level 0, of level 1. A copy wait that runs out sets the error flag,
// drains the warp's copies in flight and ends the warp.
template <bool BF, int NST>
__device__ __forceinline__ void apply_banks(int gw, int W, int lane, const ApplyArgs& A, const int* stop,
                                            unsigned char* s_stage, uint64_t* s_bar)
{
    constexpr uint32_t SB   = stage_bytes<BF>();
    constexpr uint32_t CB   = BF ? INV16_BYTES : INV_BYTES;
    const int          n    = A.n2 + A.n0 + A.n1 - A.heavy;
    const int          mine = gw < n ? (n - 1 - gw) / W + 1 : 0;
    auto               bank_of = [&](int j) -> int64_t
    {
        const int i = A.heavy + gw + j * W;
        if(i >= A.n2)
            return i - A.n2 < A.n0 ? i - A.n2 : (int64_t)A.g1 + (i - A.n2 - A.n0);
        return i < A.n3 ? (int64_t)A.g3 + i : (int64_t)A.g2 + i - A.n3;
    };
    auto coarse = [&](int j) { return A.heavy + gw + j * W < A.n2; };
    auto issue = [&](int j, int slot)
    { issue_bank_copy<BF>(s_stage + slot * SB, &s_bar[slot], A, bank_of(j), !coarse(j)); };
    int2 be = make_int2(0, 0);  // of a coarse bank: the first one's on its way with the flag
    if(mine > 0 && coarse(0))
        be = bank_entries(A, bank_of(0), lane);
    if(stop && *stop)
        return;
    if(lane == 0)
        for(int j = 0; j < mine && j < NST; ++j)
            issue(j, j);
    __syncwarp();
    int j = 0;
    for(; j < mine; ++j)
    {
        const int64_t  gbank = bank_of(j);
        const int      slot  = j % NST;
        const bool     use32 = BF && A.stiff != nullptr && A.stiff[gbank] != 0;
        unsigned char* stage = s_stage + slot * SB;
        if(coarse(j))
        {
            if(j > 0)
                be = bank_entries(A, gbank, lane);
            take_coarse(A, gbank, be, reinterpret_cast<float*>(stage + CB), lane);
        }
        const bool ok = mbar_wait(&s_bar[slot], (uint32_t)((j / NST) & 1), A.err, DERR_TMA_TIMEOUT);
        if(!__all_sync(0xffffffffu, ok))
            break;
        bank_product<BF>(A, stage, gbank, use32, lane);
        __syncwarp();
        if(lane == 0 && j + NST < mine)
        {
            fence_proxy_async_smem();
            issue(j + NST, slot);
        }
    }
    if(j < mine && lane == 0)
        for(int q = j; q < mine && q < j + NST; ++q)
            mbar_wait(&s_bar[q % NST], (uint32_t)((q / NST) & 1), nullptr, 0);
    __syncwarp();
}

// The level-1 sums of a block of rows (in slot order; thread t's slot is its
// row) and their part of the sums of the levels above. s_r: the residuals
// [threads][3]; cm, nl: component mask and level-1 index of the thread's slot
// (cm = 0: none); dst: its level-1 node's entries (MasState::part_dst), needed by
// the components' lowest lanes. R_1 in FP32, summed by the lowest lane in lane
// order. The levels above, whose nodes collect from many blocks, get one FP64
// partial sum per node and block, in a fixed order like the apply's sums of them
// (take_coarse): every level is complete when the kernel is, the same in every
// run. FP64 reductions in L2 (`red`) in their place left the last bits to the
// order of the blocks. A chain of restrictions from level to level inside the
// apply took 25 us (88,641 vertices) to 43 us (551,368, behind the fine level's
// traffic). Whole block; s_lead: [threads][3] floats, s_dst: [threads] int4,
// s_n: [warps].
constexpr int RESTRICT_THREADS = 256;  // slots per block: the entries' unit
template <int THREADS>
__device__ __forceinline__ void restrict_coarse(const float (*s_r)[3], uint32_t cm, int nl, int4 dst, int begin1,
                                                float* __restrict__ R, double* __restrict__ part, float (*s_lead)[3],
                                                int4* s_dst, int* s_n)
{
    static_assert(THREADS == RESTRICT_THREADS, "the entries are those of blocks of RESTRICT_THREADS slots");
    const int      t = threadIdx.x, lane = t & 31, w = t >> 5, sub = t & 15;
    const bool     lead = cm != 0 && (cm & ((1u << sub) - 1u)) == 0;
    const unsigned all  = __ballot_sync(0xffffffffu, lead);
    if(lane == 0)
        s_n[w] = __popc(all);
    float s0 = 0.f, s1 = 0.f, s2 = 0.f;
    if(lead)
    {
        const float(*b)[3] = s_r + (t & ~15);
        for(uint32_t m = cm; m; m &= m - 1)
        {
            const int l = __ffs(m) - 1;
            s0 += b[l][0];
            s1 += b[l][1];
            s2 += b[l][2];
        }
        const int64_t g = (int64_t)begin1 + nl;
        R[3 * g]     = s0;
        R[3 * g + 1] = s1;
        R[3 * g + 2] = s2;
    }
    __syncthreads();
    int at = __popc(all & ((1u << lane) - 1u)), n = 0;
#pragma unroll
    for(int q = 0; q < THREADS / 32; ++q)
    {
        at += q < w ? s_n[q] : 0;
        n += s_n[q];
    }
    if(lead)
    {
        s_lead[at][0] = s0;
        s_lead[at][1] = s1;
        s_lead[at][2] = s2;
        s_dst[at]     = dst;
    }
    __syncthreads();
    // warp lv: level 2 + lv. The block's components have one or two ancestors
    // there: one sum over the warp for each. Beyond 32 components an entry may
    // come up again; the same lanes then add to it.
    static_assert(THREADS >= 128, "a warp per level above 1");
    if(w >= 4)
        return;
    for(int base = 0; base < n; base += 32)
    {
        const int k = base + lane;
        int       e = k < n ? reinterpret_cast<const int*>(s_dst + k)[w] : -1;
        float     v[3] = {0.f, 0.f, 0.f};
        if(k < n)
#pragma unroll
            for(int c = 0; c < 3; ++c)
                v[c] = s_lead[k][c];
        while(true)
        {
            const int best = (int)__reduce_min_sync(0xffffffffu, (unsigned)e);  // -1: the largest
            if(best < 0)
                break;
            const bool in = e >= 0 && (e >> 1) == (best >> 1);  // best: its first component of the block, if here
            double     a[3];
#pragma unroll
            for(int c = 0; c < 3; ++c)
                a[c] = in ? (double)v[c] : 0.0;
#pragma unroll
            for(int o = 16; o > 0; o >>= 1)
#pragma unroll
                for(int c = 0; c < 3; ++c)
                    a[c] += __shfl_xor_sync(0xffffffffu, a[c], o);
            if(lane < 3)
            {
                double* q = part + 3 * (int64_t)(best >> 1) + lane;
                double  d = lane == 0 ? a[0] : (lane == 1 ? a[1] : a[2]);
                if(best & 1)
                    d += *q;
                *q = d;
            }
            if(in)
                e = -1;
        }
    }
}

// the arguments of an apply from the current build (b2s_mas.cu)
ApplyArgs mas_apply_args(b2s_solver* s, bool bf16);
}  // namespace b2s
