// Triplet -> block-upper BSR assembly (deterministic), and the device scan.
//
// Semantics follow MatrixConverter<Float,3>::convert_sym
// (src/backends/cuda/algorithm/details/matrix_converter.inl:1550-1701):
// keep row >= 0 && row <= col, order by (row, col) with ties in source
// order, sum each run. The reference sorts a 64-bit key with CUB and sums
// runs with cross-warp FP64 atomics (rounding-nondeterministic). Here the
// sort is a counting sort on the row followed by an in-warp rank sort of each
// row's (col, source) pairs, and every run is summed by one lane in source
// order -- the pattern is identical, the values are bit-reproducible.
#include "b2s_internal.cuh"

#include <algorithm>

namespace b2s
{
namespace
{
constexpr int SCAN_BLOCK = 256;
constexpr int SCAN_ITEMS = 16;  // elements per thread
constexpr int SCAN_TILE  = SCAN_BLOCK * SCAN_ITEMS;
constexpr int SCAN_DIRECT_TILES = 2048;  // tiles whose sums every block adds up by itself

// block-wide inclusive scan of one int per thread (warp shuffles + smem)
__device__ __forceinline__ int block_inclusive_scan(int v, int* warp_sums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if(lane >= o)
            v += t;
    }
    if(lane == 31)
        warp_sums[warp] = v;
    __syncthreads();
    if(warp == 0)
    {
        int w = (lane < (int)(blockDim.x >> 5)) ? warp_sums[lane] : 0;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            int t = __shfl_up_sync(0xffffffffu, w, o);
            if(lane >= o)
                w += t;
        }
        if(lane < (int)(blockDim.x >> 5))
            warp_sums[lane] = w;
    }
    __syncthreads();
    if(warp > 0)
        v += warp_sums[warp - 1];
    return v;
}

// the sum of each tile
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_sums(const int32_t* __restrict__ in, int64_t n,
                                                          int32_t* __restrict__ tile_sums)
{
    __shared__ int warp_sums[SCAN_BLOCK / 32];
    const int64_t  base = (int64_t)blockIdx.x * SCAN_TILE;
    int            v    = 0;
#pragma unroll
    for(int k = 0; k < SCAN_ITEMS; ++k)
    {
        const int64_t j = base + k * SCAN_BLOCK + threadIdx.x;
        v += j < n ? in[j] : 0;
    }
    v = block_inclusive_scan(v, warp_sums);
    if(threadIdx.x == SCAN_BLOCK - 1)
        tile_sums[blockIdx.x] = v;
}

// out[0 .. n] of one tile, from the tiles before it: their sums (added up by
// every block: at most SCAN_DIRECT_TILES of them) or their scanned offsets.
// out must not alias in.
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_tiles(const int32_t* __restrict__ in, int32_t* __restrict__ out,
                                                           int64_t n, const int32_t* __restrict__ tile_sums,
                                                           const int32_t* __restrict__ tile_offsets)
{
    __shared__ int warp_sums[SCAN_BLOCK / 32], pre_sums[SCAN_BLOCK / 32];
    __shared__ int s_in[SCAN_TILE + SCAN_TILE / 32];  // padded: a thread reads 16 in a row
    __shared__ int s_pre;
    const int64_t  base = (int64_t)blockIdx.x * SCAN_TILE;
    int            p    = 0;
    if(tile_offsets)
        p = threadIdx.x == 0 ? tile_offsets[blockIdx.x] : 0;
    else
        for(int t = threadIdx.x; t < (int)blockIdx.x; t += SCAN_BLOCK)
            p += tile_sums[t];
#pragma unroll
    for(int k = 0; k < SCAN_ITEMS; ++k)
    {
        const int     i = k * SCAN_BLOCK + threadIdx.x;
        const int64_t j = base + i;
        s_in[i + i / 32] = j < n ? in[j] : 0;
    }
    p = block_inclusive_scan(p, pre_sums);
    if(threadIdx.x == SCAN_BLOCK - 1)
        s_pre = p;
    __syncthreads();
    int local = 0;
#pragma unroll
    for(int k = 0; k < SCAN_ITEMS; ++k)
    {
        const int i = threadIdx.x * SCAN_ITEMS + k;
        local += s_in[i + i / 32];
    }
    const int incl = block_inclusive_scan(local, warp_sums);
    int       run  = s_pre + incl - local;
#pragma unroll
    for(int k = 0; k < SCAN_ITEMS; ++k)
    {
        const int i = threadIdx.x * SCAN_ITEMS + k, v = s_in[i + i / 32];
        s_in[i + i / 32] = run;
        run += v;
    }
    if(threadIdx.x == SCAN_BLOCK - 1 && base + SCAN_TILE >= n)
        out[n] = run;
    __syncthreads();
#pragma unroll
    for(int k = 0; k < SCAN_ITEMS; ++k)
    {
        const int     i = k * SCAN_BLOCK + threadIdx.x;
        const int64_t j = base + i;
        if(j < n)
            out[j] = s_in[i + i / 32];
    }
}
}  // namespace

// Exclusive scan of n int32 into out[0..n] (out[n] = total); in != out. One
// launch up to SCAN_TILE elements, two up to SCAN_DIRECT_TILES tiles (every
// block adds the sums before its own: 8 M elements at most 8 loads a thread),
// beyond that the tile sums are scanned first.
void exclusive_scan(b2s_solver* s, const int32_t* in, int32_t* out, int64_t n, DBuf<int32_t>& tmp)
{
    B2S_REQUIRE(n <= 0 || in + n <= out || out + n + 1 <= in, B2S_ERR_STATE, "exclusive_scan in place");
    cudaStream_t st = s->stream;
    if(n <= 0)
    {
        B2S_CUDA(cudaMemsetAsync(out, 0, sizeof(int32_t), st));
        return;
    }
    auto    tiles_of = [](int64_t m) { return (m + SCAN_TILE - 1) / SCAN_TILE; };
    int64_t need = 0;
    for(int64_t m = n; tiles_of(m) > 1; m = tiles_of(m))
        need += 2 * tiles_of(m) + 1;
    tmp.resize(need + 1, 1.5);
    auto scan = [&](auto& self, const int32_t* src, int32_t* dst, int64_t m, int32_t* room) -> void
    {
        const int64_t t    = tiles_of(m);
        int32_t*      sums = room;
        int32_t*      offs = nullptr;
        if(t > 1)
        {
            k_scan_sums<<<(unsigned)t, SCAN_BLOCK, 0, st>>>(src, m, sums);
            B2S_CHECK_LAUNCH();
            if(t > SCAN_DIRECT_TILES)
            {
                offs = room + t;
                self(self, sums, offs, t, room + 2 * t + 1);
            }
        }
        k_scan_tiles<<<(unsigned)t, SCAN_BLOCK, 0, st>>>(src, dst, m, sums, offs);
        B2S_CHECK_LAUNCH();
    };
    scan(scan, in, out, n, tmp.data());
}

namespace
{
constexpr int ASM_BLOCK = 256;
constexpr int ROW_CAP   = 256;  // (col, src) pairs per row that one warp sorts in registers

// The triplets of a warp mostly come from one or two elements, so few
// distinct rows: the lanes holding the same row (__match_any_sync) add their
// count with one atomic by the lowest of them. The loops step warp by warp so
// all lanes take part in every match.
__global__ void k_count_rows(const int32_t* __restrict__ rows, const int32_t* __restrict__ cols, int64_t T,
                             int32_t nb, int32_t* __restrict__ row_count, int* err)
{
    const int     lane   = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for(int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < T; base += stride)
    {
        const int64_t t = base + lane;
        int32_t       r = -1, c = 0;
        if(t < T)
        {
            r = rows[t];
            c = cols[t];
        }
        bool ok = t < T && r >= 0 && r <= c;
        if(ok && c >= nb)
        {
            atomicOr(err, DERR_TRIPLET_INDEX);
            ok = false;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, ok ? r : -1 - lane);
        if(ok && lane == __ffs(peers) - 1)
            atomicAdd(&row_count[r], __popc(peers));
    }
}

// (column, source) of every kept triplet into its row's bucket; the lanes of
// a row take consecutive places from one atomic of the lowest of them, which
// counts row_count back down
__global__ void k_scatter_rows(const int32_t* __restrict__ rows, const int32_t* __restrict__ cols, int64_t T,
                               int32_t nb, const int32_t* __restrict__ row_start, int32_t* __restrict__ row_count,
                               int2* __restrict__ bucket, int* err)
{
    const int     lane   = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for(int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < T; base += stride)
    {
        const int64_t t = base + lane;
        int32_t       r = -1, c = 0;
        if(t < T)
        {
            r = rows[t];
            c = cols[t];
        }
        const bool ok  = t < T && r >= 0 && r <= c && c < nb;
        int32_t    beg = 0, len = 0;
        if(ok)
        {
            beg = row_start[r];
            len = row_start[r + 1] - beg;
        }
        const unsigned peers  = __match_any_sync(0xffffffffu, ok ? r : -1 - lane);
        const int      leader = __ffs(peers) - 1;
        int32_t        pos    = 0;
        if(ok && lane == leader)
            pos = atomicSub(&row_count[r], __popc(peers)) - __popc(peers);
        pos = __shfl_sync(0xffffffffu, pos, leader);
        if(!ok)
            continue;
        const int32_t k = pos + __popc(peers & ((1u << lane) - 1u));
        if(k < 0 || k >= len)
        {
            atomicOr(err, DERR_ROW_OVERFLOW);
            continue;
        }
        bucket[beg + k] = make_int2(c, (int32_t)t);
    }
}

// One row of at most 32 K pairs by one warp, K keys per lane (positions
// j * 32 + lane): bitonic sort in registers, partners 32 apart or more in the
// same lane, the others by shuffles; padding = max key. Then the sources in
// order and the runs over the row's pairs. Returns the number of runs.
template <int K>
__device__ __forceinline__ int sort_row(int2* bucket, int32_t* __restrict__ sorted_src, int32_t beg, int32_t L, int lane)
{
    uint64_t key[K];
#pragma unroll
    for(int j = 0; j < K; ++j)
    {
        const int p = j * 32 + lane;
        key[j]      = ~0ull;
        if(p < L)
        {
            const int2 q = bucket[beg + p];
            key[j]       = ((uint64_t)(uint32_t)q.x << 32) | (uint64_t)(uint32_t)q.y;
        }
    }
#pragma unroll
    for(int k = 2; k <= 32 * K; k <<= 1)
#pragma unroll
        for(int s = k >> 1; s > 0; s >>= 1)
        {
            if(s >= 32)
            {
#pragma unroll
                for(int j = 0; j < K; ++j)
                {
                    const int o = j ^ (s / 32);
                    if(o > j)
                    {
                        const bool     up = ((j * 32) & k) == 0;  // k > s >= 32: the lane does not matter
                        const uint64_t lo = key[j] < key[o] ? key[j] : key[o];
                        const uint64_t hi = key[j] < key[o] ? key[o] : key[j];
                        key[j]            = up ? lo : hi;
                        key[o]            = up ? hi : lo;
                    }
                }
            }
            else
            {
#pragma unroll
                for(int j = 0; j < K; ++j)
                {
                    const int      p     = j * 32 + lane;
                    const uint64_t other = __shfl_xor_sync(0xffffffffu, key[j], s);
                    const bool     keep_min = ((p & s) == 0) == ((p & k) == 0);
                    key[j] = keep_min ? (key[j] < other ? key[j] : other) : (key[j] < other ? other : key[j]);
                }
            }
        }
    __syncwarp();  // every lane holds its pairs: the runs may replace them
    int      uniq = 0;
    uint64_t last = ~0ull;  // key at the position before this group's first
#pragma unroll
    for(int j = 0; j < K; ++j)
    {
        const int      p    = j * 32 + lane;
        const uint64_t up1  = __shfl_up_sync(0xffffffffu, key[j], 1);
        const uint64_t prev = lane > 0 ? up1 : last;
        last                = __shfl_sync(0xffffffffu, key[j], 31);
        const bool     head = p < L && (p == 0 || (prev >> 32) != (key[j] >> 32));
        const unsigned hm   = __ballot_sync(0xffffffffu, head);
        if(p < L)
            sorted_src[beg + p] = (int32_t)(key[j] & 0xFFFFFFFFull);
        if(head)
            bucket[beg + uniq + __popc(hm & ((1u << lane) - 1u))] = make_int2((int32_t)(key[j] >> 32), beg + p);
        uniq += __popc(hm);
    }
    return uniq;
}

// One warp per row: the row's (col, src) pairs sorted; out go the sources in
// that order (sorted_src) and, in place of the row's pairs from its first on,
// each distinct column with the position of its first source, and their number
// (uniq_count). The columns of all pairs are not written: marking the
// runs from them in a second pass cost 126 MB out and in on 31 M triplets
// (sort + mark 544 us; 454 now). Rows of more than 64 pairs are only listed
// here: four or eight keys per lane would cost the common rows registers (the
// whole assembly of the 31 M triplets 1.66 -> 1.68 ms).
__global__ void __launch_bounds__(ASM_BLOCK) k_sort_rows(int32_t nb, const int32_t* __restrict__ row_start,
                                                         int2* bucket,
                                                         int32_t* __restrict__ sorted_src,
                                                         int32_t* __restrict__ uniq_count, int32_t* long_rows,
                                                         int32_t* n_long, int32_t* n_mid)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int warps_total = gridDim.x * (ASM_BLOCK / 32);
    for(int32_t r = blockIdx.x * (ASM_BLOCK / 32) + w; r < nb; r += warps_total)
    {
        const int32_t beg = row_start[r], L = row_start[r + 1] - beg;
        int           uniq;
        if(L <= 32)
            uniq = sort_row<1>(bucket, sorted_src, beg, L, lane);
        else if(L <= 64)
            uniq = sort_row<2>(bucket, sorted_src, beg, L, lane);
        else
        {
            // more keys per lane, or a CTA per row: k_sort_long_rows
            if(lane == 0)
            {
                if(L > ROW_CAP)
                    long_rows[atomicAdd(n_long, 1)] = (int32_t)r;
                else
                    long_rows[nb - 1 - atomicAdd(n_mid, 1)] = (int32_t)r;
            }
            continue;
        }
        if(lane == 0)
            uniq_count[r] = uniq;
    }
}

// The rows listed by k_sort_rows. Up to ROW_CAP pairs, most rows of a coarse
// MAS level: a warp per row, four or eight keys per lane (ranked before by
// counting the smaller pairs of the row for every pair; MAS build of 551,368
// vertices 1.72 -> 1.64 ms). Longer (e.g. an affine body touched by
// thousands of cloth vertices): one CTA per row (persistent over the
// list). The keys (column << 32 | source; unique) are sorted LONG_TILE at a
// time in shared memory (bitonic); with several tiles every key's rank is its
// place in its tile plus a binary search in each of the others. Counting the
// smaller keys of the whole row for every key, O(L^2), took 25 us a launch on
// the rows of 25 bodies under a cloth of 128^2 vertices (1,200 pairs; 9 us now).
constexpr int LONG_THREADS = 1024;
constexpr int LONG_TILE    = 4096;

__device__ __forceinline__ uint64_t pair_key(int2 q)
{
    return ((uint64_t)(uint32_t)q.x << 32) | (uint64_t)(uint32_t)q.y;
}

// keys [0, n) of s_key ascending (whole CTA); n <= LONG_TILE, the slots up to
// the next power of two hold ~0
__device__ __forceinline__ void sort_tile(uint64_t* s_key, int n)
{
    int size2 = 32;
    while(size2 < n)
        size2 <<= 1;
    for(int i = n + (int)threadIdx.x; i < size2; i += LONG_THREADS)
        s_key[i] = ~0ull;
    __syncthreads();
    for(int size = 2; size <= size2; size <<= 1)
        for(int stride = size >> 1; stride > 0; stride >>= 1)
        {
            for(int i = threadIdx.x; i < size2 / 2; i += LONG_THREADS)
            {
                const int      lo = 2 * i - (i & (stride - 1));
                const int      hi = lo + stride;
                const bool     up = (lo & size) == 0;
                const uint64_t a = s_key[lo], b = s_key[hi];
                if((a > b) == up)
                {
                    s_key[lo] = b;
                    s_key[hi] = a;
                }
            }
            __syncthreads();
        }
}

__global__ void __launch_bounds__(LONG_THREADS) k_sort_long_rows(int32_t nb, const int32_t* __restrict__ long_rows,
                                                                 const int32_t* __restrict__ n_rows,
                                                                 const int32_t* __restrict__ n_mid,
                                                                 const int32_t* __restrict__ row_start, int2* bucket,
                                                                 int32_t* sorted_col, int32_t* sorted_src,
                                                                 int32_t* __restrict__ uniq_count)
{
    __shared__ uint64_t s_key[LONG_TILE];
    __shared__ int      s_heads[LONG_THREADS / 32];
    // the rows of 65 to 256 pairs (listed from the end), a warp each
    const int lane = threadIdx.x & 31, mid = *n_mid;
    for(int e = blockIdx.x * (LONG_THREADS / 32) + (threadIdx.x >> 5); e < mid; e += gridDim.x * (LONG_THREADS / 32))
    {
        const int32_t r = long_rows[nb - 1 - e], beg = row_start[r], L = row_start[r + 1] - beg;
        const int     u = L <= 128 ? sort_row<4>(bucket, sorted_src, beg, L, lane) :
                                     sort_row<8>(bucket, sorted_src, beg, L, lane);
        if(lane == 0)
            uniq_count[r] = u;
    }
    const int n_long = *n_rows;
    for(int e = blockIdx.x; e < n_long; e += gridDim.x)
    {
        const int32_t r = long_rows[e], beg = row_start[r], L = row_start[r + 1] - beg;
        const bool    many = L > LONG_TILE;
        // sort the tiles (one tile: straight to the result; several: in place)
        for(int t0 = 0; t0 < L; t0 += LONG_TILE)
        {
            const int n = min(LONG_TILE, L - t0);
            __syncthreads();  // the previous tile is written
            for(int k = threadIdx.x; k < n; k += LONG_THREADS)
                s_key[k] = pair_key(bucket[beg + t0 + k]);
            __syncthreads();
            sort_tile(s_key, n);
            for(int k = threadIdx.x; k < n; k += LONG_THREADS)
            {
                const int32_t c = (int32_t)(s_key[k] >> 32), sr = (int32_t)(s_key[k] & 0xFFFFFFFFull);
                if(many)
                    bucket[beg + t0 + k] = make_int2(c, sr);
                else
                {
                    sorted_col[beg + k] = c;
                    sorted_src[beg + k] = sr;
                }
            }
        }
        __syncthreads();
        if(many)
            for(int own = 0; own < L; own += LONG_TILE)
            {
                constexpr int PER = LONG_TILE / LONG_THREADS;
                uint64_t      key[PER];
                int           rank[PER];
#pragma unroll
                for(int j = 0; j < PER; ++j)
                {
                    const int i = own + j * LONG_THREADS + (int)threadIdx.x;
                    key[j]      = i < L ? pair_key(bucket[beg + i]) : ~0ull;
                    rank[j]     = i - own;
                }
                for(int t0 = 0; t0 < L; t0 += LONG_TILE)
                {
                    if(t0 == own)
                        continue;
                    const int n = min(LONG_TILE, L - t0);
                    __syncthreads();  // the previous tile is read
                    for(int k = threadIdx.x; k < n; k += LONG_THREADS)
                        s_key[k] = pair_key(bucket[beg + t0 + k]);
                    __syncthreads();
#pragma unroll
                    for(int j = 0; j < PER; ++j)
                    {
                        int lo = 0, hi = n;
                        while(lo < hi)
                        {
                            const int m = (lo + hi) >> 1;
                            if(s_key[m] < key[j])
                                lo = m + 1;
                            else
                                hi = m;
                        }
                        rank[j] += lo;
                    }
                }
#pragma unroll
                for(int j = 0; j < PER; ++j)
                    if(own + j * LONG_THREADS + (int)threadIdx.x < L)
                    {
                        sorted_col[beg + rank[j]] = (int32_t)(key[j] >> 32);
                        sorted_src[beg + rank[j]] = (int32_t)(key[j] & 0xFFFFFFFFull);
                    }
            }
        __syncthreads();  // the sorted row is visible to the CTA
        // the row's distinct columns, in order
        int before = 0;
        for(int base = 0; base < L; base += LONG_THREADS)
        {
            const int      i    = base + (int)threadIdx.x;
            const int32_t  c    = i < L ? sorted_col[beg + i] : 0;
            const bool     head = i < L && (i == 0 || sorted_col[beg + i - 1] != c);
            const unsigned hm   = __ballot_sync(0xffffffffu, head);
            __syncthreads();  // s_heads of the previous round is read
            if((threadIdx.x & 31) == 0)
                s_heads[threadIdx.x >> 5] = __popc(hm);
            __syncthreads();
            int mine = before;
#pragma unroll
            for(int q = 0; q < LONG_THREADS / 32; ++q)
            {
                mine += q < (int)(threadIdx.x >> 5) ? s_heads[q] : 0;
                before += s_heads[q];
            }
            if(head)
                bucket[beg + mine + __popc(hm & ((1u << (threadIdx.x & 31)) - 1u))] = make_int2(c, beg + i);
        }
        if(threadIdx.x == 0)
            uniq_count[r] = before;
        __syncthreads();  // s_heads and s_key are free for the next row
    }
}

// One warp per row: the row's runs become slots of the block-upper BSR: row,
// column and the position of the first source in the sorted order (run_start;
// run_start[U] = the kept triplets). The stream's padding past U gets row -1 /
// column 0 (never used: every reader checks). Rows of more than ROW_CAP pairs,
// which may have thousands of blocks, are k_mark_long_rows's.
__global__ void __launch_bounds__(ASM_BLOCK) k_mark_runs(int32_t nb, int64_t U, int64_t S,
                                                         const int32_t* __restrict__ row_start,
                                                         const int2* __restrict__ runs,
                                                         const int32_t* __restrict__ rowptr,
                                                         int32_t* __restrict__ out_rows, int32_t* __restrict__ out_cols,
                                                         int32_t* __restrict__ run_start,
                                                         int32_t* __restrict__ diag_index)
{
    // eight lanes per row: a mesh row has about eight blocks
    constexpr int LANES = 8;
    const int     lane = threadIdx.x % LANES, groups = gridDim.x * (ASM_BLOCK / LANES);
    if(blockIdx.x == 0 && threadIdx.x < 32)
    {
        if(U + threadIdx.x < S)
        {
            out_rows[U + threadIdx.x] = -1;
            out_cols[U + threadIdx.x] = 0;
        }
        if(threadIdx.x == 0)
            run_start[U] = row_start[nb];
    }
    for(int32_t r = blockIdx.x * (ASM_BLOCK / LANES) + threadIdx.x / LANES; r < nb; r += groups)
    {
        const int32_t beg = row_start[r], o = rowptr[r], n = rowptr[r + 1] - o;
        if(row_start[r + 1] - beg > ROW_CAP)
            continue;
        int32_t c0 = -1;
        for(int k = lane; k < n; k += LANES)
        {
            const int2 q     = runs[beg + k];
            out_rows[o + k]  = r;
            out_cols[o + k]  = q.x;
            run_start[o + k] = q.y;
            if(k == 0)
                c0 = q.x;
        }
        if(lane == 0)
            diag_index[r] = c0 == r ? o : -1;
    }
}

// the rows listed by k_sort_rows, one CTA per row
__global__ void __launch_bounds__(LONG_THREADS) k_mark_long_rows(const int32_t* __restrict__ long_rows,
                                                                 const int32_t* __restrict__ n_rows,
                                                                 const int32_t* __restrict__ row_start,
                                                                 const int2* __restrict__ runs,
                                                                 const int32_t* __restrict__ rowptr,
                                                                 int32_t* __restrict__ out_rows,
                                                                 int32_t* __restrict__ out_cols,
                                                                 int32_t* __restrict__ run_start,
                                                                 int32_t* __restrict__ diag_index)
{
    const int n_long = *n_rows;
    for(int e = blockIdx.x; e < n_long; e += gridDim.x)
    {
        const int32_t r = long_rows[e], beg = row_start[r], o = rowptr[r], n = rowptr[r + 1] - o;
        for(int k = threadIdx.x; k < n; k += LONG_THREADS)
        {
            const int2 q     = runs[beg + k];
            out_rows[o + k]  = r;
            out_cols[o + k]  = q.x;
            run_start[o + k] = q.y;
            if(k == 0)
                diag_index[r] = q.x == r ? o : -1;
        }
    }
}

// One thread per (unique block, column of its 3x3): the column's 3 values
// summed over the run's sources in source order (the sorted order). The
// three threads of a block read its sources' 72 contiguous bytes together;
// four sources are fetched ahead, the additions stay in order from the first.
// Runs longer than `run_cap` go to long_runs (count, then the blocks) instead.
__global__ void __launch_bounds__(ASM_BLOCK) k_sum_runs(int64_t U, const int32_t* __restrict__ run_start,
                                                         const int32_t* __restrict__ sorted_src,
                                                         const double* __restrict__ src_vals,
                                                         double* __restrict__ out_vals, int64_t S, int run_cap,
                                                         int32_t* long_runs)
{
    for(int64_t t = (int64_t)blockIdx.x * ASM_BLOCK + threadIdx.x; t < 3 * U; t += (int64_t)gridDim.x * ASM_BLOCK)
    {
        const int64_t o = t / 3;
        const int     c = (int)(t - 3 * o);
        const int32_t b = run_start[o], e = run_start[o + 1];
        if(e - b > run_cap)
        {
            if(c == 0)
                long_runs[1 + atomicAdd(long_runs, 1)] = (int32_t)o;
            continue;
        }
        double        acc[3] = {};
        for(int32_t k = b; k < e; k += 4)
        {
            int64_t src[4];
#pragma unroll
            for(int u = 0; u < 4; ++u)
                src[u] = k + u < e ? (int64_t)sorted_src[k + u] : -1;
            double v[4][3];
#pragma unroll
            for(int u = 0; u < 4; ++u)
#pragma unroll
                for(int q = 0; q < 3; ++q)
                    v[u][q] = src[u] >= 0 ? src_vals[src[u] * 9 + 3 * c + q] : 0.0;
#pragma unroll
            for(int u = 0; u < 4; ++u)
                if(src[u] >= 0)
#pragma unroll
                    for(int q = 0; q < 3; ++q)
                        acc[q] = k + u == b ? v[u][q] : acc[q] + v[u][q];
        }
#pragma unroll
        for(int q = 0; q < 3; ++q)
            out_vals[(int64_t)(3 * c + q) * S + o] = acc[q];
    }
}

// The listed long runs (the diagonal blocks of an affine body collect one
// source per contact), one warp each: 4 x 32 sources are gathered together
// (coalesced, 9 doubles each) into shared memory, then lanes 0-8 add their
// component over them, in source order from the first as k_sum_runs does. Its
// one thread per column waited for memory once per four sources.
constexpr int LONG_RUN       = 64;
constexpr int LONG_RUN_WARPS = 4;
__global__ void __launch_bounds__(LONG_RUN_WARPS * 32) k_sum_long_runs(const int32_t* __restrict__ long_runs,
                                                                       const int32_t* __restrict__ run_start,
                                                                       const int32_t* __restrict__ sorted_src,
                                                                       const double* __restrict__ src_vals,
                                                                       double* __restrict__ out_vals, int64_t S)
{
    constexpr int     CH = 128;
    __shared__ double s_v[LONG_RUN_WARPS][CH * 9];
    const int         lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int         n = long_runs[0];
    for(int i = blockIdx.x * LONG_RUN_WARPS + w; i < n; i += gridDim.x * LONG_RUN_WARPS)
    {
        const int64_t o = long_runs[1 + i];
        const int32_t b = run_start[o], e = run_start[o + 1];
        double        acc = 0.0;
        for(int32_t k0 = b; k0 < e; k0 += CH)
        {
            const int m = min(CH, e - k0);
            int       src[CH / 32];
#pragma unroll
            for(int j = 0; j < CH / 32; ++j)
                src[j] = 32 * j + lane < m ? sorted_src[k0 + 32 * j + lane] : -1;
#pragma unroll
            for(int j = 0; j < CH / 32; ++j)
            {
                double v[9];
#pragma unroll
                for(int q = 0; q < 9; ++q)
                {
                    const int t  = 32 * q + lane, k = t / 9;
                    const int sk = __shfl_sync(0xffffffffu, src[j], k);
                    v[q]         = sk >= 0 ? src_vals[(int64_t)sk * 9 + (t - 9 * k)] : 0.0;
                }
#pragma unroll
                for(int q = 0; q < 9; ++q)
                    s_v[w][288 * j + 32 * q + lane] = v[q];
            }
            __syncwarp();
            if(lane < 9)
                for(int k = 0; k < m; ++k)
                    acc = k0 + k == b ? s_v[w][9 * k + lane] : acc + s_v[w][9 * k + lane];
            __syncwarp();
        }
        if(lane < 9)
            out_vals[(int64_t)lane * S + o] = acc;
    }
}

// rank of every block in (column, index) order within its SPMV_TILE-block
// tile: bitonic sort of the unique keys (column << 16 | index) in shared memory
constexpr int RANK_THREADS = 512;
__global__ void __launch_bounds__(RANK_THREADS) k_tile_rank(int64_t U, const int32_t* __restrict__ cols,
                                                            uint16_t* __restrict__ trank)
{
    static_assert(SPMV_TILE <= 65536 && (SPMV_TILE & (SPMV_TILE - 1)) == 0, "tile: power of two <= 2^16");
    __shared__ uint64_t key[SPMV_TILE];
    const int64_t base = (int64_t)blockIdx.x * SPMV_TILE;
    const int64_t rem  = U - base;
    const int     n    = rem < SPMV_TILE ? (int)rem : SPMV_TILE;
    for(int i = threadIdx.x; i < SPMV_TILE; i += RANK_THREADS)
        key[i] = i < n ? ((uint64_t)(uint32_t)cols[base + i] << 16) | (uint64_t)i : ~0ull;
    __syncthreads();
    for(int size = 2; size <= SPMV_TILE; size <<= 1)
        for(int stride = size >> 1; stride > 0; stride >>= 1)
        {
            for(int i = threadIdx.x; i < SPMV_TILE / 2; i += RANK_THREADS)
            {
                const int      lo = 2 * i - (i & (stride - 1));
                const int      hi = lo + stride;
                const bool     up = (lo & size) == 0;
                const uint64_t a = key[lo], b = key[hi];
                if((a > b) == up)
                {
                    key[lo] = b;
                    key[hi] = a;
                }
            }
            __syncthreads();
        }
    for(int i = threadIdx.x; i < n; i += RANK_THREADS)
        trank[base + (int64_t)(key[i] & 0xFFFFu)] = (uint16_t)i;
}

// value planes -> 9 consecutive doubles per block, OUT_BLOCKS blocks per CTA:
// plane reads and block writes both in whole lines through shared memory.
// Bound by HBM, 144 B per block. (One strided copy per component moved 8 bytes
// at a time: 4.1 ms for 4.3 M blocks.)
constexpr int OUT_BLOCKS = 256;
constexpr int OUT_ROOM   = 4096;  // blocks that a read-back to host memory takes at a time, at least
__global__ void __launch_bounds__(OUT_BLOCKS) k_blocks_out(int64_t k0, int64_t n, const double* __restrict__ vals,
                                                           int64_t S, double* __restrict__ out)
{
    __shared__ double s_b[OUT_BLOCKS * 9];
    const int64_t     base = (int64_t)blockIdx.x * OUT_BLOCKS;
    const int         m    = (int)(n - base < OUT_BLOCKS ? n - base : OUT_BLOCKS);
    const int         t    = threadIdx.x;
    if(t < m)
#pragma unroll
        for(int q = 0; q < 9; ++q)
            s_b[9 * t + q] = vals[(int64_t)q * S + k0 + base + t];
    __syncthreads();
    for(int e = t; e < 9 * m; e += OUT_BLOCKS)
        out[9 * base + e] = s_b[e];
}

__global__ void k_publish(const int32_t* nnz, const int* err, const int32_t* n_long, int32_t* info)
{
    info[0] = *nnz;
    info[1] = *err;
    info[2] = *n_long;
}

int asm_grid(int64_t work, int block)
{
    int64_t g = (work + block - 1) / block;
    const int64_t cap = (int64_t)NUM_SMS_HINT * 16;
    if(g > cap)
        g = cap;
    if(g < 1)
        g = 1;
    return (int)g;
}
}  // namespace

void copy_blocks_out(b2s_solver* s, const Matrix& A, double* out)
{
    cudaStream_t st     = s->stream;
    auto         launch = [&](int64_t k0, int64_t n, double* dst)
    {
        k_blocks_out<<<(unsigned)((n + OUT_BLOCKS - 1) / OUT_BLOCKS), OUT_BLOCKS, 0, st>>>(k0, n, A.vals.data(),
                                                                                       A.stride, dst);
        B2S_CHECK_LAUNCH();
    };
    cudaPointerAttributes at{};
    const cudaError_t     e = cudaPointerGetAttributes(&at, out);
    if(e != cudaSuccess)
        cudaGetLastError();  // memory the runtime does not know: plain host memory
    const bool on_device = e == cudaSuccess
                           && ((at.type == cudaMemoryTypeDevice && at.device == s->device)
                               || at.type == cudaMemoryTypeManaged);
    if(on_device)
    {
        launch(0, A.nnz, out);
        return;
    }
    // host (or another device's) memory: in pieces through the assembly's scratch
    // (8 bytes per triplet, OUT_ROOM blocks at least, idle between assemblies: a
    // buffer made for the call took 600 us of a 20,000-block read-back to pinned
    // memory, the nine strided copies before it 264)
    double* const tmp   = reinterpret_cast<double*>(s->asmb.bucket.data());
    const int64_t piece = std::min<int64_t>({A.nnz, (int64_t)(s->asmb.bucket.cap / 9), 1 << 20});
    for(int64_t k = 0; k < A.nnz; k += piece)
    {
        const int64_t n = std::min<int64_t>(piece, A.nnz - k);
        launch(k, n, tmp);
        B2S_CUDA(cudaMemcpyAsync(out + 9 * k, tmp, sizeof(double) * 9 * (size_t)n, cudaMemcpyDefault, st));
    }
}

void assemble_triplets(b2s_solver* s, Matrix& M, int32_t nb, int64_t T, const int32_t* rows, const int32_t* cols,
                       const double* vals)
{
    B2S_REQUIRE(nb >= 0 && T >= 0, B2S_ERR_ARGUMENT, "negative matrix size");
    B2S_REQUIRE(T < (int64_t)INT32_MAX, B2S_ERR_ARGUMENT, "more than 2^31-1 triplets");
    cudaStream_t     st = s->stream;
    AssemblyScratch& w  = s->asmb;
    M.valid             = false;
    M.generation += 1;
    M.nb                = nb;
    // row counts, then the error bits and the numbers of long and of mid rows:
    // one fill
    w.row_count.resize((size_t)nb + 4, 1.25);
    w.row_start.resize((size_t)nb + 1, 1.25);
    int* const     err    = w.row_count.data() + nb + 1;
    int32_t* const n_long_dev = w.row_count.data() + nb + 2;
    int32_t* const n_mid_dev  = w.row_count.data() + nb + 3;
    w.uniq_count.resize((size_t)nb + 1, 1.25);
    M.rowptr.resize((size_t)nb + 1, 1.25);
    M.diag_index.resize((size_t)std::max(nb, 1), 1.25);
    B2S_CUDA(cudaMemsetAsync(w.row_count.data(), 0, sizeof(int32_t) * ((size_t)nb + 4), st));
    if(T > 0)
    {
        w.bucket.resize(std::max<int64_t>(T, 9 * OUT_ROOM), 1.25);
        w.sorted_col.resize(T, 1.25);
        w.sorted_src.resize(T, 1.25);
        k_count_rows<<<asm_grid(T, ASM_BLOCK), ASM_BLOCK, 0, st>>>(rows, cols, T, nb, w.row_count.data(), err);
        B2S_CHECK_LAUNCH();
    }
    exclusive_scan(s, w.row_count.data(), w.row_start.data(), nb, w.scan_tmp);
    if(T > 0)
    {
        k_scatter_rows<<<asm_grid(T, ASM_BLOCK), ASM_BLOCK, 0, st>>>(rows, cols, T, nb, w.row_start.data(),
                                                                     w.row_count.data(), w.bucket.data(), err);
        B2S_CHECK_LAUNCH();
    }
    if(nb > 0)
    {
        w.long_rows.resize((size_t)nb, 1.25);
        k_sort_rows<<<asm_grid((int64_t)nb * 32, ASM_BLOCK), ASM_BLOCK, 0, st>>>(
            nb, w.row_start.data(), w.bucket.data(), w.sorted_src.data(), w.uniq_count.data(), w.long_rows.data(),
            n_long_dev, n_mid_dev);
        B2S_CHECK_LAUNCH();
        // the mid and the long rows (their numbers are read on the device)
        k_sort_long_rows<<<NUM_SMS_HINT * 2, LONG_THREADS, 0, st>>>(
            nb, w.long_rows.data(), n_long_dev, n_mid_dev, w.row_start.data(), w.bucket.data(), w.sorted_col.data(),
            w.sorted_src.data(), w.uniq_count.data());
        B2S_CHECK_LAUNCH();
    }
    exclusive_scan(s, w.uniq_count.data(), M.rowptr.data(), nb, w.scan_tmp);
    // the sizes the host needs, written by the device straight into pinned host
    // memory (a copy to pageable memory is ~9 us each, and a MAS build assembles
    // five coarse levels)
    k_publish<<<1, 1, 0, st>>>(M.rowptr.data() + nb, err, n_long_dev, s->host->info);
    B2S_CHECK_LAUNCH();
    B2S_CUDA(cudaStreamSynchronize(st));
    const int32_t U = s->host->info[0], n_long = s->host->info[2];
    const int     herr = s->host->info[1];
    B2S_REQUIRE(!(herr & DERR_TRIPLET_INDEX), B2S_ERR_ARGUMENT,
                "triplet column index outside [0, n_block_rows)");
    B2S_REQUIRE(!(herr & DERR_ROW_OVERFLOW), B2S_ERR_ARGUMENT,
                "triplet arrays changed during assembly (row bucket overflow)");
    M.nnz    = U;
    M.stride = ((std::max<int64_t>(U, 1) + 15) / 16) * 16;
    M.rows.resize(M.stride, 1.2);
    M.cols.resize(M.stride, 1.2);
    M.vals.resize((size_t)9 * M.stride, 1.2);
    if(nb > 0)
    {
        // slots of the runs, then their sums (values as planes with stride M.stride)
        w.run_start.resize((size_t)U + 1, 1.2);
        k_mark_runs<<<asm_grid((int64_t)nb * 8, ASM_BLOCK), ASM_BLOCK, 0, st>>>(
            nb, U, M.stride, w.row_start.data(), w.bucket.data(), M.rowptr.data(), M.rows.data(), M.cols.data(),
            w.run_start.data(), M.diag_index.data());
        B2S_CHECK_LAUNCH();
        if(n_long > 0)
        {
            k_mark_long_rows<<<std::min(n_long, NUM_SMS_HINT * 2), LONG_THREADS, 0, st>>>(
                w.long_rows.data(), n_long_dev, w.row_start.data(), w.bucket.data(), M.rowptr.data(), M.rows.data(),
                M.cols.data(), w.run_start.data(), M.diag_index.data());
            B2S_CHECK_LAUNCH();
        }
        if(U > 0)
        {
            // one pass in block order (no grid-stride loop): the CTAs in
            // flight cover neighbouring rows, whose sources share cache lines
            // (runs above LONG_RUN are set apart only when there are long
            // rows: elsewhere a run has at most ROW_CAP sources, and a few
            // dozen in the meshes)
            if(n_long > 0)
            {
                w.long_runs.resize((size_t)U + 1, 1.2);
                B2S_CUDA(cudaMemsetAsync(w.long_runs.data(), 0, sizeof(int32_t), st));
            }
            k_sum_runs<<<(unsigned)((3 * (int64_t)U + ASM_BLOCK - 1) / ASM_BLOCK), ASM_BLOCK, 0, st>>>(
                U, w.run_start.data(), w.sorted_src.data(), vals, M.vals.data(), M.stride,
                n_long > 0 ? LONG_RUN : INT32_MAX, w.long_runs.data());
            B2S_CHECK_LAUNCH();
            if(n_long > 0)
            {
                k_sum_long_runs<<<NUM_SMS_HINT, LONG_RUN_WARPS * 32, 0, st>>>(
                    w.long_runs.data(), w.run_start.data(), w.sorted_src.data(), vals, M.vals.data(), M.stride);
                B2S_CHECK_LAUNCH();
            }
        }
    }
    else
    {
        B2S_CUDA(cudaMemsetAsync(M.rows.data(), 0xff, sizeof(int32_t) * M.stride, st));
        B2S_CUDA(cudaMemsetAsync(M.cols.data(), 0, sizeof(int32_t) * M.stride, st));
    }
    M.has_trank = false;  // built when the FP64 SpMV is to run more than once or twice
    M.products  = 0;
    M.valid     = true;
}

void build_tile_ranks(b2s_solver* s, Matrix& M)
{
    M.trank.resize(M.stride, 1.2);
    k_tile_rank<<<(unsigned)((M.nnz + SPMV_TILE - 1) / SPMV_TILE), RANK_THREADS, 0, s->stream>>>(
        M.nnz, M.cols.data(), M.trank.data());
    B2S_CHECK_LAUNCH();
    M.has_trank = true;
}
}  // namespace b2s
