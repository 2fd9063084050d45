// spgemm.cu -- block SpGEMM C = A * B on BSR matrices with 16 x 16 tiles.
//
// Reference path (src/sparse/spgemm/2d/block_spgemm_2d_half_mma.cu):
//   spgemm_symbolic_kernel (:58-86)  per block-row a dense flag array over
//                                    the block columns, then a count;
//   thrust::exclusive_scan (:806)    RowPtrC;
//   cudaMemcpy D2H of nnzC (:808)    so the host can allocate ColIdxC/ValC;
//   spgemm_symbolic_col_kernel (:88-116)  ColIdxC, ascending per row;
//   block_spgemm_2d_half_mma (:171-555)   numeric: per warp, local CSR
//                                    slices, staged exchange, and a linear
//                                    search for each product's C column.
//
// This implementation keeps the same three phases, the same outputs (RowPtrC,
// ColIdxC ascending per row, ValC tiles in ColIdxC order) and the same tile
// layouts (A and B tiles row-major 16 x 16, B used as K x N), re-designed for
// B200 and for large matrices (the reference handles one <= 192^2 block per
// CTA):
//   * symbolic: one warp per block-row builds the row's column set as a
//     bitmap in shared memory (shared atomics), counts it with popc, and the
//     column fill walks the bitmap words in order (ascending by
//     construction);  the scan is a single-CTA in-place scan; no scratch.
//   * numeric: one CTA per block-row of C enumerates the row's products once,
//     groups them by C tile, and its warps take the tiles in turn, each
//     accumulating its products A(i,k) * B(k,j) with two m16n8k16 MMAs (FP32
//     accumulation) in ascending k -- the order of the reference's sparse
//     accumulator.  The column fill can ride along.  No C tile is touched twice,
//     so the kernel writes C once (the HBM floor of the product).  Rows beyond
//     what a CTA stages search each tile's products (column indices sorted
//     ascending, as the reference generator emits them), and so does a warp per
//     C tile where the tile arrays are not 16-byte aligned.
#include <atomic>
#include <cstdint>
#include <mutex>

#include "kami_common.cuh"
#include "launch.cuh"
#include "spgemm_tiles.cuh"

namespace kami {

int fail(int code, const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);

// Grid barriers of the fused symbolic pass: [slot][0] arrivals, [slot][1]
// generation.  Each launch takes the next slot (zeroed on its stream just
// before it), so launches in flight on different streams do not share one.
constexpr int kFuseSlots = 64;
__device__ unsigned int g_spg_bar[kFuseSlots][2];
// device status of the fused pass's bounded barrier waits (read and cleared
// by kami_device_status)
__device__ int g_spg_error = 0;
// Look-back flags of the single-pass symbolic kernel: one 64-bit word per
// chunk of block-rows, [epoch (31 bits) | inclusive (1 bit) | value (32
// bits)].  Each launch takes the next slot and a new epoch, so a word left by
// an earlier launch never reads as ready and nothing is reset between
// launches.
constexpr int kLbSlots = 16;
constexpr int kLbMaxChunks = 16384;
__device__ unsigned long long g_spg_flags[kLbSlots][kLbMaxChunks];

namespace {

using namespace sptile;

constexpr int kBsr = 16;

// ---------------------------------------------------------------------------
// symbolic
// ---------------------------------------------------------------------------
__device__ __forceinline__ void build_row_bitmap(uint32_t *bm, int words, int row, const int *rpa, const int *cia,
                                                 const int *rpb, const int *cib, int lane)
{
    for (int w = lane; w < words; w += 32)
        bm[w] = 0u;
    __syncwarp();
    const int a0 = rpa[row], a1 = rpa[row + 1];
    for (int e = a0 + lane; e < a1; e += 32)
    {
        const int k = cia[e];
        const int b1 = rpb[k + 1];
        for (int b = rpb[k]; b < b1; ++b)
        {
            const int c = cib[b];
            atomicOr(&bm[c >> 5], 1u << (c & 31));
        }
    }
    __syncwarp();
}

__global__ void spgemm_count_kernel(int mb, int nb, const int *rpa, const int *cia, const int *rpb, const int *cib,
                                    int *rpc)
{
    extern __shared__ uint32_t bm_all[];
    wait_for_previous();
    const int words = (nb + 31) >> 5;
    const int wpc = blockDim.x >> 5;
    const int lane = threadIdx.x & 31;
    uint32_t *bm = bm_all + (threadIdx.x >> 5) * words;
    for (int row = blockIdx.x * wpc + (threadIdx.x >> 5); row < mb; row += gridDim.x * wpc)
    {
        build_row_bitmap(bm, words, row, rpa, cia, rpb, cib, lane);
        int cnt = 0;
        for (int w = lane; w < words; w += 32)
            cnt += __popc(bm[w]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0)
            rpc[row] = cnt;
        __syncwarp();
    }
}

// In-place exclusive scan of rpc[0..n-1] by one CTA of 1024 threads; the
// total lands in rpc[n].
__global__ void __launch_bounds__(1024) spgemm_scan_kernel(int n, int *rpc)
{
    __shared__ int warp_sums[32];
    __shared__ int carry_s;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    wait_for_previous();
    if (t == 0)
        carry_s = 0;
    __syncthreads();
    for (int base = 0; base < n; base += 1024)
    {
        const int i = base + t;
        const int v = i < n ? rpc[i] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o)
                x += y;
        }
        if (lane == 31)
            warp_sums[wid] = x;
        __syncthreads();
        if (wid == 0)
        {
            int s = warp_sums[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o)
                    s += y;
            }
            warp_sums[lane] = s; // inclusive over warps
        }
        __syncthreads();
        const int carry = carry_s;
        const int incl = x + (wid > 0 ? warp_sums[wid - 1] : 0);
        if (i < n)
            rpc[i] = carry + incl - v;
        __syncthreads();
        if (t == 1023)
            carry_s = carry + incl;
        __syncthreads();
    }
    if (t == 0)
        rpc[n] = carry_s;
}

__global__ void spgemm_colfill_kernel(int mb, int nb, const int *__restrict__ rpa, const int *__restrict__ cia,
                                      const int *__restrict__ rpb, const int *__restrict__ cib,
                                      const int *__restrict__ rpc, int *__restrict__ cic, int64_t cap)
{
    extern __shared__ uint32_t bm_all[];
    const int words = (nb + 31) >> 5;
    const int wpc = blockDim.x >> 5;
    const int lane = threadIdx.x & 31;
    uint32_t *bm = bm_all + (threadIdx.x >> 5) * words;
    for (int row = blockIdx.x * wpc + (threadIdx.x >> 5); row < mb; row += gridDim.x * wpc)
    {
        build_row_bitmap(bm, words, row, rpa, cia, rpb, cib, lane);
        int out = rpc[row];
        for (int w0 = 0; w0 < words; w0 += 32)
        {
            const int w = w0 + lane;
            uint32_t bits = w < words ? bm[w] : 0u;
            const int c = __popc(bits);
            int pre = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, pre, o);
                if (lane >= o)
                    pre += y;
            }
            int pos = out + pre - c;
            while (bits)
            {
                const int b = __ffs(bits) - 1;
                if (pos < cap) // entries beyond the caller's capacity are not written
                    cic[pos] = w * 32 + b;
                ++pos;
                bits &= bits - 1;
            }
            out += __shfl_sync(0xffffffffu, pre, 31);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// The symbolic pass in ONE launch: count, scan and column fill as phases of a
// cooperative persistent kernel, separated by grid barriers (the reference
// runs three launches with a device-to-host copy of nnzC between them,
// block_spgemm_2d_half_mma.cu:805-812).  A cooperative launch keeps every CTA
// resident, so the barrier cannot wait for a CTA that never runs; its waits
// are bounded all the same, and a timeout sets g_spg_error and ends the CTA.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t spg_globaltimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Every CTA of the grid arrives; returns false (block-uniform) on a timeout.
__device__ __forceinline__ bool spg_grid_barrier(unsigned int *bar, uint64_t limit_ns)
{
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0)
    {
        volatile unsigned int *gen = bar + 1;
        const unsigned int g0 = *gen;
        __threadfence(); // the generation read and this CTA's writes precede its arrival
        if (atomicAdd(bar, 1u) == gridDim.x - 1)
        {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        }
        else
        {
            const uint64_t t0 = spg_globaltimer();
            while (*gen == g0)
            {
                if (spg_globaltimer() - t0 > limit_ns)
                {
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
    }
    return __syncthreads_and(ok) != 0;
}

// In-place exclusive scan of rpc[0..n-1] by the calling CTA; total in rpc[n].
__device__ __forceinline__ void spg_block_scan(int n, int *__restrict__ rpc)
{
    __shared__ int warp_sums[32];
    __shared__ int carry_s;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
    if (t == 0)
        carry_s = 0;
    __syncthreads();
    for (int base = 0; base < n; base += blockDim.x)
    {
        const int i = base + t;
        const int v = i < n ? rpc[i] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o)
                x += y;
        }
        if (lane == 31)
            warp_sums[wid] = x;
        __syncthreads();
        if (wid == 0)
        {
            int sum = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o)
                    sum += y;
            }
            if (lane < nw)
                warp_sums[lane] = sum; // inclusive over warps
        }
        __syncthreads();
        const int carry = carry_s;
        const int incl = x + (wid > 0 ? warp_sums[wid - 1] : 0);
        if (i < n)
            rpc[i] = carry + incl - v;
        __syncthreads();
        if (t == (int)blockDim.x - 1)
            carry_s = carry + incl;
        __syncthreads();
    }
    if (t == 0)
        rpc[n] = carry_s;
}

// keep_rows > 0: every warp holds at most keep_rows block-rows and keeps
// each row's bitmap in shared memory from phase 1 to phase 3 (the column fill
// then re-reads neither A's row nor B's rows); 0: one bitmap per warp,
// rebuilt in phase 3.
__global__ void spgemm_symbolic_fused_kernel(int mb, int nb, const int *__restrict__ rpa,
                                             const int *__restrict__ cia, const int *__restrict__ rpb,
                                             const int *__restrict__ cib, int *__restrict__ rpc,
                                             int *__restrict__ cic, int64_t cap, unsigned int *bar,
                                             uint64_t limit_ns, int keep_rows)
{
    extern __shared__ uint32_t bm_all[];
    const int words = (nb + 31) >> 5;
    const int wpc = blockDim.x >> 5;
    const int lane = threadIdx.x & 31;
    const int keep = keep_rows > 0;
    uint32_t *bm_warp = bm_all + (size_t)(threadIdx.x >> 5) * (keep ? keep_rows : 1) * words;
    // phase 1: nnz of every C block-row
    int r = 0;
    for (int row = blockIdx.x * wpc + (threadIdx.x >> 5); row < mb; row += gridDim.x * wpc, ++r)
    {
        uint32_t *bm = bm_warp + (keep ? r * words : 0);
        build_row_bitmap(bm, words, row, rpa, cia, rpb, cib, lane);
        int cnt = 0;
        for (int w = lane; w < words; w += 32)
            cnt += __popc(bm[w]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0)
            rpc[row] = cnt;
        __syncwarp();
    }
    if (!spg_grid_barrier(bar, limit_ns))
    {
        if (threadIdx.x == 0)
            atomicExch(&g_spg_error, 1);
        return;
    }
    // phase 2: exclusive scan into RowPtrC (one CTA; the others wait)
    if (blockIdx.x == 0)
        spg_block_scan(mb, rpc);
    if (!spg_grid_barrier(bar, limit_ns))
    {
        if (threadIdx.x == 0)
            atomicExch(&g_spg_error, 2);
        return;
    }
    if (cap == 0)
        return;
    // phase 3: ColIdxC, ascending per block-row, up to the capacity
    r = 0;
    for (int row = blockIdx.x * wpc + (threadIdx.x >> 5); row < mb; row += gridDim.x * wpc, ++r)
    {
        uint32_t *bm = bm_warp + (keep ? r * words : 0);
        if (!keep)
            build_row_bitmap(bm, words, row, rpa, cia, rpb, cib, lane);
        int out = rpc[row];
        for (int w0 = 0; w0 < words; w0 += 32)
        {
            const int w = w0 + lane;
            uint32_t bits = w < words ? bm[w] : 0u;
            const int c = __popc(bits);
            int pre = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, pre, o);
                if (lane >= o)
                    pre += y;
            }
            int pos = out + pre - c;
            while (bits)
            {
                const int b = __ffs(bits) - 1;
                if (pos < cap)
                    cic[pos] = w * 32 + b;
                ++pos;
                bits &= bits - 1;
            }
            out += __shfl_sync(0xffffffffu, pre, 31);
        }
        __syncwarp();
    }
}


// ---------------------------------------------------------------------------
// The symbolic pass in one launch and one pass: chunk c of block-rows (R
// consecutive rows, c = blockIdx.x, + gridDim.x, ...) is counted by its CTA,
// which publishes the chunk's total, finds the exclusive prefix of the
// chunks before it by a decoupled look-back over their flags (a chunk's flag
// carries its own total, or the inclusive prefix once its CTA found it), writes
// RowPtrC for its rows and fills their ColIdxC.  No grid barrier: a chunk's
// fill starts as soon as its prefix is known.  The launch is cooperative, so
// every chunk's CTA is resident and a look-back never waits for a CTA that
// does not run; the waits are bounded all the same (a timeout sets
// g_spg_error).
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long lb_word(unsigned epoch, bool incl, int value)
{
    return ((unsigned long long)epoch << 33) | ((unsigned long long)incl << 32) | (uint32_t)value;
}

// Exclusive prefix of chunk c (c > 0), by warp 0 of its CTA: lane l reads the
// flag of chunk p - l for a window of 32 predecessors; the window's sum up to
// and including the nearest inclusive flag ends the walk.  Returns false on
// a timeout.
__device__ __forceinline__ bool lb_prefix(const unsigned long long *flags, int c, unsigned epoch, uint64_t limit_ns,
                                          int lane, int *prefix)
{
    int acc = 0;
    int p = c - 1;
    const uint64_t t0 = spg_globaltimer();
    while (p >= 0)
    {
        const int q = p - lane;
        unsigned long long w = 0;
        bool ready = true;
        if (q >= 0)
        {
            w = *reinterpret_cast<const volatile unsigned long long *>(&flags[q]);
            ready = (unsigned)(w >> 33) == epoch;
        }
        const bool incl = q >= 0 && ready && ((w >> 32) & 1ull);
        const unsigned incl_mask = __ballot_sync(0xffffffffu, incl);
        // lanes up to the nearest inclusive flag (or all 32 / down to chunk 0)
        const int last = incl_mask ? __ffs(incl_mask) - 1 : 31;
        const bool need = lane <= last && q >= 0;
        if (!__all_sync(0xffffffffu, !need || ready))
        {
            if (spg_globaltimer() - t0 > limit_ns)
                return false;
            __nanosleep(32);
            continue; // a predecessor has not published yet: read the window again
        }
        int v = need ? (int)(uint32_t)w : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_xor_sync(0xffffffffu, v, o);
        acc += v;
        if (incl_mask)
            break;
        p -= 32;
    }
    *prefix = acc;
    return true;
}

// rows_per_warp (k): each warp takes rows r0 + w + wpc t of its chunk (R =
// wpc k rows); with k = 1 the row's bitmap stays in shared memory from the
// count to the fill, otherwise it is rebuilt for the fill.
__global__ void spgemm_symbolic_lookback_kernel(int mb, int nb, const int *__restrict__ rpa,
                                                const int *__restrict__ cia, const int *__restrict__ rpb,
                                                const int *__restrict__ cib, int *__restrict__ rpc,
                                                int *__restrict__ cic, int64_t cap, unsigned long long *flags,
                                                unsigned epoch, int rows_per_warp, uint64_t limit_ns)
{
    extern __shared__ uint32_t bm_all[];
    __shared__ int s_cnt[1024]; // row counts of the chunk, then their exclusive offsets
    __shared__ int s_prefix, s_ok;
    const int words = (nb + 31) >> 5;
    const int wpc = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = rows_per_warp, R = wpc * k;
    uint32_t *bm = bm_all + (size_t)warp * words;
    const int nchunks = (mb + R - 1) / R;
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x)
    {
        const int r0 = c * R;
        // ---- count: row r0 + w + wpc t of the chunk ----
        for (int t = 0; t < k; ++t)
        {
            const int lr = warp + wpc * t, row = r0 + lr;
            int cnt = 0;
            if (row < mb)
            {
                build_row_bitmap(bm, words, row, rpa, cia, rpb, cib, lane);
                for (int w = lane; w < words; w += 32)
                    cnt += __popc(bm[w]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
            }
            if (lane == 0)
                s_cnt[lr] = cnt;
            __syncwarp();
        }
        __syncthreads();
        // ---- warp 0: the chunk's exclusive row offsets and total, publish,
        //      look back, publish the inclusive prefix ----
        if (warp == 0)
        {
            int carry = 0;
            for (int b = 0; b < R; b += 32)
            {
                const int v = b + lane < R ? s_cnt[b + lane] : 0;
                int x = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o)
                        x += y;
                }
                if (b + lane < R)
                    s_cnt[b + lane] = carry + x - v;
                carry += __shfl_sync(0xffffffffu, x, 31);
            }
            const int total = carry;
            if (lane == 0)
                atomicExch(&flags[c], lb_word(epoch, c == 0, total));
            int prefix = 0;
            bool ok = true;
            if (c > 0)
                ok = lb_prefix(flags, c, epoch, limit_ns, lane, &prefix);
            if (lane == 0)
            {
                if (ok && c > 0)
                    atomicExch(&flags[c], lb_word(epoch, true, prefix + total));
                if (!ok)
                    atomicExch(&g_spg_error, 3);
                s_prefix = prefix;
                s_ok = ok;
                if (r0 + R >= mb) // the last chunk: the total of all rows
                    rpc[mb] = prefix + total;
            }
        }
        __syncthreads();
        if (!s_ok)
            return;
        const int prefix = s_prefix;
        for (int lr = threadIdx.x; lr < R; lr += blockDim.x)
            if (r0 + lr < mb)
                rpc[r0 + lr] = prefix + s_cnt[lr];
        // ---- fill: ColIdxC ascending per row, up to the capacity ----
        if (cap > 0)
            for (int t = 0; t < k; ++t)
            {
                const int lr = warp + wpc * t, row = r0 + lr;
                if (row >= mb)
                    break;
                if (k > 1)
                    build_row_bitmap(bm, words, row, rpa, cia, rpb, cib, lane);
                int out = prefix + s_cnt[lr];
                for (int w0 = 0; w0 < words; w0 += 32)
                {
                    const int w = w0 + lane;
                    uint32_t bits = w < words ? bm[w] : 0u;
                    const int cb = __popc(bits);
                    int pre = cb;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1)
                    {
                        const int y = __shfl_up_sync(0xffffffffu, pre, o);
                        if (lane >= o)
                            pre += y;
                    }
                    int pos = out + pre - cb;
                    while (bits)
                    {
                        const int b = __ffs(bits) - 1;
                        if (pos < cap)
                            cic[pos] = w * 32 + b;
                        ++pos;
                        bits &= bits - 1;
                    }
                    out += __shfl_sync(0xffffffffu, pre, 31);
                }
                __syncwarp();
            }
        __syncthreads(); // s_cnt and the bitmaps are reused by the next chunk
    }
}

// ---------------------------------------------------------------------------
// numeric
// ---------------------------------------------------------------------------
// How C is written: by value to push_store, which would read the kernel's
// parameters again after each store otherwise, and ask for the second half of the
// old tile only then (numeric pass with alpha and beta, 4096 rows of 6: 117 us, 84
// so).
struct PushOut
{
    void *vc;
    int type;
    bool read; // beta is not 0
    float alpha, beta;
};

struct SpNumArgs
{
    int mb, nb;
    const int *rpa, *cia, *rpb, *cib, *rpc, *cic;
    int *cic_out; // the array of cic, where the pass fills it
    const uint16_t *va, *vb;
    void *vc;
    int64_t nnzc;
    int out_type;
    float alpha, beta;
    int num_iter;
    PushOut push; // C as above
};

// Store one C tile with alpha / beta (lane layout of store_tile_frag).
__device__ __forceinline__ void store_c_tile(const SpNumArgs &p, int64_t c, int gq, int tq, const float (&acc0)[4],
                                             const float (&acc1)[4])
{
    store_tile_frag(p.vc, c, p.out_type, p.alpha, p.beta, gq, tq, acc0, acc1);
}

template <bool BF16>
__global__ void __launch_bounds__(256) spgemm_numeric_kernel(const SpNumArgs p)
{
    const int lane = threadIdx.x & 31;
    const int64_t c = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (c >= p.nnzc || c >= p.rpc[p.mb]) // nnz_c may be an upper bound
        return;
    // block-row of this C tile: last i with rpc[i] <= c
    int lo = 0, hi = p.mb - 1;
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        if (p.rpc[mid] <= c)
            lo = mid;
        else
            hi = mid - 1;
    }
    const int i = lo;
    const int j = p.cic[c];
    const int gq = lane >> 2, tq = lane & 3;

    float acc0[4] = {0.f, 0.f, 0.f, 0.f}; // C columns 0..7
    float acc1[4] = {0.f, 0.f, 0.f, 0.f}; // C columns 8..15
    const int a_begin = p.rpa[i], a_end = p.rpa[i + 1];
    for (int it = 0; it < p.num_iter; ++it)
    {
        for (int base = a_begin; base < a_end; base += 32)
        {
            // each lane searches one A block of the row for a matching B block
            const int e = base + lane;
            int match = -1;
            if (e < a_end)
            {
                const int k = p.cia[e];
                int l = p.rpb[k], h = p.rpb[k + 1] - 1;
                while (l <= h)
                {
                    const int m = (l + h) >> 1;
                    const int v = p.cib[m];
                    if (v == j)
                    {
                        match = m;
                        break;
                    }
                    if (v < j)
                        l = m + 1;
                    else
                        h = m - 1;
                }
            }
            uint32_t hits = __ballot_sync(0xffffffffu, match >= 0);
            while (hits)
            {
                const int src = __ffs(hits) - 1;
                hits &= hits - 1;
                const int eb = __shfl_sync(0xffffffffu, match, src);
                const int ea = base + src;
                const uint16_t *ta = p.va + (int64_t)ea * 256;
                const uint16_t *tb = p.vb + (int64_t)eb * 256;
                // A fragment with the k index permuted inside the k-step: lane
                // (g, t) holds A[g][4t..4t+3] and A[g+8][4t..4t+3]
                const uint2 ra = __ldg(reinterpret_cast<const uint2 *>(ta + gq * 16 + 4 * tq));
                const uint2 rb = __ldg(reinterpret_cast<const uint2 *>(ta + (gq + 8) * 16 + 4 * tq));
                // B fragment (K x N, row-major tile), same k permutation
                uint32_t b00, b01, b10, b11;
                {
                    const uint16_t *col0 = tb + gq;     // n = g      (columns 0..7)
                    const uint16_t *col1 = tb + gq + 8; // n = g + 8  (columns 8..15)
                    const int k0 = 4 * tq;
                    b00 = (uint32_t)__ldg(col0 + (k0 + 0) * 16) | ((uint32_t)__ldg(col0 + (k0 + 1) * 16) << 16);
                    b01 = (uint32_t)__ldg(col0 + (k0 + 2) * 16) | ((uint32_t)__ldg(col0 + (k0 + 3) * 16) << 16);
                    b10 = (uint32_t)__ldg(col1 + (k0 + 0) * 16) | ((uint32_t)__ldg(col1 + (k0 + 1) * 16) << 16);
                    b11 = (uint32_t)__ldg(col1 + (k0 + 2) * 16) | ((uint32_t)__ldg(col1 + (k0 + 3) * 16) << 16);
                }
                mma16816<BF16>(acc0, ra.x, rb.x, ra.y, rb.y, b00, b01);
                mma16816<BF16>(acc1, ra.x, rb.x, ra.y, rb.y, b10, b11);
            }
        }
    }

    store_c_tile(p, c, gq, tq, acc0, acc1);
}

// ---------------------------------------------------------------------------
// numeric, rows beyond the capacities of the kernel below (16-byte aligned tiles)
//
// The C tiles of block-row i all multiply the same A tiles A(i, k) and search
// the same B block-rows k for their column j.  So the CTA stages, once, the
// A tiles of row i (ldmatrix layout) and the column indices of every B row k
// it touches in shared memory; each of its 8 warps then takes C tiles
// (i, j) in turn: lanes binary-search j in the staged lists (shared-memory
// latency instead of dependent global loads), and every match costs one
// coalesced 512-byte load of the B tile into the warp's slot, one ldmatrix
// (transposed) for its fragments, and two MMAs.  Products are accumulated in
// ascending k, as the reference's sparse accumulator does.  Rows whose A
// tiles or B lists exceed the staging capacity read them from global memory.
// ---------------------------------------------------------------------------
constexpr int kMaxBList = 2048;  // 8 KB of B column indices

// The row's C tiles pulled one at a time (the per-tile search form); the
// CTA's shared buffers are passed in: sA MAXA * 512 bytes, sB WARPS * 512,
// sList kMaxBList ints, sOff MAXA + 1, sK MAXA.
template <bool BF16, int WARPS, int MAXA>
__device__ __forceinline__ void numeric_row_pull(const SpNumArgs &p, const int i, uint8_t *sA, uint8_t *sB,
                                                 int *sList, int *sOff, int *sK)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = p.rpc[i];
    const int c1 = (int)min((int64_t)p.rpc[i + 1], p.nnzc); // tiles past the caller's bound are untouched
    if (c1 <= c0)
        return;
    const int a0 = p.rpa[i], na = p.rpa[i + 1] - a0;
    const bool a_staged = na <= MAXA;

    // ---- staging (whole CTA): A tiles, B row lengths, their prefix, lists ----
    bool l_staged = false;
    if (a_staged)
    {
        for (int e = warp; e < na; e += WARPS)
            stage_tile(sA + e * 512, p.va + (int64_t)(a0 + e) * 256, lane);
        if (warp == 0)
        {
            // lengths of the B rows, exclusive prefix over the (<= 48) entries
            int total = 0;
            for (int base = 0; base < na; base += 32)
            {
                const int e = base + lane;
                int len = 0;
                if (e < na)
                {
                    const int k = p.cia[a0 + e];
                    sK[e] = k;
                    len = p.rpb[k + 1] - p.rpb[k];
                }
                int pre = len;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    const int y = __shfl_up_sync(0xffffffffu, pre, o);
                    if (lane >= o)
                        pre += y;
                }
                if (e < na)
                    sOff[e] = total + pre - len;
                total += __shfl_sync(0xffffffffu, pre, 31);
            }
            if (lane == 0)
                sOff[na] = total;
        }
        __syncthreads();
        l_staged = sOff[na] <= kMaxBList;
        if (l_staged)
            for (int e = warp; e < na; e += WARPS)
            {
                const int b0 = p.rpb[sK[e]], len = sOff[e + 1] - sOff[e];
                for (int q = lane; q < len; q += 32)
                    sList[sOff[e] + q] = p.cib[b0 + q];
            }
        __syncthreads();
    }

    const int gq = lane >> 2, tq = lane & 3;
    const uint32_t sA_u = (uint32_t)__cvta_generic_to_shared(sA);
    const uint32_t slot = (uint32_t)__cvta_generic_to_shared(sB + warp * 512);
    uint8_t *slot_p = sB + warp * 512;
    for (int c = c0 + warp; c < c1; c += WARPS)
    {
        const int j = p.cic[c];
        float acc0[4] = {0.f, 0.f, 0.f, 0.f}; // C columns 0..7
        float acc1[4] = {0.f, 0.f, 0.f, 0.f}; // C columns 8..15
        for (int it = 0; it < p.num_iter; ++it)
            for (int base = 0; base < na; base += 32)
            {
                // lane e: position of column j in B row k_e (global B entry), or -1
                const int e = base + lane;
                int match = -1;
                if (e < na)
                {
                    const int k = a_staged ? sK[e] : p.cia[a0 + e];
                    const int bstart = p.rpb[k];
                    if (l_staged)
                    {
                        int l = sOff[e], h = sOff[e + 1] - 1;
                        const int o = l;
                        while (l <= h)
                        {
                            const int m = (l + h) >> 1, v = sList[m];
                            if (v == j)
                            {
                                match = bstart + (m - o);
                                break;
                            }
                            if (v < j)
                                l = m + 1;
                            else
                                h = m - 1;
                        }
                    }
                    else
                    {
                        int l = bstart, h = p.rpb[k + 1] - 1;
                        while (l <= h)
                        {
                            const int m = (l + h) >> 1, v = p.cib[m];
                            if (v == j)
                            {
                                match = m;
                                break;
                            }
                            if (v < j)
                                l = m + 1;
                            else
                                h = m - 1;
                        }
                    }
                }
                uint32_t hits = __ballot_sync(0xffffffffu, match >= 0);
                while (hits)
                {
                    const int src = __ffs(hits) - 1;
                    hits &= hits - 1;
                    const int eb = __shfl_sync(0xffffffffu, match, src);
                    const int ea = base + src;
                    uint32_t a[4];
                    if (a_staged)
                        ldsm4(tile_ldsm_addr(sA_u + ea * 512, lane), a);
                    else
                    {
                        const uint32_t *ta = reinterpret_cast<const uint32_t *>(p.va + (int64_t)(a0 + ea) * 256);
                        a[0] = load_operand(ta + (gq * 16 + 2 * tq) / 2);
                        a[1] = load_operand(ta + ((gq + 8) * 16 + 2 * tq) / 2);
                        a[2] = load_operand(ta + (gq * 16 + 2 * tq + 8) / 2);
                        a[3] = load_operand(ta + ((gq + 8) * 16 + 2 * tq + 8) / 2);
                    }
                    __syncwarp(); // the slot's previous tile has been read
                    stage_tile(slot_p, p.vb + (int64_t)eb * 256, lane);
                    __syncwarp();
                    uint32_t b[4];
                    ldsm4_t(tile_ldsm_addr(slot, lane), b); // (k lo, n 0-7), (k hi, n 0-7), (k lo, n 8-15), (k hi, n 8-15)
                    mma16816<BF16>(acc0, a[0], a[1], a[2], a[3], b[0], b[1]);
                    mma16816<BF16>(acc1, a[0], a[1], a[2], a[3], b[2], b[3]);
                }
            }
        store_c_tile(p, c, gq, tq, acc0, acc1);
    }
}

// ---------------------------------------------------------------------------
// numeric, one CTA per block-row of C, products pushed to their tiles
//
// The per-tile search above costs one binary search per (C tile, A entry)
// pair -- about ten per tile at 1 % density -- in dependent shared-memory
// loads, and each tile's B tile load is exposed.  Here the row's products
// are enumerated once: all threads walk the flattened (A entry, B entry)
// space, find each product's C position, and a counting sort by position
// groups them per C tile (each tile's short list then re-sorted by
// enumeration index, so products still accumulate in ascending k).  The
// position comes from a bitmap of the row's columns (words of 32 with their
// running counts) when the kernel writes ColIdxC as well (FILL: the pass that
// would only fill it takes 7 us more at n = 16384, 1 %), else from a binary
// search in the row's ColIdxC.
// The warps then take the tiles in turn.  A product's B tile goes straight from
// global memory into the fragments of two m16n8k16 MMAs, kPushDepth products
// ahead: a lane's columns are 2 gq and 2 gq + 1, so four 4-byte loads and four
// byte permutes make both fragments, and C leaves as float4 (through a ring
// in shared memory and ldmatrix, the stores' halves exchanged by shuffles:
// n = 16384, 1 % 37.3 us against 34.5; 4096 rows of 6 tiles 51 against 48).
// What bounds it is the longest rows: the mean CTA runs 32 thousand cycles (9 of
// them before its first product), the longest 50 thousand.  Runs of C tiles
// dealt to warps across rows were even, and slower: 42 .. 56 us, each run
// searching its products anew.  Rows beyond the staging capacities fall back to
// the per-tile form.
// ---------------------------------------------------------------------------
// Warps of a CTA: eight while every block-row has a place at once (four CTAs of
// eight warps per SM), so that a row takes less time (numeric pass of 300 rows
// of 9 entries 13.9 us against 17.1, 128 rows 13.0 against 17.1), and where rows have
// 96 C tiles or more on average (1024 rows of 12 entries, 134 tiles: 39 us against 45; of
// 20, 330 tiles: 196 against 425, as more of them fit the wider staging); four
// otherwise (4096 rows of 8, 64 tiles: 72 us against 81).
constexpr int kPushWarps = 4, kPushWarpsMany = 8, kPushFewPerSm = 4, kPushManyTiles = 96;
// What a CTA of so many warps stages of a row: A tiles (a lane each), C tiles, products
template <int WARPS> constexpr int kPushMaxA = WARPS == kPushWarpsMany ? 32 : 24;
template <int WARPS> constexpr int kPushMaxC = WARPS == kPushWarpsMany ? 896 : 512;
constexpr int kPushDepth = 4;     // B tiles on their way per warp, in registers
constexpr int kFillWords = 512;   // FILL: words of 32 block columns

__device__ __forceinline__ uint32_t pack16(float x, float y, bool bf)
{
    if (bf)
    {
        const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
        return *reinterpret_cast<const uint32_t *>(&v);
    }
    const __half2 v = __floats2half2_rn(x, y);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// two 16-bit neighbours of C, was: their old values (the type known where it is
// compiled: per element at run time, 1024 rows of 10 took 52 us instead of 41)
template <bool BF16> __device__ __forceinline__ uint32_t scale16(const PushOut &o, float x, float y, uint32_t was)
{
    x *= o.alpha;
    y *= o.alpha;
    if (o.read)
    {
        x += o.beta * to_float((uint16_t)was, BF16);
        y += o.beta * to_float((uint16_t)(was >> 16), BF16);
    }
    return pack16(x, y, BF16);
}

// C tile c with alpha / beta in any output type: lane (gq, tq) holds columns
// 4 tq .. 4 tq + 3 of rows gq (lo) and gq + 8 (hi).  beta == 0 never reads C.
__device__ __noinline__ void push_store(const PushOut o, int64_t c, int gq, int tq, float4 lo, float4 hi)
{
    const int64_t at = c * 256 + gq * 16 + 4 * tq;
    auto scale = [&](float4 &v, float4 was) {
        v = make_float4(o.alpha * v.x + o.beta * was.x, o.alpha * v.y + o.beta * was.y, o.alpha * v.z + o.beta * was.z,
                        o.alpha * v.w + o.beta * was.w);
    };
    if (o.type == KAMI_F32)
    {
        float *const q = reinterpret_cast<float *>(o.vc) + at;
        if (!(reinterpret_cast<uintptr_t>(o.vc) & 15))
        {
            float4 *const p0 = reinterpret_cast<float4 *>(q), *const p1 = reinterpret_cast<float4 *>(q + 128);
            if (o.alpha != 1.f || o.read)
            {
                float4 w0 = make_float4(0.f, 0.f, 0.f, 0.f), w1 = w0;
                if (o.read)
                    w0 = *p0, w1 = *p1;
                scale(lo, w0);
                scale(hi, w1);
            }
            *p0 = lo;
            *p1 = hi;
            return;
        }
        float2 *const p0 = reinterpret_cast<float2 *>(q), *const p1 = reinterpret_cast<float2 *>(q + 128);
        if (o.alpha != 1.f || o.read)
        {
            float2 w00 = make_float2(0.f, 0.f), w01 = w00, w10 = w00, w11 = w00;
            if (o.read)
                w00 = p0[0], w01 = p0[1], w10 = p1[0], w11 = p1[1];
            scale(lo, make_float4(w00.x, w00.y, w01.x, w01.y));
            scale(hi, make_float4(w10.x, w10.y, w11.x, w11.y));
        }
        p0[0] = make_float2(lo.x, lo.y);
        p0[1] = make_float2(lo.z, lo.w);
        p1[0] = make_float2(hi.x, hi.y);
        p1[1] = make_float2(hi.z, hi.w);
        return;
    }
    uint2 *const p0 = reinterpret_cast<uint2 *>(reinterpret_cast<uint16_t *>(o.vc) + at), *const p1 = p0 + 32;
    uint2 w0 = make_uint2(0u, 0u), w1 = w0;
    if (o.read)
        w0 = *p0, w1 = *p1;
    if (o.type == KAMI_BF16)
    {
        *p0 = make_uint2(scale16<true>(o, lo.x, lo.y, w0.x), scale16<true>(o, lo.z, lo.w, w0.y));
        *p1 = make_uint2(scale16<true>(o, hi.x, hi.y, w1.x), scale16<true>(o, hi.z, hi.w, w1.y));
    }
    else
    {
        *p0 = make_uint2(scale16<false>(o, lo.x, lo.y, w0.x), scale16<false>(o, lo.z, lo.w, w0.y));
        *p1 = make_uint2(scale16<false>(o, hi.x, hi.y, w1.x), scale16<false>(o, hi.z, hi.w, w1.y));
    }
}

// The row's columns from its bitmap: pre[w] = columns before word w, and
// ColIdxC's entries, the first `room` of them.  By the whole CTA.
__device__ __forceinline__ void row_columns(const uint32_t *bm, int words, int *pre, int *cic, int room)
{
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32)
    {
        int carry = 0;
        for (int b = 0; b < words; b += 32)
        {
            const int v = b + lane < words ? __popc(bm[b + lane]) : 0;
            int x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o)
                    x += y;
            }
            if (b + lane < words)
                pre[b + lane] = carry + x - v;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    __syncthreads();
    for (int w = threadIdx.x; w < words; w += blockDim.x)
    {
        int at = pre[w];
        for (uint32_t bits = bm[w]; bits && at < room; bits &= bits - 1)
            cic[at++] = w * 32 + __ffs(bits) - 1;
    }
}

template <bool BF16, bool FILL, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) spgemm_numeric_push_kernel(const __grid_constant__ SpNumArgs p)
{
    constexpr int MAXA = kPushMaxA<WARPS>, MAXC = kPushMaxC<WARPS>; // products: up to MAXC too
    __shared__ __align__(16) uint8_t sA[MAXA * 512];
    __shared__ __align__(16) uint8_t sB[WARPS * 512]; // of the per-tile fallback
    __shared__ uint32_t sBits[FILL ? kFillWords : 1];      // the row's columns
    __shared__ int sPre[FILL ? kFillWords : 1];
    // one pool of indices (the per-tile fallback uses its first kMaxBList
    // entries as its list buffer): the row's ColIdxC, then per tile the
    // product count / range end; per product (A entry << 16) | C position
    // (-1 when absent), its B entry, and the products grouped by C tile
    __shared__ int sPool[5 * MAXC];
    static_assert(5 * MAXC >= kMaxBList && MAXA <= 32, "fallback list buffer, a lane per A tile");
    int *sCol = sPool, *sCnt = sPool + MAXC, *sPep = sPool + 2 * MAXC, *sPb = sPool + 3 * MAXC,
        *sOrd = sPool + 4 * MAXC;
    __shared__ int sOff[MAXA + 1];
    __shared__ int sK[MAXA];
    __shared__ int sRb[MAXA];
    wait_for_previous();
    const int i = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kT = WARPS * 32;
    const int c0 = p.rpc[i];
    const int c1 = (int)min((int64_t)p.rpc[i + 1], p.nnzc); // tiles past the caller's bound are untouched
    if (c1 <= c0)
        return;
    const int nt = c1 - c0;
    const int a0 = p.rpa[i], na = p.rpa[i + 1] - a0;
    const int words = (p.nb + 31) >> 5;
    if constexpr (FILL)
        for (int w = tid; w < words; w += kT)
            sBits[w] = 0u;
    bool pull = nt > MAXC || na > MAXA;
    int np = 0;
    if (!pull)
    {
        // ---- stage: ColIdxC, B row ranges and their prefix, A tiles ----
        for (int t = tid; t < nt; t += kT)
        {
            if constexpr (!FILL)
                sCol[t] = p.cic[c0 + t];
            sCnt[t] = 0;
        }
        if (warp == 0)
        {
            int len = 0;
            if (lane < na)
            {
                const int k = p.cia[a0 + lane];
                const int rb = p.rpb[k];
                len = p.rpb[k + 1] - rb;
                sK[lane] = k;
                sRb[lane] = rb;
            }
            int pre = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, pre, o);
                if (lane >= o)
                    pre += y;
            }
            if (lane < na)
                sOff[lane] = pre - len;
            if (lane == 31)
                sOff[na] = pre;
        }
        for (int e = warp; e < na; e += WARPS)
            stage_tile(sA + e * 512, p.va + (int64_t)(a0 + e) * 256, lane);
        __syncthreads();
        np = sOff[na];
        pull = np > MAXC;
    }
    if (pull)
    {
        __syncthreads();
        if constexpr (FILL)
        {
            for (int e = a0 + tid; e < a0 + na; e += kT)
            {
                const int k = p.cia[e], b1 = p.rpb[k + 1];
                for (int b = p.rpb[k]; b < b1; ++b)
                    atomicOr(&sBits[p.cib[b] >> 5], 1u << (p.cib[b] & 31));
            }
            __syncthreads();
            row_columns(sBits, words, sPre, p.cic_out + c0, nt);
            __syncthreads();
        }
        numeric_row_pull<BF16, WARPS, MAXA>(p, i, sA, sB, sPool, sOff, sK);
        return;
    }
    // ---- enumerate the products and count them per C tile ----
    for (int f = tid; f < np; f += kT)
    {
        int lo = 0, hi = na - 1; // entry e with sOff[e] <= f < sOff[e + 1]
        while (lo < hi)
        {
            const int m = (lo + hi + 1) >> 1;
            if (sOff[m] <= f)
                lo = m;
            else
                hi = m - 1;
        }
        const int e = lo;
        const int eb = sRb[e] + (f - sOff[e]);
        const int j = p.cib[eb];
        sPb[f] = eb;
        if constexpr (FILL)
        {
            sPep[f] = e << 16;
            sOrd[f] = j;
            atomicOr(&sBits[j >> 5], 1u << (j & 31));
            continue;
        }
        int l = 0, h = nt;
        while (l < h)
        {
            const int m = (l + h) >> 1;
            if (sCol[m] < j)
                l = m + 1;
            else
                h = m;
        }
        const bool hit = l < nt && sCol[l] == j;
        sPep[f] = hit ? ((e << 16) | l) : -1;
        if (hit)
            atomicAdd(&sCnt[l], 1);
    }
    __syncthreads();
    if constexpr (FILL)
    {
        row_columns(sBits, words, sPre, p.cic_out + c0, nt);
        for (int f = tid; f < np; f += kT)
        {
            const int j = sOrd[f], l = sPre[j >> 5] + __popc(sBits[j >> 5] & ((1u << (j & 31)) - 1));
            if (l >= nt) // a tile past the caller's bound
            {
                sPep[f] = -1;
                continue;
            }
            sPep[f] |= l;
            atomicAdd(&sCnt[l], 1);
        }
        __syncthreads();
    }
    // ---- exclusive scan of the counts (warp 0, 32 consecutive entries per lane) ----
    if (warp == 0)
    {
        const int per = (nt + 31) >> 5;
        const int b0 = lane * per, b1 = min(nt, b0 + per);
        int run = 0;
        for (int t = b0; t < b1; ++t)
            run += sCnt[t];
        int pre = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o)
                pre += y;
        }
        int acc = pre - run;
        for (int t = b0; t < b1; ++t)
        {
            const int c = sCnt[t];
            sCnt[t] = acc;
            acc += c;
        }
    }
    __syncthreads();
    // ---- scatter: afterwards sCnt[t] is the end of tile t's range ----
    for (int f = tid; f < np; f += kT)
    {
        const int v = sPep[f];
        if (v >= 0)
            sOrd[atomicAdd(&sCnt[v & 0xffff], 1)] = f;
    }
    __syncthreads();
    // ---- each tile's products in enumeration order (ascending k) ----
    for (int t = tid; t < nt; t += kT)
    {
        const int b = t ? sCnt[t - 1] : 0, e = sCnt[t];
        for (int x = b + 1; x < e; ++x)
        {
            const int v = sOrd[x];
            int y = x - 1;
            while (y >= b && sOrd[y] > v)
            {
                sOrd[y + 1] = sOrd[y];
                --y;
            }
            sOrd[y + 1] = v;
        }
    }
    __syncthreads();

    // ---- multiply: warp w takes the contiguous tile range [t0, t1), whose
    //      products are contiguous in sOrd (ascending tile, then k) ----
    const int t0 = (nt * warp) / WARPS, t1 = (nt * (warp + 1)) / WARPS;
    const int q0 = t0 ? sCnt[t0 - 1] : 0, q1 = t1 ? sCnt[t1 - 1] : 0;
    const int gq = lane >> 2, tq = lane & 3;
    const bool f32 = p.out_type == KAMI_F32, bf = p.out_type == KAMI_BF16;
    const bool plain = p.alpha == 1.f && p.beta == 0.f && !(reinterpret_cast<uintptr_t>(p.vc) & (f32 ? 15 : 7));
    uint8_t *const out = reinterpret_cast<uint8_t *>(p.vc) + ((int64_t)c0 * 256 + gq * 16 + 4 * tq) * (f32 ? 4 : 2);
    // tiles without products hold zeros
    for (int base = t0; base < t1; base += 32)
    {
        const int t = base + lane;
        unsigned none = __ballot_sync(0xffffffffu, t < t1 && sCnt[t] == (t ? sCnt[t - 1] : 0));
        for (; none; none &= none - 1)
            push_store(p.push, c0 + base + __ffs(none) - 1, gq, tq, make_float4(0.f, 0.f, 0.f, 0.f),
                       make_float4(0.f, 0.f, 0.f, 0.f));
    }
    const uint32_t a_lane = tile_ldsm_addr((uint32_t)__cvta_generic_to_shared(sA), lane);
    const uint8_t *const b_lane = reinterpret_cast<const uint8_t *>(p.vb) + tq * 64 + gq * 4;
    float acc0[4] = {0.f, 0.f, 0.f, 0.f}; // columns 4 tq, 4 tq + 2
    float acc1[4] = {0.f, 0.f, 0.f, 0.f}; // columns 4 tq + 1, 4 tq + 3
    uint32_t nx[kPushDepth][4];           // rows 2 tq, 2 tq + 1, 2 tq + 8, 2 tq + 9 of the next products' B tiles
    for (int base = q0; base < q1; base += 32)
    {
        // lane l: product base + l, as its A tile's place, its C tile (bit 31:
        // the last product of that tile) and its B entry
        const int n = min(32, q1 - base);
        int place = 0, tile = 0, eb = 0;
        if (lane < n)
        {
            const int f = sOrd[base + lane], pep = sPep[f];
            place = (pep >> 16) * 512;
            tile = pep & 0xffff;
            if (base + lane + 1 == sCnt[tile])
                tile |= (int)0x80000000;
            eb = sPb[f];
        }
        auto fetch = [&](int x, uint32_t(&v)[4]) {
            const uint8_t *const b = b_lane + (int64_t)__shfl_sync(0xffffffffu, eb, x) * 512;
            v[0] = load_operand(reinterpret_cast<const uint32_t *>(b));
            v[1] = load_operand(reinterpret_cast<const uint32_t *>(b + 32));
            v[2] = load_operand(reinterpret_cast<const uint32_t *>(b + 256));
            v[3] = load_operand(reinterpret_cast<const uint32_t *>(b + 288));
        };
#pragma unroll
        for (int d = 0; d < kPushDepth; ++d)
            fetch(min(d, n - 1), nx[d]);
        for (int x = 0; x < n; x += kPushDepth)
        {
#pragma unroll
            for (int d = 0; d < kPushDepth; ++d)
                if (x + d < n)
                {
                    uint32_t a[4];
                    ldsm4(a_lane + __shfl_sync(0xffffffffu, place, x + d), a);
                    const int t = __shfl_sync(0xffffffffu, tile, x + d);
                    // low halves: column 2 gq of two rows; high halves: column 2 gq + 1
                    const uint32_t e0 = __byte_perm(nx[d][0], nx[d][1], 0x5410), o0 = __byte_perm(nx[d][0], nx[d][1], 0x7632);
                    const uint32_t e1 = __byte_perm(nx[d][2], nx[d][3], 0x5410), o1 = __byte_perm(nx[d][2], nx[d][3], 0x7632);
                    fetch(min(x + d + kPushDepth, n - 1), nx[d]);
                    for (int r = 0; r < p.num_iter; ++r)
                    {
                        mma16816<BF16>(acc0, a[0], a[1], a[2], a[3], e0, e1);
                        mma16816<BF16>(acc1, a[0], a[1], a[2], a[3], o0, o1);
                    }
                    if (t < 0)
                    {
                        const float4 lo = make_float4(acc0[0], acc1[0], acc0[1], acc1[1]);
                        const float4 hi = make_float4(acc0[2], acc1[2], acc0[3], acc1[3]);
                        if (plain && f32)
                        {
                            float4 *const o = reinterpret_cast<float4 *>(out + (int64_t)(t & 0xffff) * 1024);
                            o[0] = lo;
                            o[32] = hi;
                        }
                        else if (plain)
                        {
                            uint2 *const o = reinterpret_cast<uint2 *>(out + (int64_t)(t & 0xffff) * 512);
                            o[0] = make_uint2(pack16(lo.x, lo.y, bf), pack16(lo.z, lo.w, bf));
                            o[32] = make_uint2(pack16(hi.x, hi.y, bf), pack16(hi.z, hi.w, bf));
                        }
                        else
                            push_store(p.push, c0 + (t & 0xffff), gq, tq, lo, hi);
#pragma unroll
                        for (int y = 0; y < 4; ++y)
                            acc0[y] = acc1[y] = 0.f;
                    }
                }
        }
    }
}

template <bool BF16, bool FILL> cudaError_t push_launch(const SpNumArgs &p, bool many, cudaStream_t s)
{
    const void *fn = many ? (const void *)spgemm_numeric_push_kernel<BF16, FILL, kPushWarpsMany>
                         : (const void *)spgemm_numeric_push_kernel<BF16, FILL, kPushWarps>;
    void *args[] = {const_cast<SpNumArgs *>(&p)};
    return launch_overlapped(fn, dim3((unsigned)p.mb), dim3(32 * (many ? kPushWarpsMany : kPushWarps)), args, 0, s);
}

cudaError_t push_launch(const SpNumArgs &p, bool bf16, bool fill, bool many, cudaStream_t s)
{
    if (bf16)
        return fill ? push_launch<true, true>(p, many, s) : push_launch<true, false>(p, many, s);
    return fill ? push_launch<false, true>(p, many, s) : push_launch<false, false>(p, many, s);
}

int bitmap_launch(int nb, int *warps_per_cta, size_t *smem)
{
    const int words = (nb + 31) >> 5;
    int w = 8;
    while (w > 1 && (size_t)w * words * 4 > 96 * 1024)
        w >>= 1;
    if ((size_t)w * words * 4 > 200 * 1024)
        return fail(KAMI_ERR_UNSUPPORTED, "spgemm: %d block columns exceed the shared-memory bitmap", nb);
    *warps_per_cta = w;
    *smem = (size_t)w * words * 4;
    return KAMI_OK;
}

int prep_bitmap_fn(const void *fn, size_t smem)
{
    if (smem > 48 * 1024)
    {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaFuncSetAttribute(spgemm bitmap kernel)");
    }
    return KAMI_OK;
}

// Row pointers must be present; column-index arrays may be NULL when the
// matrix has no nonzero block.
int check_bsr_args(int bsr, int mb, int kb, int nb, const void *a, const void *, const void *c, const void *)
{
    if (bsr != kBsr)
        return fail(KAMI_ERR_UNSUPPORTED, "spgemm: only 16 x 16 BSR tiles are supported (got %d)", bsr);
    if (mb < 0 || kb < 0 || nb < 0)
        return fail(KAMI_ERR_INVALID_VALUE, "spgemm: negative block dimensions");
    if (mb > 0 && (!a || !c))
        return fail(KAMI_ERR_INVALID_VALUE, "spgemm: null row pointer");
    return KAMI_OK;
}

// The fused one-launch symbolic pass; KAMI_ERR_UNSUPPORTED (nothing
// launched) when the device has no cooperative launch.
int symbolic_fused(int mb, int nb, const int *rpa, const int *cia, const int *rpb, const int *cib, int *rpc, int *cic,
                   int64_t cap, cudaStream_t s)
{
    int dev = 0, sms = 0, coop = 0, occ = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess)
        return cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= 64)
        return KAMI_ERR_UNSUPPORTED;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop)
        return KAMI_ERR_UNSUPPORTED;
    static std::once_flag once[64];
    static unsigned int *bar_base[64];
    static cudaError_t bar_err[64];
    std::call_once(once[dev], [&] {
        void *ptr = nullptr;
        bar_err[dev] = cudaGetSymbolAddress(&ptr, g_spg_bar);
        bar_base[dev] = reinterpret_cast<unsigned int *>(ptr);
    });
    if (bar_err[dev] != cudaSuccess)
        return cuda_fail(bar_err[dev], "cudaGetSymbolAddress(spgemm barrier)");
    int wpc;
    size_t smem;
    int st = bitmap_launch(nb, &wpc, &smem);
    if (st)
        return st;
    const void *fn = (const void *)spgemm_symbolic_fused_kernel;
    if ((st = prep_bitmap_fn(fn, smem)))
        return st;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, wpc * 32, smem)) != cudaSuccess)
        return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor(spgemm fused)");
    if (occ < 1)
        return KAMI_ERR_UNSUPPORTED;
    const int rows_ctas = (mb + wpc - 1) / wpc;
    int grid = rows_ctas < sms * occ ? rows_ctas : sms * occ;
    // keep every row's bitmap from the count to the fill when the warps' rows
    // fit in 96 KB of shared memory at a grid that stays co-resident
    int keep_rows = 0;
    const int words = (nb + 31) >> 5;
    const int rpw = (mb + grid * wpc - 1) / (grid * wpc);
    const size_t keep_smem = (size_t)wpc * rpw * words * 4;
    if (cap > 0 && rpw > 0 && keep_smem <= 96 * 1024)
    {
        int occ_k = 0;
        if (keep_smem > smem && (st = prep_bitmap_fn(fn, keep_smem)))
            return st;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_k, fn, wpc * 32, keep_smem) == cudaSuccess &&
            grid <= sms * occ_k)
        {
            keep_rows = rpw;
            smem = keep_smem > smem ? keep_smem : smem;
        }
    }
    static std::atomic<unsigned int> next_slot{0};
    unsigned int *bar = bar_base[dev] + 2 * (next_slot.fetch_add(1) % kFuseSlots);
    if ((e = cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned int), s)) != cudaSuccess)
        return cuda_fail(e, "cudaMemsetAsync(spgemm barrier)");
    // generous: a barrier waits for the slowest CTA's share of the rows
    uint64_t limit = (uint64_t)2e9 + (uint64_t)mb * 20000ull;
    void *args[] = {&mb, &nb, &rpa, &cia, &rpb, &cib, &rpc, &cic, &cap, &bar, &limit, &keep_rows};
    if ((e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(wpc * 32), args, smem, s)) != cudaSuccess)
        return cuda_fail(e, "cudaLaunchCooperativeKernel(spgemm_symbolic_fused_kernel)");
    return KAMI_OK;
}


// The single-pass symbolic launch; KAMI_ERR_UNSUPPORTED (nothing launched)
// when the device has no cooperative launch or the rows need more chunks
// than the flag array holds.
int symbolic_lookback(int mb, int nb, const int *rpa, const int *cia, const int *rpb, const int *cib, int *rpc,
                      int *cic, int64_t cap, cudaStream_t s)
{
    int dev = 0, sms = 0, coop = 0, occ = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess)
        return cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= 64)
        return KAMI_ERR_UNSUPPORTED;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop || mb < 1)
        return KAMI_ERR_UNSUPPORTED;
    static std::once_flag once[64];
    static unsigned long long *flag_base[64];
    static cudaError_t flag_err[64];
    std::call_once(once[dev], [&] {
        void *ptr = nullptr;
        flag_err[dev] = cudaGetSymbolAddress(&ptr, g_spg_flags);
        flag_base[dev] = reinterpret_cast<unsigned long long *>(ptr);
    });
    if (flag_err[dev] != cudaSuccess)
        return cuda_fail(flag_err[dev], "cudaGetSymbolAddress(spgemm look-back flags)");
    int wpc;
    size_t smem;
    int st = bitmap_launch(nb, &wpc, &smem);
    if (st)
        return st;
    // rows per warp per chunk: the chunks must fit the flag array and R = wpc k
    // rows the kernel's offset array
    const int64_t k64 = ((int64_t)mb + (int64_t)wpc * kLbMaxChunks - 1) / ((int64_t)wpc * kLbMaxChunks);
    if (k64 < 1 || wpc * k64 > 1024)
        return KAMI_ERR_UNSUPPORTED;
    const int k = (int)k64, R = wpc * k;
    const int nchunks = (mb + R - 1) / R;
    const void *fn = (const void *)spgemm_symbolic_lookback_kernel;
    if ((st = prep_bitmap_fn(fn, smem)))
        return st;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, wpc * 32, smem)) != cudaSuccess)
        return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor(spgemm look-back)");
    if (occ < 1)
        return KAMI_ERR_UNSUPPORTED;
    const int grid = nchunks < sms * occ ? nchunks : sms * occ;
    static std::atomic<unsigned int> next_launch{0};
    const unsigned int n = next_launch.fetch_add(1);
    unsigned long long *flags = flag_base[dev] + (size_t)(n % kLbSlots) * kLbMaxChunks;
    unsigned epoch = (n % 0x7fffffffu) + 1; // never 0, the value of untouched flags
    uint64_t limit = (uint64_t)2e9 + (uint64_t)mb * 20000ull;
    void *args[] = {&mb, &nb, &rpa, &cia, &rpb, &cib, &rpc, &cic, &cap, &flags, &epoch, (void *)&k, &limit};
    if ((e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(wpc * 32), args, smem, s)) != cudaSuccess)
        return cuda_fail(e, "cudaLaunchCooperativeKernel(spgemm_symbolic_lookback_kernel)");
    return KAMI_OK;
}

} // namespace

int spgemm_tc05_launch(bool bf16, int mb, int64_t nnzc, const int *rpa, const int *cia, const int *rpb, const int *cib,
                       const int *rpc, const int *cic, const void *va, const void *vb, void *vc, int out_type,
                       double alpha, double beta, int num_iter, cudaStream_t s);

// AUTO's choice of the numeric kernel: the mma.sync row kernel (false) or
// the tcgen05 kernel (true).
bool spgemm_auto_tc05() { return false; }

int spgemm_read_error(int *flag)
{
    int v = 0, z = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_spg_error, sizeof(int));
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbol(g_spg_error, &z, sizeof(int));
    if (e != cudaSuccess)
        return cuda_fail(e, "reading the spgemm status");
    *flag = v;
    return KAMI_OK;
}

} // namespace kami

using namespace kami;

extern "C" {

int kami_spgemm_bsr_symbolic(int bsr, int mb, int kb, int nb, const int *row_ptr_a, const int *col_idx_a,
                             const int *row_ptr_b, const int *col_idx_b, int *row_ptr_c, int *nnz_c_host,
                             void *stream)
{
    int st = check_bsr_args(bsr, mb, kb, nb, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b);
    if (st)
        return st;
    if (!row_ptr_c)
        return fail(KAMI_ERR_INVALID_VALUE, "spgemm: row_ptr_c is NULL");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    cudaError_t e;
    if (mb > 0 && nb > 0)
    {
        int wpc;
        size_t smem;
        if ((st = bitmap_launch(nb, &wpc, &smem)))
            return st;
        if ((st = prep_bitmap_fn((const void *)spgemm_count_kernel, smem)))
            return st;
        const int grid = (mb + wpc - 1) / wpc;
        void *count_args[] = {&mb, &nb, &row_ptr_a, &col_idx_a, &row_ptr_b, &col_idx_b, &row_ptr_c};
        if ((e = launch_overlapped((const void *)spgemm_count_kernel, dim3(grid), dim3(wpc * 32), count_args, smem, s)) !=
            cudaSuccess)
            return cuda_fail(e, "spgemm_count_kernel");
        void *scan_args[] = {&mb, &row_ptr_c};
        if ((e = launch_overlapped((const void *)spgemm_scan_kernel, dim3(1), dim3(1024), scan_args, 0, s)) != cudaSuccess)
            return cuda_fail(e, "spgemm_scan_kernel");
    }
    else
    {
        if ((e = cudaMemsetAsync(row_ptr_c, 0, sizeof(int) * (size_t)(mb + 1), s)) != cudaSuccess)
            return cuda_fail(e, "cudaMemsetAsync(row_ptr_c)");
    }
    if (nnz_c_host)
    {
        if ((e = cudaMemcpyAsync(nnz_c_host, row_ptr_c + mb, sizeof(int), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
            return cuda_fail(e, "cudaMemcpyAsync(nnzC)");
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess)
            return cuda_fail(e, "cudaStreamSynchronize");
    }
    return KAMI_OK;
}

// ColIdxC from RowPtrC, entries at or past `cap` left out.
static int fill_colidx(int bsr, int mb, int kb, int nb, const int *row_ptr_a, const int *col_idx_a,
                       const int *row_ptr_b, const int *col_idx_b, const int *row_ptr_c, int *col_idx_c, int64_t cap,
                       void *stream)
{
    int st = check_bsr_args(bsr, mb, kb, nb, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b);
    if (st)
        return st;
    if (mb == 0 || nb == 0)
        return KAMI_OK;
    if (!row_ptr_c || !col_idx_c)
        return fail(KAMI_ERR_INVALID_VALUE, "spgemm: row_ptr_c / col_idx_c is NULL");
    int wpc;
    size_t smem;
    if ((st = bitmap_launch(nb, &wpc, &smem)))
        return st;
    if ((st = prep_bitmap_fn((const void *)spgemm_colfill_kernel, smem)))
        return st;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    spgemm_colfill_kernel<<<(mb + wpc - 1) / wpc, wpc * 32, smem, s>>>(mb, nb, row_ptr_a, col_idx_a, row_ptr_b,
                                                                      col_idx_b, row_ptr_c, col_idx_c, cap);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return cuda_fail(e, "spgemm_colfill_kernel");
    return KAMI_OK;
}

int kami_spgemm_bsr_fill_colidx(int bsr, int mb, int kb, int nb, const int *row_ptr_a, const int *col_idx_a,
                                const int *row_ptr_b, const int *col_idx_b, const int *row_ptr_c, int *col_idx_c,
                                void *stream)
{
    return fill_colidx(bsr, mb, kb, nb, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b, row_ptr_c, col_idx_c, INT64_MAX,
                       stream);
}

int kami_spgemm_bsr_symbolic_device(int bsr, int mb, int kb, int nb, const int *row_ptr_a, const int *col_idx_a,
                                    const int *row_ptr_b, const int *col_idx_b, int *row_ptr_c, int *col_idx_c,
                                    int64_t capacity, void *stream)
{
    if (capacity < 0 || (capacity > 0 && !col_idx_c))
        return fail(KAMI_ERR_INVALID_VALUE, "spgemm symbolic: capacity must be >= 0 with a column array");
    if (mb > 0 && nb > 0)
    {
        const int st0 = check_bsr_args(bsr, mb, kb, nb, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b);
        if (st0)
            return st0;
        if (!row_ptr_c)
            return fail(KAMI_ERR_INVALID_VALUE, "spgemm: row_ptr_c is NULL");
        // one pass with a decoupled look-back; past the flag array's capacity
        // the three-phase form with grid barriers
        const int stl = symbolic_lookback(mb, nb, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b, row_ptr_c, col_idx_c,
                                          capacity, reinterpret_cast<cudaStream_t>(stream));
        if (stl != KAMI_ERR_UNSUPPORTED)
            return stl;
        const int st1 = symbolic_fused(mb, nb, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b, row_ptr_c, col_idx_c,
                                       capacity, reinterpret_cast<cudaStream_t>(stream));
        if (st1 != KAMI_ERR_UNSUPPORTED)
            return st1;
    }
    // count + scan, with no copy of nnzC to the host
    int st = kami_spgemm_bsr_symbolic(bsr, mb, kb, nb, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b, row_ptr_c,
                                      nullptr, stream);
    if (st || mb == 0 || nb == 0 || capacity == 0)
        return st;
    int wpc;
    size_t smem;
    if ((st = bitmap_launch(nb, &wpc, &smem)))
        return st;
    if ((st = prep_bitmap_fn((const void *)spgemm_colfill_kernel, smem)))
        return st;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    spgemm_colfill_kernel<<<(mb + wpc - 1) / wpc, wpc * 32, smem, s>>>(mb, nb, row_ptr_a, col_idx_a, row_ptr_b,
                                                                      col_idx_b, row_ptr_c, col_idx_c, capacity);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return cuda_fail(e, "spgemm_colfill_kernel");
    return KAMI_OK;
}

int kami_spgemm_bsr_numeric(kami_dtype_t in_type, kami_dtype_t out_type, int bsr, int mb, int kb, int nb,
                            const int *row_ptr_a, const int *col_idx_a, const void *val_a, const int *row_ptr_b,
                            const int *col_idx_b, const void *val_b, const int *row_ptr_c, const int *col_idx_c,
                            void *val_c, int64_t nnz_c, double alpha, double beta, int num_iter, void *stream)
{
    return kami_spgemm_bsr_numeric_variant(KAMI_VARIANT_AUTO, in_type, out_type, bsr, mb, kb, nb, row_ptr_a,
                                           col_idx_a, val_a, row_ptr_b, col_idx_b, val_b, row_ptr_c, col_idx_c,
                                           val_c, nnz_c, alpha, beta, num_iter, stream);
}

// The numeric pass; fill: ColIdxC is written too (col_idx_c is then an output).
static int numeric_pass(bool fill, kami_variant_t variant, kami_dtype_t in_type, kami_dtype_t out_type, int bsr,
                        int mb, int kb, int nb, const int *row_ptr_a, const int *col_idx_a,
                        const void *val_a, const int *row_ptr_b, const int *col_idx_b, const void *val_b,
                        const int *row_ptr_c, int *col_idx_c, void *val_c, int64_t nnz_c,
                        double alpha, double beta, int num_iter, void *stream)
{
    if (variant != KAMI_VARIANT_AUTO && variant != KAMI_VARIANT_MMA_SYNC && variant != KAMI_VARIANT_TCGEN05)
        return fail(KAMI_ERR_INVALID_VALUE, "spgemm numeric: variant must be AUTO, MMA_SYNC or TCGEN05");
    int st = check_bsr_args(bsr, mb, kb, nb, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b);
    if (st)
        return st;
    if (in_type != KAMI_F16 && in_type != KAMI_BF16)
        return fail(KAMI_ERR_UNSUPPORTED, "spgemm numeric: FP16/BF16 tiles only");
    if (out_type != KAMI_F32 && out_type != KAMI_F16 && out_type != KAMI_BF16)
        return fail(KAMI_ERR_UNSUPPORTED, "spgemm numeric: FP32/FP16/BF16 output only");
    if (num_iter < 1 || nnz_c < 0)
        return fail(KAMI_ERR_INVALID_VALUE, "spgemm numeric: num_iter >= 1 and nnz_c >= 0 required");
    if (nnz_c == 0 || mb == 0)
        return KAMI_OK;
    // val_a / val_b may be NULL for an operand without entries (nothing is read)
    if (!row_ptr_c || !col_idx_c || !val_c)
        return fail(KAMI_ERR_INVALID_VALUE, "spgemm numeric: null pointer");
    if ((reinterpret_cast<uintptr_t>(val_a) & 7) || (reinterpret_cast<uintptr_t>(val_b) & 1) ||
        (reinterpret_cast<uintptr_t>(val_c) & 7))
        return fail(KAMI_ERR_MISALIGNED, "spgemm numeric: tile arrays must be 8-byte aligned");
    SpNumArgs p{};
    p.mb = mb;
    p.nb = nb;
    p.rpa = row_ptr_a;
    p.cia = col_idx_a;
    p.rpb = row_ptr_b;
    p.cib = col_idx_b;
    p.rpc = row_ptr_c;
    p.cic = p.cic_out = col_idx_c;
    p.va = reinterpret_cast<const uint16_t *>(val_a);
    p.vb = reinterpret_cast<const uint16_t *>(val_b);
    p.vc = val_c;
    p.nnzc = nnz_c;
    p.out_type = out_type;
    p.alpha = (float)alpha;
    p.beta = (float)beta;
    p.num_iter = num_iter;
    p.push = PushOut{val_c, out_type, p.beta != 0.f, p.alpha, p.beta};
    const int64_t grid = (nnz_c + 7) / 8;
    if (grid > 0x7fffffff)
        return fail(KAMI_ERR_UNSUPPORTED, "spgemm numeric: too many C tiles");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const bool aligned16 = !(reinterpret_cast<uintptr_t>(val_a) & 15) && !(reinterpret_cast<uintptr_t>(val_b) & 15);
    const bool tc_ok = aligned16 && !(reinterpret_cast<uintptr_t>(val_c) & 15);
    if (variant == KAMI_VARIANT_TCGEN05 && !tc_ok)
        return fail(KAMI_ERR_MISALIGNED, "spgemm numeric (tcgen05): tile arrays must be 16-byte aligned");
    const bool tc = variant == KAMI_VARIANT_TCGEN05 || (variant == KAMI_VARIANT_AUTO && tc_ok && spgemm_auto_tc05());
    // the push kernel fills ColIdxC itself, up to 16384 block columns
    const bool with = fill && !tc && aligned16 && nb <= kFillWords * 32;
    if (fill && !with && (st = fill_colidx(bsr, mb, kb, nb, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b, row_ptr_c,
                                           col_idx_c, nnz_c, stream)))
        return st;
    if (tc)
        return spgemm_tc05_launch(in_type == KAMI_BF16, mb, nnz_c, row_ptr_a, col_idx_a, row_ptr_b, col_idx_b, row_ptr_c,
                                  col_idx_c, val_a, val_b, val_c, out_type, alpha, beta, num_iter, s);
    if (aligned16) // one CTA per block-row, products pushed to their tiles
    {
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const cudaError_t el = push_launch(p, in_type == KAMI_BF16, with,
                                           mb <= kPushFewPerSm * sms || nnz_c >= (int64_t)kPushManyTiles * mb, s);
        return el == cudaSuccess ? KAMI_OK : cuda_fail(el, "spgemm_numeric_push_kernel");
    }
    if (in_type == KAMI_BF16)
        spgemm_numeric_kernel<true><<<(unsigned)grid, 256, 0, s>>>(p);
    else
        spgemm_numeric_kernel<false><<<(unsigned)grid, 256, 0, s>>>(p);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return cuda_fail(e, "spgemm_numeric_kernel");
    return KAMI_OK;
}

int kami_spgemm_bsr_numeric_variant(kami_variant_t variant, kami_dtype_t in_type, kami_dtype_t out_type, int bsr,
                                    int mb, int kb, int nb, const int *row_ptr_a, const int *col_idx_a,
                                    const void *val_a, const int *row_ptr_b, const int *col_idx_b, const void *val_b,
                                    const int *row_ptr_c, const int *col_idx_c, void *val_c, int64_t nnz_c,
                                    double alpha, double beta, int num_iter, void *stream)
{
    return numeric_pass(false, variant, in_type, out_type, bsr, mb, kb, nb, row_ptr_a, col_idx_a, val_a, row_ptr_b,
                        col_idx_b, val_b, row_ptr_c, const_cast<int *>(col_idx_c), val_c, nnz_c, alpha, beta, num_iter,
                        stream);
}

int kami_spgemm_bsr_fill_numeric(kami_variant_t variant, kami_dtype_t in_type, kami_dtype_t out_type, int bsr, int mb,
                                 int kb, int nb, const int *row_ptr_a, const int *col_idx_a, const void *val_a,
                                 const int *row_ptr_b, const int *col_idx_b, const void *val_b, const int *row_ptr_c,
                                 int *col_idx_c, void *val_c, int64_t nnz_c, double alpha, double beta, int num_iter,
                                 void *stream)
{
    return numeric_pass(true, variant, in_type, out_type, bsr, mb, kb, nb, row_ptr_a, col_idx_a, val_a, row_ptr_b,
                        col_idx_b, val_b, row_ptr_c, col_idx_c, val_c, nnz_c, alpha, beta, num_iter, stream);
}

} // extern "C"
