// f64_ring.cu -- batches of FP64 problems (each M, N, K <= 128) on the DMMA
// pipe (m16n8k8), uneven (a plan's descriptors) or uniform (one shape, three
// problem strides), in one persistent launch.
//
// At these sizes HBM and the DMMA pipe carry about the same load (64^3: 64 KB
// in, 32 KB out and 0.5 MFLOP, ~0.12 ms of either per 8192 problems), so the
// time is set by how well one overlaps the other and by what stands between
// them.  One CTA per SM walks its share of the batch through a ring of shared
// memory:
//   parts       C is cut into parts of at most 16 tiles of 16 x 16, a row block
//               of A times a row block of B.  A part of packed rows and at most
//               kWholeMax bytes is copied whole, as two bulk copies of its
//               blocks exactly as they lie in memory: a small problem costs two
//               instructions and the bytes it has, and many are in flight at
//               once.  Small problems of a uniform batch that follow one
//               another in memory share a part.  Other parts arrive in chunks
//               of K, a bulk copy per row into padded rows (16-byte cp.async
//               instead measured the same or slower: it takes the load
//               pipe's cycles from the multiplying warps).
//   warps 16-19 copy, taking turns at the chunks.  Where a chunk goes and which
//               earlier chunk must be gone is worked out beforehand (by the
//               plan, or by a division for a uniform batch), so the four need
//               not agree on anything and the ~1000 cycles that a chunk costs
//               its warp pass four at a time (one warp, or four that keep the
//               ring's state together: 650-1100 cycles a chunk, which bound
//               every problem below ~24 KB).
//   warps 0-15  multiply.  A part's tiles are dealt to the warps in turn, the
//               deal continuing from part to part (a fixed start gave warp 0
//               a tile of every problem and left the others idle on the small
//               ones), at most one per warp, its accumulators in registers
//               over the part's chunks; C is stored from there.  A warp
//               without a tile passes a chunk by in some twenty instructions.
//               The code of a tile is kept short: with two tiles a warp and
//               every case unrolled (41 KB of code) the warps mostly waited
//               for instructions, ~1200 cycles for a tile of one k-step.
// The copying warp writes a record per chunk (where it lies, its shape, whose
// tile comes first) beside the ring; full[s] publishes record and bytes,
// empty[s] collects the sixteen warps.
//
// Bank conflicts.  A fragment fetch is one 16-byte load per lane (lane 4g + t
// reads elements 2t, 2t + 1 of a k-step in row g; the k index is permuted
// alike in A and B); eight lanes, i.e. two rows, go out together.  Rows an odd
// multiple of 64 bytes apart (K = 8 mod 16, and padded rows) fall into
// different halves of the banks.  Rows a multiple of 128 bytes apart (K = 0
// mod 16, packed) would collide, so there the odd rows fetch the two k-steps
// of a pair in the other order and exchange them in registers: the DMMA pipe
// takes 64 cycles per instruction and scheduler, which leaves the issue slots
// for it.
//
// Rows past M and N repeat the last row (their results are not stored),
// columns past K are zeroed in registers.  Every wait is bounded; a wait that
// gives up sets g_f64r_error and ends its warp's loop.
#include <algorithm>
#include <cstdint>
#include <mutex>
#include <vector>

#include "grouped.cuh"
#include "kami_common.cuh"
#include "launch.cuh"
#include "ring.cuh"
#include "tc05_ptx.cuh"

namespace kami {

int fail(int code, const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);

// device status of the bounded waits (read and cleared by kami_device_status)
__device__ int g_f64r_error = 0;

namespace {

using namespace ring;

constexpr int kWarps = 16;                  // computing warps
constexpr int kCopyWarps = 4;               // warps kWarps .. copy
constexpr int kThreads = (kWarps + kCopyWarps) * 32;
constexpr int kRing = 224 * 1024;           // bytes of staged operands
constexpr int kWholeMax = 72 * 1024;        // bytes of a part copied whole: three fit the ring
constexpr int kGroupMax = 16 * 1024;        // bytes of a part of several problems
constexpr int kChunk = 64;                  // k values of a chunk at most (128 rows: three chunks fit the ring)

struct __align__(16) Rec
{
    uint32_t sa, sb;    // shared addresses of the chunk's A and B rows
    uint32_t pitch_k;   // their row stride in bytes | k values << 16
    uint32_t hdr;       // tiles | warp of tile 0 << 6 | kExchange ... | M << 16 | N << 24
    int64_t c_off;      // element offset of C
    int ldc;
    uint32_t inv;       // ceil(65536 / tiles per row of C)
};
constexpr uint32_t kExchange = 1u << 10, kFirst = 1u << 11, kLast = 1u << 12;
constexpr int kSmem = kRing + kRecs * (int)sizeof(Rec) + 2 * kRecs * 8 + 128;
static_assert(kSmem <= 227 * 1024, "f64 ring kernel: shared memory");

// A chunk as the copying warps take it: the record (its addresses relative to
// the ring), where it comes from, and what has to come before it (ring.cuh).
struct __align__(16) ChunkDesc
{
    Rec r;
    int64_t a_off, b_off; // elements
    uint16_t na, nb;      // rows of A and B
    int ld;               // 0: copied whole; a plan's row stride (a uniform batch has its own two)
    int dep, land;
};
static_assert(sizeof(ChunkDesc) == 64, "chunk descriptor");

// a uniform batch: problem i at i * stride, cut into mp x np parts of mb x nb,
// or `group` consecutive problems to a part
struct Uniform
{
    int M, N, K, lda, ldb, ldc;
    int64_t batch, sA, sB, sC;
    int mb, nb, mp, np;
    int group, whole;
    int kc, nk;        // k values of a chunk, chunks of a part
    int pitch, bytes;  // of the largest chunk: row stride, ring bytes of a slot
    int slots;
    int ahead0, ahead; // chunks in flight at most, while the ring fills (kAhead rounded down) and then
    int tiles;         // 16 x 16 tiles of one problem, for parts of several
    uint32_t inv;      // ceil(65536 / tiles)
    uint32_t inv_row[9]; // ceil(65536 / i)
};

struct RingParams
{
    GroupedParams p;
    const ChunkDesc *chunks; // a plan's chunks, null for a uniform batch
    Uniform u;
    uint64_t timeout_ns;
};

__device__ __forceinline__ void ring_flag(int code) { atomicExch(&g_f64r_error, code); }

__device__ __forceinline__ double2 lds_d2(uint32_t a)
{
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}

__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double a2, double a3, double b0, double b1)
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
                 : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// a 16 x 16 tile's four fragment rows: A rows g and g + 8, B rows (columns of
// C) g and g + 8, as shared addresses of this lane's elements of k-step 0
struct TileAt
{
    uint32_t a0, a1, b0, b1;
};

// one k-step of 8 of a tile; two: its second n8 half lies inside C
__device__ __forceinline__ void step(const double2 &a0, const double2 &a1, const double2 &b0, const double2 &b1, bool two,
                                     double (&acc)[2][4])
{
    dmma(acc[0], a0.x, a1.x, a0.y, a1.y, b0.x, b0.y);
    if (two)
        dmma(acc[1], a0.x, a1.x, a0.y, a1.y, b1.x, b1.y);
}

__device__ __forceinline__ void exchange(bool odd, double2 &x, double2 &y)
{
    const double2 u = x, v = y;
    x.x = odd ? v.x : u.x;
    x.y = odd ? v.y : u.y;
    y.x = odd ? u.x : v.x;
    y.y = odd ? u.y : v.y;
}

// one tile of a staged chunk, over its kv values of k: pairs of k-steps (odd:
// this lane's row fetches a pair's second step first), then what is left, the
// lanes past K multiplying zeros
__device__ __forceinline__ void tile_product(const TileAt &t, int kv, bool two, bool odd, int tq, double (&acc)[2][4])
{
    const uint32_t o = odd ? 64 : 0, pairs = (uint32_t)(kv & ~15) * 8;
#pragma unroll 1
    for (uint32_t k = 0; k < pairs; k += 128)
    {
        const uint32_t f = k + o, s = k + (o ^ 64);
        double2 a0 = lds_d2(t.a0 + f), c0 = lds_d2(t.a0 + s);
        double2 a1 = lds_d2(t.a1 + f), c1 = lds_d2(t.a1 + s);
        double2 b0 = lds_d2(t.b0 + f), d0 = lds_d2(t.b0 + s);
        double2 b1 = lds_d2(t.b1 + f), d1 = lds_d2(t.b1 + s);
        exchange(odd, a0, c0);
        exchange(odd, a1, c1);
        exchange(odd, b0, d0);
        exchange(odd, b1, d1);
        step(a0, a1, b0, b1, two, acc);
        step(c0, c1, d0, d1, two, acc);
    }
#pragma unroll 1
    for (int k = kv & ~15; k < kv; k += 8)
    {
        // (a partial step may read past the row, into bytes of the ring or the
        // records behind it)
        double2 a0 = lds_d2(t.a0 + k * 8), a1 = lds_d2(t.a1 + k * 8), b0 = lds_d2(t.b0 + k * 8), b1 = lds_d2(t.b1 + k * 8);
        if (k + 2 * tq >= kv)
            a0 = a1 = b0 = b1 = make_double2(0.0, 0.0);
        step(a0, a1, b0, b1, two, acc);
    }
}

// The tile's C, rows r and r + 8, columns c, c + 1, c + 8, c + 9 of this lane.
// alpha 1 and beta 0 take no FP64 arithmetic: it would queue behind the other
// warps' DMMAs on the same pipe.
__device__ __forceinline__ void store_tile(double *Cb, int M, int N, int ldc, bool vec, bool plain, double alpha,
                                           double beta, int r, int c, double (&acc)[2][4])
{
    double *q = Cb + (int64_t)r * ldc + c;
    if (plain && vec && __all_sync(0xffffffffu, r + 8 < M && c + 9 < N))
    {
        double *q8 = q + 8 * (int64_t)ldc;
        *reinterpret_cast<double2 *>(q) = make_double2(acc[0][0], acc[0][1]);
        *reinterpret_cast<double2 *>(q + 8) = make_double2(acc[1][0], acc[1][1]);
        *reinterpret_cast<double2 *>(q8) = make_double2(acc[0][2], acc[0][3]);
        *reinterpret_cast<double2 *>(q8 + 8) = make_double2(acc[1][2], acc[1][3]);
        return;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int n = 0; n < 2; ++n)
        {
            double *w = q + h * 8 * (int64_t)ldc + n * 8;
            double v0 = acc[n][2 * h], v1 = acc[n][2 * h + 1];
            const bool in0 = r + 8 * h < M && c + 8 * n < N, in1 = in0 && c + 8 * n + 1 < N;
            if (!plain)
            {
                v0 = alpha * v0 + (in0 && beta != 0.0 ? beta * w[0] : 0.0);
                v1 = alpha * v1 + (in1 && beta != 0.0 ? beta * w[1] : 0.0);
            }
            if (in1 && vec)
                *reinterpret_cast<double2 *>(w) = make_double2(v0, v1);
            else
            {
                if (in0)
                    w[0] = v0;
                if (in1)
                    w[1] = v1;
            }
        }
}

// rows of `bytes` bytes: the row stride of a chunk's padded rows, an odd multiple of 64
__host__ __device__ constexpr int padded(int bytes) { return ((bytes + 63) & ~127) + 64; }

// chunk j of a CTA's share of a uniform batch, parts first, first + stride, ...
__device__ __forceinline__ ChunkDesc uniform_chunk(const Uniform &u, int64_t first, int j, int stride)
{
    ChunkDesc d;
    // (no division where there is nothing to divide: it delays the first copies)
    const int pj = u.nk == 1 ? j : j / u.nk, k0 = (j - pj * u.nk) * u.kc, kv = min(u.kc, u.K - k0);
    const int64_t part = first + (int64_t)pj * stride;
    int M = u.M, N = u.N, n = 1, r0 = 0, c0 = 0;
    int64_t prob;
    if (u.group > 1)
    {
        prob = part * u.group;
        n = (int)min((int64_t)u.group, u.batch - prob);
    }
    else
    {
        prob = u.mp * u.np == 1 ? part : part / (u.mp * u.np);
        const int q = (int)(part - prob * (u.mp * u.np)), pm = q / u.np;
        r0 = pm * u.mb;
        c0 = (q - pm * u.np) * u.nb;
        M = min(u.mb, M - r0);
        N = min(u.nb, N - c0);
    }
    const int nf = (N + 15) >> 4, T = ((M + 15) >> 4) * nf * n;
    d.na = (uint16_t)(M * n);
    d.nb = (uint16_t)(N * n);
    d.r.sa = (uint32_t)(j % u.slots * u.bytes);
    d.r.sb = d.r.sa + up128(d.na * u.pitch);
    d.r.pitch_k = (uint32_t)(u.pitch | kv << 16);
    // the deal: parts of one size class follow one another, so the part's
    // number times its tiles continues it closely enough
    d.r.hdr = (uint32_t)T | (uint32_t)(pj * T & (kWarps - 1)) << 6 | (u.whole && u.K % 16 == 0 ? kExchange : 0u) |
              (k0 == 0 ? kFirst : 0u) | (k0 + kv == u.K ? kLast : 0u) | (uint32_t)M << 16 | (uint32_t)N << 24;
    d.r.c_off = prob * u.sC + (int64_t)r0 * u.ldc + c0;
    d.r.ldc = u.ldc;
    d.r.inv = u.inv_row[nf];
    d.a_off = prob * u.sA + (int64_t)r0 * u.lda + k0;
    d.b_off = prob * u.sB + (int64_t)c0 * u.ldb + k0;
    d.ld = !u.whole;
    d.dep = j - u.slots;
    d.land = j - (j < u.slots ? u.ahead0 : u.ahead);
    return d;
}

// ---- copying warp cw: of the CTA's n chunks, every kCopyWarps-th one that is
// copied whole, and its share of the rows of all others ----
__device__ __forceinline__ void copy_chunks(const RingParams &rp, uint8_t *smem, Rec *recs, uint64_t *full,
                                            uint64_t *empty, int64_t first, int n, int stride, int cw,
                                            int lane)
{
    const uint64_t limit = rp.timeout_ns;
    const uint8_t *A = reinterpret_cast<const uint8_t *>(rp.p.A), *B = reinterpret_cast<const uint8_t *>(rp.p.B);
    const uint32_t ring = tc::smem_u32(smem);
    int gone = -1; // the chunks up to this one are known to be done with
    bool ok = true;
    // 32 chunks at a time, one to a lane; a plan's next 32 already on their way
    ChunkDesc next{};
    if (!rp.chunks)
        next = uniform_chunk(rp.u, first, lane, stride);
    else if (lane < n)
        next = rp.chunks[first + lane];
    __syncthreads(); // barriers initialised
    int j = 0;
    for (int j0 = 0; j0 < n && ok; j0 += 32)
    {
        const ChunkDesc d = rp.chunks || j0 == 0 ? next : uniform_chunk(rp.u, first, j0 + lane, stride);
        if (rp.chunks && j0 + 32 + lane < n)
            next = rp.chunks[first + j0 + 32 + lane];
        uint32_t todo = __ballot_sync(0xffffffffu, j0 + lane < n && (d.ld != 0 || lane % kCopyWarps == cw));
        for (; todo; todo &= todo - 1)
        {
            const int l = __ffs(todo) - 1;
            j = j0 + l;
            const int s = j % kRecs;
            ok = wait_gone(empty, __shfl_sync(0xffffffffu, d.dep, l), gone, limit) &&
                 wait_landed(full, empty, __shfl_sync(0xffffffffu, d.land, l), gone, limit);
            if (!ok)
            {
                if (lane == 0)
                    ring_flag(1);
                break;
            }
            if (lane == l && l % kCopyWarps == cw)
            {
                Rec r = d.r;
                const uint32_t row = (r.pitch_k >> 16) * 8;
                r.sa += ring;
                r.sb += ring;
                recs[s] = r;
                tc::mbar_expect_tx(&full[s], (uint32_t)(d.na + d.nb) * row);
                if (d.ld == 0)
                {
                    tc::bulk_g2s(smem + d.r.sa, A + d.a_off * 8, (uint32_t)d.na * row, &full[s]);
                    tc::bulk_g2s(smem + d.r.sb, B + d.b_off * 8, (uint32_t)d.nb * row, &full[s]);
                }
            }
            __syncwarp();
            const int ld = __shfl_sync(0xffffffffu, d.ld, l);
            if (ld == 0)
                continue;
            const int64_t la = (rp.chunks ? ld : rp.u.lda) * 8ll, lb = (rp.chunks ? ld : rp.u.ldb) * 8ll;
            const int na = __shfl_sync(0xffffffffu, (int)d.na, l), nb = __shfl_sync(0xffffffffu, (int)d.nb, l);
            const uint32_t sa = __shfl_sync(0xffffffffu, d.r.sa, l), sb = __shfl_sync(0xffffffffu, d.r.sb, l);
            const uint32_t pk = __shfl_sync(0xffffffffu, d.r.pitch_k, l), pitch = pk & 0xffff, row = (pk >> 16) * 8;
            const uint8_t *pa = A + __shfl_sync(0xffffffffu, d.a_off, l) * 8;
            const uint8_t *pb = B + __shfl_sync(0xffffffffu, d.b_off, l) * 8;
            for (int m = cw + kCopyWarps * lane; m < na + nb; m += 32 * kCopyWarps)
                tc::bulk_g2s(smem + (m < na ? sa + m * pitch : sb + (m - na) * pitch),
                             m < na ? pa + m * la : pb + (m - na) * lb, row, &full[s]);
        }
    }
    // No copy may still be landing when the CTA exits: the computing warps wait
    // for every chunk, unless a wait has failed.
    for (int q = max(0, j + 1 - kRecs); !ok && q < j; ++q)
        if (!tc::mbar_wait_bounded(&full[q % kRecs], (q / kRecs) & 1, limit))
        {
            ring_flag(2);
            break;
        }
}

__global__ void __launch_bounds__(kThreads, 1) f64_ring_kernel(const __grid_constant__ RingParams rp)
{
    const GroupedParams &p = rp.p;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((128u - (tc::smem_u32(smem_raw) & 127u)) & 127u);
    Rec *recs = reinterpret_cast<Rec *>(smem + kRing);
    uint64_t *full = reinterpret_cast<uint64_t *>(recs + kRecs);
    uint64_t *empty = full + kRecs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0)
    {
        static_assert(kRecs == 32, "one record's barriers per lane");
        tc::mbar_init(&full[lane], 1);
        tc::mbar_init(&empty[lane], kWarps);
        tc::fence_mbar_init();
    }
    wait_for_previous();
    // this CTA's chunks: a plan's list, or a share of the batch's parts
    int64_t first;
    int n, stride = 1;
    if (rp.chunks)
    {
        first = p.cta_begin[blockIdx.x];
        n = p.cta_begin[blockIdx.x + 1] - (int)first;
    }
    else
    {
        const Uniform &u = rp.u;
        if (u.mp * u.np > 1)
        {
            // a problem's parts share operands: consecutive parts
            const int64_t parts = u.batch * (u.mp * u.np);
            first = parts * blockIdx.x / gridDim.x;
            n = (int)(parts * (blockIdx.x + 1) / gridDim.x - first);
        }
        else
        {
            const int64_t parts = (u.batch + u.group - 1) / u.group;
            first = blockIdx.x;
            n = (int)((parts - blockIdx.x + gridDim.x - 1) / gridDim.x);
            stride = gridDim.x;
        }
        n *= u.nk;
    }
    if (warp >= kWarps)
    {
        copy_chunks(rp, smem, recs, full, empty, first, n, stride, warp - kWarps, lane);
        return;
    }
    __syncthreads(); // barriers initialised

    const uint64_t limit = rp.timeout_ns;
    const int gq = lane >> 2, tq = lane & 3;
    const bool plain = p.alpha == 1.0 && p.beta == 0.0;
    // this warp's tile of the current part
    int M = 0, N = 0, r0 = 0, cb = 0;
    TileAt off{};
    int64_t c_more = 0;
    double acc[2][4] = {};
    for (int j = 0; j < n; ++j)
    {
        const int s = j % kRecs;
        if (!__all_sync(0xffffffffu, tc::mbar_wait_bounded(&full[s], (j / kRecs) & 1, limit)))
        {
            if (lane == 0)
                ring_flag(3);
            return;
        }
        const uint4 ra = *reinterpret_cast<const uint4 *>(&recs[s]); // sa, sb, pitch_k, hdr
        const uint32_t hdr = ra.w;
        int t = (warp - (hdr >> 6)) & (kWarps - 1);
        if (t >= (int)(hdr & 63))
        {
            __syncwarp();
            if (lane == 0)
                tc::mbar_arrive(&empty[s]);
            continue;
        }
        if (hdr & kFirst)
        {
            M = (hdr >> 16) & 255;
            N = hdr >> 24;
            // the tile's problem among several (a plan's parts have one: inv 0)
            const int q = (t * rp.u.inv) >> 16, pitch = ra.z & 0xffff;
            t -= q * rp.u.tiles;
            const int tr = (t * recs[s].inv) >> 16;
            c_more = q * rp.u.sC;
            r0 = tr * 16 + gq;
            cb = (t - tr * ((N + 15) >> 4)) * 16;
            off.a0 = (q * M + min(r0, M - 1)) * pitch + tq * 16;
            off.a1 = (q * M + min(r0 + 8, M - 1)) * pitch + tq * 16;
            off.b0 = (q * N + min(cb + gq, N - 1)) * pitch + tq * 16;
            off.b1 = (q * N + min(cb + gq + 8, N - 1)) * pitch + tq * 16;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                acc[0][e] = acc[1][e] = 0.0;
        }
        const TileAt at{ra.x + off.a0, ra.x + off.a1, ra.y + off.b0, ra.y + off.b1};
        const int64_t c_off = recs[s].c_off + c_more;
        const int ldc = recs[s].ldc;
#pragma unroll 1
        for (int it = 0; it < p.num_iter; ++it)
            tile_product(at, ra.z >> 16, cb + 8 < N, (hdr & kExchange) && (gq & 1), tq, acc);
        __syncwarp();
        if (lane == 0)
            tc::mbar_arrive(&empty[s]);
        if (hdr & kLast)
        {
            double *Cb = reinterpret_cast<double *>(p.C) + c_off;
            store_tile(Cb, M, N, ldc, !(ldc & 1) && !(reinterpret_cast<uintptr_t>(Cb) & 15), plain, p.alpha, p.beta,
                       r0, cb + 2 * tq, acc);
        }
    }
}

int launch_ring(const RingParams &rp, int ctas, cudaStream_t s)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev >= 64)
        return e != cudaSuccess ? cuda_fail(e, "cudaGetDevice") : KAMI_ERR_UNSUPPORTED;
    static std::once_flag once[64];
    static cudaError_t attr[64];
    std::call_once(once[dev], [&] {
        attr[dev] =
            cudaFuncSetAttribute((const void *)&f64_ring_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    });
    if (attr[dev] != cudaSuccess)
        return cuda_fail(attr[dev], "cudaFuncSetAttribute(f64_ring_kernel)");
    void *args[] = {const_cast<RingParams *>(&rp)};
    e = launch_overlapped((const void *)&f64_ring_kernel, dim3(ctas), dim3(kThreads), args, kSmem, s);
    if (e != cudaSuccess)
        return cuda_fail(e, "cudaLaunchKernel(f64_ring_kernel)");
    return KAMI_OK;
}

} // namespace

int f64_ring_smem() { return kSmem; }

// Cut of an M x N problem into parts of mb x nb (multiples of 16 unless whole)
// with at most a tile for each computing warp: the one that reads the fewest
// rows, M np + N mp; of equals one whose parts are copied whole, then the one
// of fewer parts.
static void ring_cut(int M, int N, int K, bool packed, int *mb, int *nb)
{
    *mb = M;
    *nb = N;
    if ((M + 15) / 16 * ((N + 15) / 16) <= kWarps)
        return; // uncut: no row is read twice
    int best = 1 << 30;
    for (int m = 1; m <= (M + 15) / 16; ++m)
        for (int n = 1; n <= (N + 15) / 16; ++n)
        {
            if ((M * n + N * m) * 256 >= best)
                continue;
            const int mf = ((M + 15) / 16 + m - 1) / m, nf = ((N + 15) / 16 + n - 1) / n;
            const bool whole = packed && (std::min(M, mf * 16) + std::min(N, nf * 16)) * K * 8 <= kWholeMax;
            const int cost = (M * n + N * m) * 256 + (whole ? 0 : 128) + m * n;
            if (mf * nf > kWarps || cost >= best)
                continue;
            best = cost;
            *mb = std::min(M, mf * 16);
            *nb = std::min(N, nf * 16);
        }
}

// How a part of `rows` rows comes: whole (returns true), or in equal chunks of
// kc k values, whole k-steps; pitch: the row stride.
static bool ring_chunks(int rows, int K, bool packed, int *kc, int *pitch)
{
    const bool whole = packed && rows * K * 8 <= kWholeMax;
    const int nk = std::max((K + kChunk - 1) / kChunk, (rows * K * 8 + kWholeMax - 1) / kWholeMax);
    *kc = whole ? K : std::min(K, ((K + nk - 1) / nk + 7) & ~7);
    *pitch = whole ? K * 8 : padded(*kc * 8);
    return whole;
}

// The chunks of a plan's problems (packed rows), list by list, placed in the
// ring: chunk after chunk, from the start again where the rest is too short.
size_t f64_ring_schedule(const std::vector<std::vector<int>> &lists, const int *M, const int *N, const int *K,
                         const int64_t *ao, const int64_t *bo, const int64_t *co, std::vector<char> *out,
                         std::vector<int> *begin)
{
    size_t problems = 0, count = 0;
    for (const auto &l : lists)
        problems += l.size();
    out->clear();
    out->reserve((problems + problems / 2) * sizeof(ChunkDesc));
    Placer placer(kRing);
    // one shape's problems follow one another in a plan's order of cost: cut once
    // (plan of 4000 128^3: 1.26 ms to create, 1.07 so)
    int cut[3] = {0, 0, 0}, mb = 0, nb = 0;
    for (size_t c = 0; c < lists.size(); ++c)
    {
        (*begin)[c] = (int)count;
        placer.clear();
        int deal = 0;
        for (int i : lists[c])
        {
            if (M[i] != cut[0] || N[i] != cut[1] || K[i] != cut[2])
                ring_cut(cut[0] = M[i], cut[1] = N[i], cut[2] = K[i], true, &mb, &nb);
            for (int r0 = 0; r0 < M[i]; r0 += mb)
                for (int c0 = 0; c0 < N[i]; c0 += nb)
                {
                    ChunkDesc d{};
                    const int m = std::min(mb, M[i] - r0), n = std::min(nb, N[i] - c0), k = K[i];
                    int kc, pitch;
                    const bool whole = ring_chunks(m + n, k, true, &kc, &pitch);
                    const int nf = (n + 15) / 16, T = (m + 15) / 16 * nf;
                    const int bytes = up128(m * pitch) + up128(n * pitch);
                    d.na = (uint16_t)m;
                    d.nb = (uint16_t)n;
                    d.ld = whole ? 0 : k;
                    d.r.ldc = N[i];
                    d.r.c_off = co[i] + (int64_t)r0 * N[i] + c0;
                    d.r.inv = (65535u + (uint32_t)nf) / (uint32_t)nf;
                    for (int k0 = 0; k0 < k; k0 += kc)
                    {
                        const int kv = std::min(kc, k - k0), at = placer.place(bytes, &d.dep, &d.land);
                        d.r.sa = (uint32_t)at;
                        d.r.sb = (uint32_t)(at + up128(m * pitch));
                        d.r.pitch_k = (uint32_t)(pitch | kv << 16);
                        d.r.hdr = (uint32_t)T | (uint32_t)deal << 6 | (whole && k % 16 == 0 ? kExchange : 0u) |
                                  (k0 == 0 ? kFirst : 0u) | (k0 + kv == k ? kLast : 0u) | (uint32_t)m << 16 |
                                  (uint32_t)n << 24;
                        d.a_off = ao[i] + (int64_t)r0 * k + k0;
                        d.b_off = bo[i] + (int64_t)c0 * k + k0;
                        const char *raw = reinterpret_cast<const char *>(&d);
                        out->insert(out->end(), raw, raw + sizeof(d));
                        ++count;
                    }
                    deal = (deal + T) % kWarps;
                }
        }
    }
    (*begin)[lists.size()] = (int)count;
    return count;
}

// a plan: chunks (f64_ring_schedule) on the device, p.cta_begin their lists
int f64_ring_plan_launch(const GroupedParams &p, const void *chunks, int ctas, cudaStream_t s)
{
    RingParams rp{};
    rp.p = p;
    rp.chunks = reinterpret_cast<const ChunkDesc *>(chunks);
    rp.timeout_ns = (uint64_t)(2e9 + (double)p.num_iter * 1e6); // generous: a chunk takes microseconds
    return launch_ring(rp, ctas, s);
}

// A uniform batch as the kernel takes it; returns its CTAs.
static int uniform_params(const GemmArgs &g, Uniform &u)
{
    u.M = g.M;
    u.N = g.N;
    u.K = g.K;
    u.lda = (int)g.lda;
    u.ldb = (int)g.ldb;
    u.ldc = (int)g.ldc;
    u.batch = g.batch;
    u.sA = g.sA;
    u.sB = g.sB;
    u.sC = g.sC;
    const bool packed = (g.lda == g.K || g.M == 1) && (g.ldb == g.K || g.N == 1);
    ring_cut(g.M, g.N, g.K, packed, &u.mb, &u.nb);
    u.mp = (g.M + u.mb - 1) / u.mb;
    u.np = (g.N + u.nb - 1) / u.nb;
    u.whole = ring_chunks(u.mb + u.nb, g.K, packed, &u.kc, &u.pitch);
    u.nk = (g.K + u.kc - 1) / u.kc;
    // problems one after the other in A and in B: as many as give each warp a tile
    u.group = 1;
    u.tiles = (g.M + 15) / 16 * ((g.N + 15) / 16);
    if (u.whole && g.sA == (int64_t)g.M * g.K && g.sB == (int64_t)g.N * g.K)
        u.group = std::max(1, std::min(kWarps / u.tiles, kGroupMax / ((g.M + g.N) * g.K * 8)));
    u.inv = u.group > 1 ? (65535u + (uint32_t)u.tiles) / (uint32_t)u.tiles : 0u;
    for (uint32_t i = 1; i < 9; ++i)
        u.inv_row[i] = (65535u + i) / i;
    u.bytes = up128(u.mb * u.group * u.pitch) + up128(u.nb * u.group * u.pitch);
    u.slots = std::min(kRecs, kRing / u.bytes);
    u.ahead0 = std::min(kRecs, std::max(1, kAhead / u.bytes));
    u.ahead = std::min(kRecs, (kAhead + u.bytes - 1) / u.bytes);
    const int64_t parts = u.group > 1 ? (g.batch + u.group - 1) / u.group : g.batch * (u.mp * u.np);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (int)std::min<int64_t>(parts, sms);
}

// A uniform batch, A row-major and B N x K, M, N, K <= 128, 16-byte aligned
// rows and problems (checked by the callers); KAMI_ERR_UNSUPPORTED, nothing
// launched, where the strides exceed 32 bits.
int f64_ring_launch(const GemmArgs &g, cudaStream_t s)
{
    if (g.lda > 0x7fffffff || g.ldb > 0x7fffffff || g.ldc > 0x7fffffff)
        return fail(KAMI_ERR_UNSUPPORTED, "no kernel for M=%d N=%d K=%d with rows %lld, %lld, %lld apart", g.M, g.N, g.K,
                    (long long)g.lda, (long long)g.ldb, (long long)g.ldc);
    RingParams rp{};
    rp.p.A = g.A;
    rp.p.B = g.B;
    rp.p.C = g.C;
    rp.p.out_type = KAMI_F64;
    rp.p.alpha = g.alpha;
    rp.p.beta = g.beta;
    rp.p.num_iter = g.num_iter;
    rp.timeout_ns = (uint64_t)(2e9 + (double)g.num_iter * 1e6);
    const int ctas = uniform_params(g, rp.u);
    return launch_ring(rp, ctas, s);
}

// the launch of f64_ring_launch (kami_gemm_describe)
void f64_ring_info(const GemmArgs &g, LaunchInfo *info)
{
    Uniform u{};
    const int ctas = uniform_params(g, u);
    *info = LaunchInfo{KAMI_VARIANT_MMA_SYNC, KAMI_PARTITION_1D, 1, kThreads, kSmem,
                       ctas ? (int)((g.batch + ctas - 1) / ctas) : 0, ctas};
}

int f64_ring_read_error(int *flag)
{
    int v = 0, z = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_f64r_error, sizeof(int));
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbol(g_f64r_error, &z, sizeof(int));
    if (e != cudaSuccess)
        return cuda_fail(e, "reading the FP64 ring kernel's status");
    *flag = v;
    return KAMI_OK;
}

} // namespace kami
