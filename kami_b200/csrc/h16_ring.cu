// h16_ring.cu -- batches of FP16 / BF16 problems (each M, N, K <= 128) on the
// 5th-generation tensor cores, uneven (a plan's descriptors) or uniform (one
// shape, three problem strides), in one persistent launch.
//
// At these sizes the MMAs of a problem are a handful and its bytes a few KB:
// what counts is how few instructions and hand-offs each one takes and how many
// are on their way at once.  One CTA per SM runs four independent groups, each
// with its own list of problems, its own ring of shared memory (ring.cuh, 46 KB)
// and 128 columns of tensor memory (plans of large problems: two groups, with 92 KB):
//   warps 20 + 2 g, 21 + 2 g copy A's and B's rows by 16-byte cp.async straight
//               into the 128-byte-swizzled K-major layout the MMA reads (row r
//               at r * 128, 16-byte chunk c at c ^ (r % 8)), 64 values of K to
//               a chunk.  A chunk's place in the ring has its own size.
//   warp 16 + g issues the MMAs (M = 128 accumulator rows, N rounded up to 16)
//               into one of two accumulators of 64 columns, or one of 128 while
//               N > 64.
//   warps 4 g .. 4 g + 3 store C: warp q reads the accumulator's lanes from
//               32 q, then frees it.  Warp q of every group runs on the same
//               scheduler, so a problem of few rows does not always begin at
//               lane 0: its A tile is read from 0 .. 3 times 32 rows further up
//               (whatever lies there), which puts it into the lanes of warp 0
//               .. 3 in turn.
// Small problems are bound by this chain -- a problem lands, its MMAs are
// issued, they finish, the accumulator is read out -- so four of them run side
// by side, each two problems deep.  20000 uneven problems of 8 .. 128: one
// issuing thread per CTA and two CTAs per SM 95 us; one ring for the four
// groups, each having to pass the others' chunks by, 74 us, 46 of them with
// copies and stores taken out.
// Columns past K inside the last k-step are zero-filled by the copies; rows
// past M and N are whatever the ring holds and only reach rows and columns of
// the accumulator that are never stored (an MMA reads up to 128 rows from a
// tile's start: kSlack keeps that inside shared memory).  Every wait is
// bounded; a wait that gives up sets g_h16r_error and ends its role.
#include <algorithm>
#include <cstdint>
#include <mutex>
#include <type_traits>
#include <vector>

#include "grouped.cuh"
#include "kami_common.cuh"
#include "launch.cuh"
#include "ring.cuh"
#include "tc05_epi.cuh"
#include "tc05_ptx.cuh"

namespace kami {

int fail(int code, const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);

// device status of the bounded waits (read and cleared by kami_device_status)
__device__ int g_h16r_error = 0;

namespace {

constexpr int kGroups = 4;                  // of four warps each, with 128 columns of tensor memory
constexpr int kIssue = 4 * kGroups;         // first issuing warp (one per group)
constexpr int kCopy = kIssue + kGroups;     // first copying warp (two per group)
constexpr int kThreads = (kCopy + 2 * kGroups) * 32;
constexpr int kBytes = 46 * 1024;           // of a group's ring
constexpr int kRecs = 16;                   // chunks in flight at most in a group
constexpr int kFront = 12 * 1024;           // 96 rows of 128 bytes before the first ring's first tile
constexpr int kSlack = 17 * 1024;           // 128 rows of 128 bytes past the last ring's last tile

struct __align__(16) Rec
{
    uint32_t sa, sb; // shared addresses of the A and B tiles (rows rounded up to 8)
    uint32_t shape;  // M | N << 8 | K values of the chunk << 16 | kFirst | kLast
    int ldc;
    int64_t c_off;   // element offset of C
    int quad; // 32 quad: the accumulator lane of row 0
    int pad;
};
constexpr uint32_t kFirst = 1u << 24, kLast = 1u << 25;
constexpr int kBars = (2 * kRecs + 5) * kGroups;
constexpr int kSmem = kFront + kGroups * kBytes + kSlack + (kRecs + 2) * kGroups * (int)sizeof(Rec) + kBars * 8 + 16 + 1024;
static_assert(kSmem <= 227 * 1024, "16-bit ring kernel: shared memory");

// a chunk as the copying warps take it
struct __align__(16) ChunkDesc
{
    int64_t a_off, b_off, c_off; // elements
    uint32_t shape;              // as in Rec
    int at;                      // bytes into the ring
    int lda, ldb, ldc;
    int dep;                     // ring.cuh
    int pad[2];
};

// a uniform batch: problem i at i * stride
struct Uniform
{
    int M, N, K, lda, ldb, ldc;
    int64_t batch, sA, sB, sC;
    int nk, bytes, slots; // chunks of a problem, ring bytes of one, chunks that a ring holds
};

// How C is written, by value: read from the kernel's parameters by reference, it
// would be read again after every store, which for all the compiler knows has
// changed it (1000 x 48 x 128 x 64, FP32 out, alpha 2, beta 0.5: 59 us, 21 so;
// 4000 uneven problems of 8 .. 128, most of them of ragged N, 51 and 27).
struct Out
{
    void *C;
    int type;
    bool plain, read; // alpha 1 and beta 0; beta not 0
    float alpha, beta;
};

struct RingParams
{
    GroupedParams p;
    Out out; // from p
    const ChunkDesc *chunks; // a plan's chunks, null for a uniform batch
    Uniform u;
    uint64_t timeout_ns;
};

__host__ __device__ constexpr int up8(int x) { return (x + 7) & ~7; }
// 16-byte chunks of a row that the MMAs read: whole k-steps of 16
__host__ __device__ constexpr int row_chunks(int K) { return ((K + 15) & ~15) >> 3; }

__device__ __forceinline__ void ring_flag(int code) { atomicExch(&g_h16r_error, code); }

__device__ __forceinline__ void cp16(uint32_t dst, const void *src, bool valid)
{
    // src-size 0 writes 16 zero bytes
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
// arrive (once, counted in the barrier's expected arrivals) on `bar` when
// every cp.async this thread has issued so far has completed
__device__ __forceinline__ void cp_arrive_on(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// 32 accumulator columns of this thread's lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                   "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                   "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                   "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                 : "r"(taddr)
                 : "memory");
}

// An operand's rows into a swizzled tile: 2^lg lanes (at most 8) to a row, the
// first row_chunks(K) of them copying.
__device__ __forceinline__ void copy_tile(uint32_t tile, const uint8_t *src, int rows, int ld, int K, int lg, int lane)
{
    const int q = lane & ((1 << lg) - 1), step = 32 >> lg;
    if (q >= row_chunks(K))
        return;
    const bool valid = q * 8 < K;
    int r = lane >> lg;
    src += (int64_t)r * ld + (valid ? q * 16 : 0);
    const int64_t down = (int64_t)step * ld;
#pragma unroll 4
    for (; r < rows; r += step, src += down)
        cp16(tile + r * 128 + (((q ^ r) & 7) << 4), src, valid);
}

// chunk j of a group's share of a uniform batch, problems first, first + stride, ...
__device__ __forceinline__ ChunkDesc uniform_chunk(const Uniform &u, int64_t first, int j, int stride)
{
    ChunkDesc d;
    const int pj = u.nk == 1 ? j : j >> 1, k0 = u.nk == 1 ? 0 : (j & 1) * 64; // (K <= 128)
    const int64_t prob = first + (int64_t)pj * stride;
    d.a_off = prob * u.sA + k0;
    d.b_off = prob * u.sB + k0;
    d.c_off = prob * u.sC;
    d.shape = (uint32_t)(u.M | u.N << 8 | min(64, u.K - k0) << 16) | (k0 == 0 ? kFirst : 0u) |
              (k0 + 64 >= u.K ? kLast : 0u);
    d.at = j % u.slots * u.bytes;
    d.lda = u.lda;
    d.ldb = u.ldb;
    d.ldc = u.ldc;
    d.dep = j - u.slots;
    return d;
}

// ---- copying warp: operand B (or A) of the group's n chunks ----
__device__ __forceinline__ void copy_chunks(const RingParams &rp, uint32_t base, Rec *recs, uint64_t *full,
                                            uint64_t *empty, int64_t first, int n, int stride, bool B, int lane)
{
    const uint64_t limit = rp.timeout_ns;
    const uint8_t *X = reinterpret_cast<const uint8_t *>(B ? rp.p.B : rp.p.A);
    int gone = -1;
    bool ok = true;
    auto fetch = [&](int j) {
        ChunkDesc d{};
        if (j < n)
            d = rp.chunks ? rp.chunks[first + j] : uniform_chunk(rp.u, first, j, stride);
        return d;
    };
    // 32 chunks at a time, one to a lane; a plan's next 32 already on their way
    ChunkDesc next = fetch(lane);
    __syncthreads(); // barriers initialised
    for (int j0 = 0; j0 < n && ok; j0 += 32)
    {
        const ChunkDesc d = rp.chunks || j0 == 0 ? next : fetch(j0 + lane);
        if (rp.chunks)
            next = fetch(j0 + 32 + lane);
        for (int l = 0; l < 32 && j0 + l < n; ++l)
        {
            const int s = (j0 + l) % kRecs;
            ok = ring::wait_gone<kRecs>(empty, __shfl_sync(0xffffffffu, d.dep, l), gone, limit);
            if (!ok)
            {
                if (lane == 0)
                    ring_flag(1);
                break;
            }
            const uint32_t shape = __shfl_sync(0xffffffffu, d.shape, l);
            const int M = shape & 255, N = (shape >> 8) & 255, K = (shape >> 16) & 255;
            const uint32_t sa = base + __shfl_sync(0xffffffffu, d.at, l), sb = sa + up8(M) * 128;
            const int64_t xo = __shfl_sync(0xffffffffu, B ? d.b_off : d.a_off, l);
            const int ld = __shfl_sync(0xffffffffu, B ? d.ldb : d.lda, l);
            const int lg = 32 - __clz(row_chunks(K) - 1); // 2, 4 or 8 lanes to a row
            copy_tile(B ? sb : sa, X + xo * 2, B ? N : M, ld * 2, K, lg, lane);
            cp_arrive_on(&full[s]); // this lane's copies: 64 of the 65 arrivals
            if (!B && lane == l)
            {
                recs[s] = Rec{sa, sb, shape, d.ldc, d.c_off, 0, 0};
                tc::mbar_arrive(&full[s]);
            }
            __syncwarp();
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// 16 accumulator rows x 32 columns of the lanes at taddr: lane 4g + t gets of
// each 8 columns 2t, 2t + 1 of row g, then of row g + 8
__device__ __forceinline__ void tmem_ld_frag32(uint32_t taddr, uint4 (&v)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                 "[%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[1].x), "=r"(v[1].y), "=r"(v[1].z),
                   "=r"(v[1].w), "=r"(v[2].x), "=r"(v[2].y), "=r"(v[2].z), "=r"(v[2].w), "=r"(v[3].x), "=r"(v[3].y),
                   "=r"(v[3].z), "=r"(v[3].w)
                 : "r"(taddr)
                 : "memory");
}

// 16 rows x 16 columns of fragments v, of which rows x cols are the problem's, to
// q: T is FP32's float or the 16-bit types' uint16_t, pairs: columns come in pairs
// that may be read and stored at once.  C's old values are all asked for before the
// first is used.
template <class T>
__device__ __forceinline__ void store_patch(const Out &o, const uint4 &v0, const uint4 &v1, T *q, int64_t down,
                                            bool pairs, int rows, int cols)
{
    const bool bf = o.type == KAMI_BF16;
    const int lane = threadIdx.x & 31, gq = lane >> 2, c = 2 * (lane & 3);
    // pair i: columns 8 (i / 2) + c and the next, of row gq or (odd i) gq + 8
    float x[4][2] = {{__uint_as_float(v0.x), __uint_as_float(v0.y)}, {__uint_as_float(v0.z), __uint_as_float(v0.w)},
                     {__uint_as_float(v1.x), __uint_as_float(v1.y)}, {__uint_as_float(v1.z), __uint_as_float(v1.w)}};
    bool in0[4], in1[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
        in0[i] = gq + 8 * (i & 1) < rows && 4 * (i & 2) + c < cols;
        in1[i] = in0[i] && 4 * (i & 2) + c + 1 < cols;
    }
    if (!o.plain)
    {
        // (as they lie in memory: unpacked at once, each load would be waited for)
        using Word = std::conditional_t<sizeof(T) == 4, float2, uint32_t>;
        Word word[4] = {};
        T one[4][2] = {};
        if (o.read && pairs)
        {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (in0[i])
                    word[i] = *reinterpret_cast<const Word *>(q + (i & 1) * down + 4 * (i & 2));
        }
        else if (o.read)
        {
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                const T *w = q + (i & 1) * down + 4 * (i & 2);
                one[i][0] = in0[i] ? w[0] : T(0);
                one[i][1] = in1[i] ? w[1] : T(0);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            float y0, y1;
            if constexpr (sizeof(T) == 4)
            {
                y0 = pairs ? word[i].x : one[i][0];
                y1 = pairs ? word[i].y : one[i][1];
            }
            else
            {
                y0 = to_float(pairs ? (T)word[i] : one[i][0], bf);
                y1 = to_float(pairs ? (T)(word[i] >> 16) : one[i][1], bf);
            }
            x[i][0] = o.alpha * x[i][0] + (o.read ? o.beta * y0 : 0.f);
            x[i][1] = o.alpha * x[i][1] + (o.read ? o.beta * y1 : 0.f);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
        T *w = q + (i & 1) * down + 4 * (i & 2);
        T y[2];
        if constexpr (sizeof(T) == 4)
            y[0] = x[i][0], y[1] = x[i][1];
        else
        {
            const uint32_t h = pack2(x[i][0], x[i][1], bf);
            y[0] = (T)h, y[1] = (T)(h >> 16);
        }
        if (pairs)
        {
            if constexpr (sizeof(T) == 4)
            {
                if (in0[i])
                    *reinterpret_cast<float2 *>(w) = make_float2(y[0], y[1]);
            }
            else if (in0[i])
                *reinterpret_cast<ushort2 *>(w) = make_ushort2(y[0], y[1]);
        }
        else
        {
            if (in0[i])
                w[0] = y[0];
            if (in1[i])
                w[1] = y[1];
        }
    }
}

// Any other C: `rows` rows of the accumulator's lanes at taddr, N columns, to off.
// In fragment shape, so that a store covers eight rows of up to 32 bytes however
// they are aligned (a row per lane would spread it over 32 pieces).
__device__ __noinline__ void store_general(const Out &out, uint32_t taddr, int64_t off, int ldc, int rows, int N)
{
    const Out o = out;
    const int lane = threadIdx.x & 31, gq = lane >> 2, c = 2 * (lane & 3);
    const int64_t down = 8 * (int64_t)ldc;
    off += (int64_t)gq * ldc + c;
    for (int h = 0; h < 32 && h < rows; h += 16)
        for (int c0 = 0; c0 < N; c0 += 32)
        {
            uint4 v[4];
            tmem_ld_frag32(taddr + ((uint32_t)h << 16) + c0, v);
            const int64_t at = off + (int64_t)h * ldc + c0;
            if (o.type == KAMI_F32)
            {
                float *q = reinterpret_cast<float *>(o.C) + at;
                const bool pairs = !((ldc | N) & 1) && !(reinterpret_cast<uintptr_t>(q) & 7); // the same in all lanes
                store_patch(o, v[0], v[1], q, down, pairs, rows - h, N - c0);
                store_patch(o, v[2], v[3], q + 16, down, pairs, rows - h, N - c0 - 16);
            }
            else
            {
                uint16_t *q = reinterpret_cast<uint16_t *>(o.C) + at;
                const bool pairs = !((ldc | N) & 1) && !(reinterpret_cast<uintptr_t>(q) & 3);
                store_patch(o, v[0], v[1], q, down, pairs, rows - h, N - c0);
                store_patch(o, v[2], v[3], q + 16, down, pairs, rows - h, N - c0 - 16);
            }
        }
}

// Plain C with rows of whole aligned groups of eight: 32 columns of this
// thread's row, at off, 32 bytes (FP32; 16 in 16 bits) to a store; cols: what is
// left of the row.  (In fragment shape, the lanes of a row exchanging columns
// first so that a store covers eight rows of 128 bytes: 74 us against 66 for the
// uneven problems -- it is the instructions that count.)
__device__ __forceinline__ void store_row(const GroupedParams &p, int64_t off, int cols, const uint32_t (&v)[32])
{
    if (p.out_type == KAMI_F32)
    {
        float *c = reinterpret_cast<float *>(p.C) + off;
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (8 * b < cols)
                asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(c + 8 * b), "r"(v[8 * b]),
                             "r"(v[8 * b + 1]), "r"(v[8 * b + 2]), "r"(v[8 * b + 3]), "r"(v[8 * b + 4]),
                             "r"(v[8 * b + 5]), "r"(v[8 * b + 6]), "r"(v[8 * b + 7])
                             : "memory");
        return;
    }
    const bool bf = p.out_type == KAMI_BF16;
    uint16_t *c = reinterpret_cast<uint16_t *>(p.C) + off;
#pragma unroll
    for (int b = 0; b < 4; ++b)
        if (8 * b < cols)
        {
            uint32_t h[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                h[e] = pack2(__uint_as_float(v[8 * b + 2 * e]), __uint_as_float(v[8 * b + 2 * e + 1]), bf);
            *reinterpret_cast<uint4 *>(c + 8 * b) = make_uint4(h[0], h[1], h[2], h[3]);
        }
}

template <bool BF16, int GROUPS>
__global__ void __launch_bounds__(kThreads, 1) h16_ring_kernel(const __grid_constant__ RingParams rp)
{
    const GroupedParams &p = rp.p;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // 1024-byte alignment of the swizzle atoms
    uint8_t *smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
    Rec *recs_all = reinterpret_cast<Rec *>(smem + kFront + kGroups * kBytes + kSlack);
    Rec *grec_all = recs_all + kGroups * kRecs; // a group's two problems under way
    uint64_t *bars = reinterpret_cast<uint64_t *>(grec_all + 2 * kGroups);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + kBars);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t limit = rp.timeout_ns;
    // this warp's group and what belongs to it
    // (two: groups 0 and 1 work, and the storing warps of 2 and 3 take every other
    // problem of 0 and 1, out of accumulators of their own)
    static_assert(GROUPS == kGroups || GROUPS == kGroups / 2, "groups at work");
    constexpr bool two = GROUPS < kGroups;
    const int g = warp < kIssue ? (warp >> 2) & (GROUPS - 1) : warp < kCopy ? warp - kIssue : (warp - kCopy) >> 1;
    Rec *recs = recs_all + g * kRecs, *grec = grec_all + 2 * g;
    uint64_t *full = bars + g * (2 * kRecs + 5);
    uint64_t *empty = full + kRecs;
    uint64_t *accf = empty + kRecs; // accumulator b: its product is finished (and its record there)
    uint64_t *acce = accf + 2;      // ... has been read out
    uint64_t *fin = acce + 2;       // every MMA of the group has completed
    if (warp >= kIssue && warp < kCopy)
    {
        if (lane < kRecs)
        {
            tc::mbar_init(&full[lane], 65);
            tc::mbar_init(&empty[lane], 1);
        }
        if (lane < 2)
        {
            tc::mbar_init(&accf[lane], 2);
            tc::mbar_init(&acce[lane], 4);
        }
        if (lane == 0)
            tc::mbar_init(fin, 1);
        tc::fence_mbar_init();
    }
    else if (warp == 1)
    {
        tc::tmem_alloc(tmem_slot, 128 * kGroups);
        tc::tmem_relinquish();
    }
    wait_for_previous();
    // the group's chunks: a plan's list, or every so many-th problem of the batch
    const int worker = g * gridDim.x + blockIdx.x, workers = gridDim.x * GROUPS;
    int64_t first = 0;
    int n = 0;
    if (rp.chunks && (!two || g < GROUPS))
    {
        first = p.cta_begin[worker];
        n = p.cta_begin[worker + 1] - (int)first;
    }
    else if (!two || g < GROUPS)
    {
        first = worker;
        n = worker < rp.u.batch ? (int)((rp.u.batch - worker + workers - 1) / workers) * rp.u.nk : 0;
    }
    if (warp >= kCopy)
        copy_chunks(rp, tc::smem_u32(smem) + kFront + g * (kBytes * kGroups / GROUPS), recs, full, empty, first, n, workers, (warp - kCopy) & 1,
                    lane);
    else if (warp >= kIssue)
    {
        tc::tc_fence_before();
        __syncthreads(); // barriers initialised, tensor memory there
        tc::tc_fence_after();
        if (lane == 0)
        {
            const uint32_t acc = *tmem_slot + g * 128, apart = two ? 256 : 64;
            int turn = 0;        // problems so far
            bool wide = false;   // the current or last one takes all columns
            uint32_t idesc = 0, d = 0, more = 0, up = 0;
            for (int j = 0; j < n; ++j)
            {
                const int s = j % kRecs, b = turn & 1;
                if (!tc::mbar_wait_bounded(&full[s], (j / kRecs) & 1, limit))
                {
                    ring_flag(2);
                    break;
                }
                const Rec r = recs[s];
                const int M = r.shape & 255, N = (r.shape >> 8) & 255, K = (r.shape >> 16) & 255;
                if (r.shape & kFirst)
                {
                    // the accumulator's last product (and, where one of the two
                    // takes all columns, the problem before) has been read out
                    const bool now = N > 64 && !two;
                    if ((turn >= 2 && !tc::mbar_wait_bounded(&acce[b], ((turn >> 1) - 1) & 1, limit)) ||
                        (turn >= 1 && (now || wide) &&
                         !tc::mbar_wait_bounded(&acce[b ^ 1], ((turn - 1) >> 1) & 1, limit)))
                    {
                        ring_flag(3);
                        break;
                    }
                    wide = now;
                    // the warp of row 0: any, every other, 0 or 1, or 0
                    const int quad = (turn + g) & (M <= 32 ? 3 : M <= 64 ? 2 : M <= 96 ? 1 : 0);
                    up = (uint32_t)quad * 32 * 128;
                    Rec c = r;
                    c.quad = quad;
                    grec[b] = c;
                    idesc = tc::idesc_f16(BF16, 128, (N + 15) & ~15);
                    d = acc + (now ? 0 : apart * b);
                    more = 0;
                }
                // the copies are generic-proxy writes: order them before the
                // tensor core's (async-proxy) reads
                tc::fence_proxy_async_smem();
                tc::tc_fence_after();
                for (int it = 0; it < p.num_iter; ++it)
                {
                    uint64_t da = tc::desc_kmajor_sw128(r.sa - up), db = tc::desc_kmajor_sw128(r.sb);
                    for (int ks = K; ks > 0; ks -= 16)
                    {
                        tc::mma_f16_ss(d, da, db, idesc, more);
                        more = 1;
                        da += 2; // 32 bytes
                        db += 2;
                    }
                }
                tc::mma_commit(&empty[s]);
                if (r.shape & kLast)
                {
                    tc::mma_commit(&accf[b]);
                    tc::mbar_arrive(&accf[b]); // the record
                    ++turn;
                }
            }
            tc::mma_commit(fin);
            if (!tc::mbar_wait_bounded(fin, 0, limit))
                ring_flag(4);
        }
        __syncwarp();
    }
    else
    {
        tc::tc_fence_before();
        __syncthreads();
        tc::tc_fence_after();
        const int q = warp & 3;
        const bool plain = rp.out.plain;
        const int own = rp.chunks ? p.cta_begin[workers + 1 + worker] : n / rp.u.nk; // problems
        for (int turn = two ? warp >> 3 : 0; turn < own; turn += two ? 2 : 1)
        {
            const int b = turn & 1;
            // (tcgen05.ld is .sync.aligned: the outcome must be warp-uniform)
            if (!__all_sync(0xffffffffu, tc::mbar_wait_bounded(&accf[b], (turn >> 1) & 1, limit)))
            {
                if (lane == 0)
                    ring_flag(5);
                break;
            }
            tc::tc_fence_after();
            const Rec r = grec[b];
            const int M = r.shape & 255, N = (r.shape >> 8) & 255;
            const uint32_t acc = *tmem_slot + g * 128 + (two ? 256 * b : N > 64 ? 0 : 64 * b);
            const int base = 32 * (q - r.quad); // the row in this warp's first lane
            const bool fast = plain && !((r.ldc | (int)r.c_off | N) & 7) && !(reinterpret_cast<uintptr_t>(p.C) & 31);
            const uint32_t lanes = acc + ((uint32_t)(32 * q) << 16);
            if (base >= 0 && fast)
            {
                int64_t off = r.c_off + (int64_t)(base + lane) * r.ldc;
                for (int c0 = 0; base < M && c0 < N; c0 += 32, off += 32)
                {
                    uint32_t v[32];
                    tmem_ld32(lanes + c0, v);
                    if (base + lane < M)
                        store_row(p, off, N - c0, v);
                }
            }
            else if (base >= 0 && base < M)
                store_general(rp.out, lanes, r.c_off + (int64_t)base * r.ldc, r.ldc, M - base, N);
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0)
                tc::mbar_arrive(&acce[b]);
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 1)
    {
        tc::tc_fence_after();
        tc::tmem_dealloc(*tmem_slot, 128 * kGroups);
    }
}

const void *ring_fn(bool bf16, bool two)
{
    if (two)
        return bf16 ? (const void *)&h16_ring_kernel<true, kGroups / 2> : (const void *)&h16_ring_kernel<false, kGroups / 2>;
    return bf16 ? (const void *)&h16_ring_kernel<true, kGroups> : (const void *)&h16_ring_kernel<false, kGroups>;
}

int launch_ring(RingParams &rp, bool bf16, int groups, int ctas, cudaStream_t s)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev >= 64)
        return e != cudaSuccess ? cuda_fail(e, "cudaGetDevice") : KAMI_ERR_UNSUPPORTED;
    static std::once_flag once[64][4];
    static cudaError_t attr[64][4];
    const bool two = groups < kGroups;
    const void *fn = ring_fn(bf16, two);
    const int v = bf16 + 2 * two;
    std::call_once(once[dev][v], [&] {
        attr[dev][v] = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    });
    if (attr[dev][v] != cudaSuccess)
        return cuda_fail(attr[dev][v], "cudaFuncSetAttribute(h16_ring_kernel)");
    rp.out = Out{rp.p.C, rp.p.out_type, rp.p.alpha == 1.0 && rp.p.beta == 0.0, rp.p.beta != 0.0, (float)rp.p.alpha,
                 (float)rp.p.beta};
    void *args[] = {&rp};
    e = launch_overlapped(fn, dim3(ctas), dim3(kThreads), args, kSmem, s);
    if (e != cudaSuccess)
        return cuda_fail(e, "cudaLaunchKernel(h16_ring_kernel)");
    return KAMI_OK;
}

} // namespace

int h16_ring_smem() { return kSmem; }
// Groups at work in a plan's CTAs.  A group's 46 KB hold one chunk of a large
// problem, which its MMAs have to be done with before the next is copied: where
// problems of more than half a ring carry most of the bytes, two groups of 92 KB
// (us, four groups / two: 2000 of 128^3 55 / 52, 4000 with FP16 out 80 / 71, 2000 of
// 96^3 34 / 28, 1000 of 112 .. 128 25 / 23; the other way at times, 4000 of 112 .. 128
// 84 / 90).  All sixteen storing warps stay at work: half of them, 1000 of 128^3
// with alpha and beta took 62 us instead of 45.  (A kernel of its own: the same
// choice at run time cost 20000 of 32^3 9 %.)
int h16_ring_groups(int count, const int *M, const int *N)
{
    int64_t all = 0, large = 0;
    for (int i = 0; i < count; ++i)
    {
        const int bytes = (up8(M[i]) + up8(N[i])) * 128;
        all += bytes;
        large += 2 * bytes > kBytes ? bytes : 0;
    }
    return 2 * large > all ? kGroups / 2 : kGroups;
}

// The problems of a plan's lists, one per group (list l: group l / CTAs of CTA
// l % CTAs, so that few problems spread over the CTAs first), as chunks
// placed in the groups' rings.  begin: the lists' first chunks, then (from
// lists + 1 on) their numbers of problems.
void h16_ring_schedule(const std::vector<std::vector<int>> &lists, const int *M, const int *N, const int *K,
                       const int64_t *ao, const int64_t *bo, const int64_t *co, std::vector<char> *out,
                       std::vector<int> *begin, int groups)
{
    size_t count = 0, total = 0;
    for (const auto &l : lists)
        for (int i : l)
            total += (K[i] + 63) / 64;
    out->resize(total * sizeof(ChunkDesc));
    begin->assign(2 * lists.size() + 1, 0);
    ChunkDesc *d = reinterpret_cast<ChunkDesc *>(out->data());
    ring::Placer placer(kBytes * kGroups / groups, kRecs);
    for (size_t c = 0; c < lists.size(); ++c)
    {
        (*begin)[c] = (int)count;
        (*begin)[lists.size() + 1 + c] = (int)lists[c].size();
        placer.clear();
        for (int i : lists[c])
            for (int k0 = 0; k0 < K[i]; k0 += 64)
            {
                ChunkDesc x{};
                int land;
                x.a_off = ao[i] + k0;
                x.b_off = bo[i] + k0;
                x.c_off = co[i];
                x.shape = (uint32_t)(M[i] | N[i] << 8 | std::min(64, K[i] - k0) << 16) | (k0 == 0 ? kFirst : 0u) |
                          (k0 + 64 >= K[i] ? kLast : 0u);
                x.at = placer.place((up8(M[i]) + up8(N[i])) * 128, &x.dep, &land);
                x.lda = K[i];
                x.ldb = K[i];
                x.ldc = N[i];
                d[count++] = x;
            }
    }
    (*begin)[lists.size()] = (int)count;
}

// a plan: descriptors (h16_ring_schedule) on the device, p.cta_begin their lists
int h16_ring_plan_launch(const GroupedParams &p, const void *chunks, bool bf16, int ctas, int groups, cudaStream_t s)
{
    RingParams rp{};
    rp.p = p;
    rp.chunks = reinterpret_cast<const ChunkDesc *>(chunks);
    rp.timeout_ns = (uint64_t)(2e9 + (double)p.num_iter * 1e6); // generous: a problem takes microseconds
    return launch_ring(rp, bf16, groups, ctas, s);
}

// CTAs of a uniform batch: one per SM, four problems side by side in each
static int uniform_ctas(int64_t batch)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (int)std::min<int64_t>(batch, sms);
}

// A uniform batch, A row-major and B N x K, M, N, K <= 128, K a multiple of 8,
// 16-byte aligned rows and problems (checked by the callers).
int h16_ring_launch(const GemmArgs &g, int in_type, cudaStream_t s)
{
    if (g.lda > 0x3fffffff || g.ldb > 0x3fffffff || g.ldc > 0x7fffffff)
        return fail(KAMI_ERR_UNSUPPORTED, "no kernel for M=%d N=%d K=%d with rows %lld, %lld, %lld apart", g.M, g.N, g.K,
                    (long long)g.lda, (long long)g.ldb, (long long)g.ldc);
    RingParams rp{};
    rp.p.A = g.A;
    rp.p.B = g.B;
    rp.p.C = g.C;
    rp.p.out_type = g.out_type;
    rp.p.alpha = g.alpha;
    rp.p.beta = g.beta;
    rp.p.num_iter = g.num_iter;
    Uniform &u = rp.u;
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
    u.nk = (g.K + 63) / 64;
    u.bytes = (up8(g.M) + up8(g.N)) * 128;
    u.slots = std::min(kRecs, kBytes / u.bytes);
    rp.timeout_ns = (uint64_t)(2e9 + (double)g.num_iter * 1e6);
    return launch_ring(rp, in_type == KAMI_BF16, kGroups, uniform_ctas(g.batch), s);
}

// the launch of h16_ring_launch (kami_gemm_describe)
void h16_ring_info(const GemmArgs &g, LaunchInfo *info)
{
    const int ctas = uniform_ctas(g.batch);
    *info = LaunchInfo{KAMI_VARIANT_TCGEN05, KAMI_PARTITION_1D, 1, kThreads, kSmem,
                       ctas ? (int)((g.batch + ctas - 1) / ctas) : 0, ctas};
}

int h16_ring_read_error(int *flag)
{
    int v = 0, z = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_h16r_error, sizeof(int));
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbol(g_h16r_error, &z, sizeof(int));
    if (e != cudaSuccess)
        return cuda_fail(e, "reading the 16-bit ring kernel's status");
    *flag = v;
    return KAMI_OK;
}

} // namespace kami
