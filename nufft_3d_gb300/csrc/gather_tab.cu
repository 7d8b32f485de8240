// Gather (fNUFT's H product, spmv of nufft_3d.m:259-271) from a stored H, for
// every coil width.
//
// The reference keeps H as a sparse matrix (nufft_3d.m:153-212) and multiplies
// by it.  The stored form here is blocked: two neighbouring samples share a
// row, the union of their supports, whose entries are (two weights, one grid
// point), so that one shared-memory read of a grid point (8 coils, 64 bytes)
// serves two samples.  On the 128^3 koosh ball (256 x 32768 samples) a row has
// 137 entries against 2 x 113 taps: 6.08 GB of table, against 7.87 GB for a
// row per sample.  (Rows of four samples, 43 entries a sample against 69, took
// 6.78 GB and the same time: their 64 accumulators a lane leave 15 warps, and
// on sparse trajectories their unions are much larger: uniform samples at one
// eighth of a sample a grid point take 1182 bytes a sample in fours, 849 in
// pairs, 678 singly.)
//
// Samples are sorted by tile column (tiles of 8 x 8 x 8 oversampled-grid
// points, or 32 x 32 in 2-D, z fastest), inside a tile by slab (two z cells)
// and inside a slab along a Hilbert curve, so that consecutive samples are
// close and a slab needs 2 + 2R planes of the padded tile.  A record is a run
// of at most kRecRows rows of one slab, sorted by length.
//
// The kernel is persistent and asynchronous: a producer warp streams the grid
// planes of the records through a shared-memory ring (a slab that follows its
// neighbour in z loads two new planes, not the whole padded tile: 175 KB a
// tile of 490 samples before, 45 KB now), consumer warps take tasks of four
// rows, eight lanes a row; lane l applies entries l, l + 8, ... of its row to
// all coils, and the 8 partial sums are reduced at the row's end.  A helper
// warp publishes the tasks whose planes have landed, in record order (a record
// shares planes with those before it), and asks L2 for the entries ahead.  No
// barrier spans the block after set-up.
//
// Measured at 128^3 x 8 coils: 1.78 ms (one 1024-thread block a tile piece with
// a barrier on either side, one row a sample: 3.53 ms).  The L1 data path bounds
// it, 72 % of its peak in a capture at 96^3: 24 shared wavefronts a step of 32
// entries, 16 of them the points themselves.  192^3 x 16 coils: 11.0 ms (21.2 ms).
//
// Table layout: row r holds chunks [grow[r], grow[r+1]) of 16 entries; lane l
// of the row reads entries l and l + 8 of a chunk as one float4 of gw[8 c + l]
// and one pair of points of gi[8 c + l] (plane * plane stride + y * P0 + x,
// planes counted from the slab's first).  Bank conflicts and selects are
// avoided by fixed rotations:
//   * lane l reads the 16-byte coil pairs of a point in the order
//     (l mod NP) ^ k, so the 8 lanes of a row touch all four 16-byte columns
//     in every load, two lanes each; eight entries hold even points in 0-3 and
//     odd ones in 4-7 while they can, so the two differ in their half of the
//     banks (5 % of the wavefronts conflict);
//   * entries 4-7 store the weights of samples 1, 0, so the first reduction
//     step (lanes l and l ^ 4) keeps accumulator 0 in every lane;
//   * the pair rotation makes the next steps keep accumulators by their own
//     register number too: the reduction has no selects.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

#include <cub/device/device_scan.cuh>

#include "async.h"
#include "internal.h"
#include "taps.h"
#include "waits.h"

namespace nufft3d {

constexpr int kRow = 2;          // samples of a row
constexpr int kChunk = 16;       // entries of a chunk: two for each of a row's 8 lanes
constexpr int kRecRows = 64;     // rows of a record
constexpr int kRingPlanes = 24;  // most planes of the ring
constexpr int kStages = 8;       // records in flight
constexpr int kRowsAhead = 256;  // rows in flight

// Warps, blocks per SM and chunks of a row each lane keeps in flight.  With 8
// coils the ring takes the whole shared memory, and 16 warps of 128 registers
// measured faster (1.88 ms at 128^3 then) than 20 of 96 (2.15 ms) or 24 of 80, which
// spill: the ring leaves the L1 cache too small for spills.  Fewer coils leave
// room for more blocks, which hide the latency of short records.
template <int CB>
struct GatherCfg;
template <> struct GatherCfg<8> { static constexpr int WARPS = 16, MINB = 1, DEPTH = 3; };
template <> struct GatherCfg<4> { static constexpr int WARPS = 10, MINB = 2, DEPTH = 3; };
template <> struct GatherCfg<2> { static constexpr int WARPS = 8, MINB = 4, DEPTH = 2; };
template <> struct GatherCfg<1> { static constexpr int WARPS = 8, MINB = 4, DEPTH = 2; };
// (3, 5 and 7 coils: the whole of an odd coil count, points of 24, 40 or 56 bytes)
template <> struct GatherCfg<3> { static constexpr int WARPS = 10, MINB = 2, DEPTH = 2; };
template <> struct GatherCfg<5> { static constexpr int WARPS = 10, MINB = 2, DEPTH = 2; };
template <> struct GatherCfg<7> { static constexpr int WARPS = 20, MINB = 1, DEPTH = 2; };
// one warp asks L2 for the entries of the records as they are issued (narrow
// passes are bound by the bandwidth and do without)
template <int CB>
constexpr bool kPrefetch = CB >= 3;

// A point is read in 16-byte units of two coils, or in single coils where
// their number is odd.
template <int CB>
constexpr bool kPaired = CB % 2 == 0;
template <int CB>
constexpr int kUnits = kPaired<CB> ? CB / 2 : CB;

struct GatherArgs {
    const float2 *G;
    float2 *ks;
    int nc, c0, cb;
    int pairs;    // coil pairs are 16-byte aligned in G and ks
    float scale;
    const float *wsample;
    const GatherRec *recs;
    const int2 *chunks;  // record ranges
    int nchunks;
    int merge;           // ranges taken as one
    const uint32_t *grow;
    const float4 *gw;    // [chunk][8]: weights of entries l (x, y) and l + 8 (z, w)
    const uint32_t *gi;  // [chunk][8]: their points, l in the low half
    int K[3];
    int P0, P1;   // plane of the padded tile
    int PS;       // plane stride in points
    int npl;      // planes of a slab
    int S;        // planes of the ring
    unsigned rbytes;  // its bytes
    int rcpP0;    // 2^16 / P0 + 1: divides plane points by P0
    int small;    // the padded tile is wider than the grid on some axis
    int use_tma;
    int *work;    // [2]: next chunk, blocks done
    InterpStatus st;
};

constexpr int kTaskRows = 4;                              // rows of a task
constexpr int kTasks = kStages * kRecRows / kTaskRows;    // task descriptors (a ring)

// A task as the consumers see it.
struct GatherTask {
    int s0, ns;         // first sample, samples
    unsigned base;      // ring byte of the slab's first plane
    int stage;          // record stage
    uint32_t c[kTaskRows + 1];  // first chunk of each row (equal past the record's end)
    uint32_t pad[3];
};

__device__ __forceinline__ int ring_wrap(int x, int K)
{
    x %= K;
    return x < 0 ? x + K : x;
}

// The same for positions at most one period outside the grid.
__device__ __forceinline__ int near_wrap(int x, int K) { return x < 0 ? x + K : x >= K ? x - K : x; }

// Grid offsets of the points of a plane of the padded tile at (ox, oy) that
// thread t of nt copies below in PER parts each, in points; once per tile column
// (a producer warp reads only what it wrote: the warps may be at different
// columns).
template <int PER>
__device__ __forceinline__ void plane_offsets(const GatherArgs &a, uint32_t *poff, int ox, int oy, int t, int nt)
{
    for (int q = t; q < a.P0 * a.P1 * PER; q += nt) {
        const int pt = q / PER;
        const int y = (int)(((unsigned)pt * (unsigned)a.rcpP0) >> 16), x = pt - y * a.P0;
        int gx = ox + x, gy = oy + y;
        if (a.small) {  // the padded tile is wider than the grid
            gx = ring_wrap(gx, a.K[0]);
            gy = ring_wrap(gy, a.K[1]);
        } else {
            gx = near_wrap(gx, a.K[0]);
            gy = near_wrap(gy, a.K[1]);
        }
        poff[pt] = (uint32_t)(gy * a.K[0] + gx);
    }
}

// z plane of the grid
__device__ __forceinline__ size_t grid_plane(const GatherArgs &a, int z)
{
    return (size_t)(a.small ? ring_wrap(z, a.K[2]) : near_wrap(z, a.K[2])) * a.K[1] * a.K[0];
}

// Planes [z0, z0 + n) of a padded tile at (ox, oy) that wraps around the grid
// edge, into ring slots slot, slot + 1, ...  Where the pass takes every coil, a
// row of points is one contiguous run, or two: bulk copies that the lanes of one
// warp issue.  (Runs start at even points and have an even number, whole 16-byte
// units: K1 and P0 are even and so is ox, see tile_shift.)
template <int CB>
__device__ __forceinline__ void load_rows(const GatherArgs &a, unsigned ring, unsigned pbytes, int slot, int ox, int oy,
                                          int z0, int n, int lane, unsigned bar)
{
    constexpr unsigned SLOT = CB * 8;
    if (lane == 0) mbar_expect_bytes(bar, (unsigned)n * (unsigned)(a.P0 * a.P1) * SLOT);
    __syncwarp();
    const int x0 = near_wrap(ox, a.K[0]), n0 = min(a.P0, a.K[0] - x0);
    for (int q = lane; q < n * a.P1; q += 32) {
        const int t = q / a.P1, y = q - t * a.P1;
        const int sl = slot + t < a.S ? slot + t : slot + t - a.S;
        const float2 *row = a.G + (grid_plane(a, z0 + t) + (size_t)near_wrap(oy + y, a.K[1]) * a.K[0]) * CB;
        const unsigned dst = ring + (unsigned)sl * pbytes + (unsigned)(y * a.P0) * SLOT;
        bulk_load(dst, row + (size_t)x0 * CB, (unsigned)n0 * SLOT, bar);
        if (n0 < a.P0) bulk_load(dst + (unsigned)n0 * SLOT, row, (unsigned)(a.P0 - n0) * SLOT, bar);
    }
}

// The others are copied by the producer warps: 16-byte asynchronous copies of
// coil pairs ...
template <int CB>
__device__ __forceinline__ void copy_pairs(const GatherArgs &a, const uint32_t *poff, unsigned ring, unsigned pbytes,
                                           int slot, int z0, int n, int t, int nt)
{
    constexpr int PER = kUnits<CB>;
    for (int p = 0; p < n; ++p) {
        const float2 *plane = a.G + grid_plane(a, z0 + p) * a.nc + a.c0;
        const unsigned dst = ring + (unsigned)slot * pbytes;
#pragma unroll 4
        for (int q = t; q < a.P0 * a.P1 * PER; q += nt) {
            const int pt = q / PER, c = q % PER;
            if (2 * c < a.cb) copy_async16(dst + (unsigned)q * 16, plane + (size_t)poff[pt] * a.nc + 2 * c);
        }
        if (++slot == a.S) slot = 0;
    }
}

// ... and coil counts whose points are not whole 16-byte units coil by coil,
// through registers, several loads in flight (8-byte asynchronous copies took
// three times as long).  A warp takes whole points, 32 at a time, so that it
// reads only the offsets that it wrote, whatever the coil count (5 coils on
// 88 x 112 x 100: forward 747 us, indices found by division a coil 857 us).
template <int CB, int NPW>
__device__ __forceinline__ void copy_coils(const GatherArgs &a, const uint32_t *poff, unsigned char *ring,
                                           unsigned pbytes, int slot, int z0, int n, int pw, int lane)
{
    constexpr int M = CB >= 7 ? 2 : CB == 5 ? 3 : CB == 3 ? 5 : CB == 1 ? 8 : 4;  // groups of 32 points in flight
    const int npt = a.P0 * a.P1;
    const int per = (npt + 32 * NPW - 1) / (32 * NPW);  // groups of a warp in a plane
    int i = 0, p = 0;
    size_t plane = grid_plane(a, z0);
    while (p < n) {
        float2 v[M * CB];
        unsigned d[M * CB];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int pt0 = (pw + NPW * i) * 32;
#pragma unroll
            for (int j = 0; j < CB; ++j) {
                const int e = j * 32 + lane, pt = pt0 + e / CB, c = e % CB;
                d[m * CB + j] = 0xffffffffu;
                if (p < n && pt < npt && c < a.cb) {
                    v[m * CB + j] = __ldcg(a.G + (plane + poff[pt]) * a.nc + a.c0 + c);
                    d[m * CB + j] = (unsigned)slot * pbytes + 8u * (unsigned)(pt0 * CB + e);
                }
            }
            if (++i == per) {
                i = 0;
                ++p;
                if (++slot == a.S) slot = 0;
                plane = grid_plane(a, z0 + p);
            }
        }
#pragma unroll
        for (int u = 0; u < M * CB; ++u)
            if (d[u] != 0xffffffffu) *reinterpret_cast<float2 *>(ring + d[u]) = v[u];
    }
}

// ROWS: a pass of every coil, see load_rows; else NPW producer warps copy the
// tiles that wrap.
template <int CB, int NPW, bool ROWS>
__global__ void __launch_bounds__(GatherCfg<CB>::WARPS * 32, GatherCfg<CB>::MINB)
k_gather_rows(const __grid_constant__ GatherArgs a, const __grid_constant__ CUtensorMap tmap)
{
    constexpr int NW = GatherCfg<CB>::WARPS - NPW - 1, DEPTH = GatherCfg<CB>::DEPTH;
    constexpr int NP = kUnits<CB>;
    constexpr int SLOT = CB * 8;
    extern __shared__ __align__(128) unsigned char gsm[];
    __shared__ unsigned long long bars[kStages];
    __shared__ __align__(16) GatherTask tasks[kTasks];
    // planes loaded up to and with a record, rows issued before it, the count
    // of finished tasks of its stage at which it is done (per producer warp)
    __shared__ int sends[NPW][kStages], srows[NPW][kStages], stasks[NPW][kStages];
    __shared__ int finished[kStages];  // tasks finished so far, by stage
    __shared__ int ctl[4];             // tasks whose planes have landed, tasks claimed, tasks in all, abort
    __shared__ uint2 ahead_of[kStages];  // chunk range of a record, for the prefetch
    __shared__ int tend[kStages];        // tasks up to and with a record
    __shared__ int nrec[2];            // records issued, records in all
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned ring = (unsigned)__cvta_generic_to_shared(gsm);
    const unsigned full = (unsigned)__cvta_generic_to_shared(bars);
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(full + 8 * i, 32 * NPW);
            finished[i] = 0;
        }
        ctl[0] = ctl[1] = ctl[3] = 0;
        ctl[2] = 0x7fffffff;
        nrec[0] = 0;
        nrec[1] = 0x7fffffff;
    }
    __syncthreads();
    const unsigned pbytes = (unsigned)a.PS * SLOT;
    // A wait that runs out is reported and ends the block's work.  A warp takes
    // that decision as one, by vote: a lane that left alone would leave the
    // others at the next warp-wide instruction.  (Lane 0 alone at the polls, the
    // others waiting for what it tells them, took longer: 2 to 15 % of a small
    // volume's gather.)
    volatile int *const ab = &ctl[3];
    auto give_up = [&]() {
        if (lane == 0) {
            if (a.st.err) atomicOr(a.st.err, 1);
            *ab = 1;
        }
    };
    auto ended = [&]() { return __any_sync(0xffffffffu, *ab != 0) != 0; };
    // records issued by the first producer warp, once it has stopped (-1: it has not)
    auto records = [&]() {
        for (int i = 0; i < kDrainPolls; ++i) {
            const int n = __reduce_min_sync(0xffffffffu, ld_acquire(&nrec[1]));
            if (n != 0x7fffffff) return n;
            __nanosleep(50);
        }
        return -1;
    };

    if (warp >= NW + NPW) {
        // ---------------------------------------------------------- helper
        // Publishes the tasks of each record once its planes and those of the
        // records before it (it shares planes with them) have landed.
        int ahead = 0, landed = 0;
        BoundedWait copy, idle;
        for (;;) {
            const int n = __reduce_min_sync(0xffffffffu, ld_acquire(&nrec[0]));
            if (ahead < n) {
                if (kPrefetch<CB> && n - ahead < kStages) {  // (else the slot may be in new use)
                    const uint2 q = ahead_of[ahead % kStages];
                    const char *w = reinterpret_cast<const char *>(a.gw + (size_t)q.x * 8);
                    for (unsigned o = 128u * lane; o < 128u * q.y; o += 128u * 32) prefetch_line(w + o);
                    const char *x = reinterpret_cast<const char *>(a.gi + (size_t)q.x * 8);
                    for (unsigned o = 128u * lane; o < 32u * q.y; o += 128u * 32) prefetch_line(x + o);
                }
                ++ahead;
                idle = BoundedWait();
                continue;
            }
            if (landed < n) {
                const int st = landed % kStages;
                const WaitTurn turn = wait_turn(copy, a.st.polls, kDrainPolls);
                // expired: reported, and waited for all the same
                if (turn == kWaitReport && lane == 0 && a.st.err) atomicOr(a.st.err, 1);
                if (turn == kWaitGiveUp) {
                    give_up();
                } else if (__all_sync(0xffffffffu, mbar_try_wait(full + 8 * st, (unsigned)(landed / kStages) & 1u))) {
                    if (lane == 0) st_release(&ctl[0], tend[st]);
                    ++landed;
                    copy = BoundedWait();
                    continue;
                } else {
                    ++copy.failed;
                }
            } else if (__all_sync(0xffffffffu, ld_acquire(&nrec[1]) <= landed)) {
                break;
            } else {
                if (wait_turn(idle, kDrainPolls, kDrainPolls) == kWaitGiveUp) give_up();
                ++idle.failed;
                __nanosleep(50);
            }
            if (ended()) break;
        }
        if (ended()) {
            // the block must not leave while planes are on their way to its memory
            const int n = records();
            for (; landed < n; ++landed)
                for (int i = 0; i < kDrainPolls; ++i)
                    if (__all_sync(0xffffffffu, mbar_try_wait(full + 8 * (landed % kStages),
                                                              (unsigned)(landed / kStages) & 1u)))
                        break;
        }
    } else if (warp >= NW) {
        // ------------------------------------------------------ producers
        const int pw = warp - NW;
        volatile int *const send = sends[pw], *const srow = srows[pw], *const stask = stasks[pw];
        if (lane == 0)
            for (int i = 0; i < kStages; ++i) stask[i] = 0;
        __syncwarp();
        int rr = 0, d = 0, endp = 0, rows = 0, ntasks = 0;  // records issued, oldest unfinished, planes, rows, tasks
        // ranges of records: claimed from the work counter (a single producer
        // warp) or in turn (several, which agree without talking)
        int turn = 0;
        auto claim = [&]() -> int {
            if (NPW > 1) return (int)blockIdx.x + (int)gridDim.x * turn++;
            const int b = lane == 0 ? atomicAdd(a.work, 1) : 0;
            return __shfl_sync(0xffffffffu, b, 0);
        };
        auto range = [&](int b) {
            const int lo = b * a.merge;
            if (lo >= a.nchunks) return make_int2(0, 0);
            return make_int2(__ldg(&a.chunks[lo]).x, __ldg(&a.chunks[min(lo + a.merge, a.nchunks) - 1]).y);
        };
        // Records are read 32 at a time, one a lane, a batch ahead: a global load
        // takes longer than a record does.
        int2 cur = make_int2(0, 0);       // the rest of the range that the batches come from
        GatherRec mine, coming;           // this lane's record of the current and the next batch
        int n_mine = 0, n_coming = 0, i_mine = 0;
        bool fresh = false, fresh_coming = false;  // the batch starts a range
        auto fetch = [&]() {
            fresh_coming = false;
            if (cur.x >= cur.y) {
                cur = range(claim());
                fresh_coming = true;
            }
            n_coming = min(32, cur.y - cur.x);
            if (lane < n_coming) coming = a.recs[cur.x + lane];
            cur.x += n_coming;
        };
        fetch();
        bool live = true, copied = false;
        int slot = 0;  // the ring slot of the next plane
        int col_x = INT_MIN, col_y = INT_MIN;  // the column of the plane offsets
        uint32_t *const poff = reinterpret_cast<uint32_t *>(gsm + a.rbytes);
        for (;;) {
            if (i_mine == n_mine) {
                mine = coming;
                n_mine = n_coming;
                fresh = fresh_coming;
                i_mine = 0;
                if (n_mine <= 0) break;
                fetch();
            }
            GatherRec rec;
            rec.ox = __shfl_sync(0xffffffffu, mine.ox, i_mine);
            rec.oy = __shfl_sync(0xffffffffu, mine.oy, i_mine);
            rec.oz = __shfl_sync(0xffffffffu, mine.oz, i_mine);
            rec.nload = __shfl_sync(0xffffffffu, mine.nload, i_mine);
            rec.row0 = __shfl_sync(0xffffffffu, mine.row0, i_mine);
            rec.nrows = __shfl_sync(0xffffffffu, mine.nrows, i_mine);
            rec.s0 = __shfl_sync(0xffffffffu, mine.s0, i_mine);
            rec.ns = __shfl_sync(0xffffffffu, mine.ns, i_mine);
            rec.chunk0 = __shfl_sync(0xffffffffu, mine.chunk0, i_mine);
            rec.nchunk = __shfl_sync(0xffffffffu, mine.nchunk, i_mine);
            if (fresh && i_mine == 0) rec.nload = a.npl;  // a range starts with all its planes
            ++i_mine;
            // wait for the stage and for the ring slots (the oldest unfinished
            // record d still reads planes from send[d] - npl on); at most
            // kRowsAhead rows are ahead, so that their prefetched entries stay in L2
            const int nt = (rec.nrows + kTaskRows - 1) / kTaskRows;
            uint32_t gr[kRecRows / 32 + 1];  // the rows' first chunks
            if (pw == 0) {
#pragma unroll
                for (int i = 0; i < kRecRows / 32 + 1; ++i) {
                    const int r = lane + 32 * i;
                    if (r <= kTaskRows * nt) gr[i] = __ldg(a.grow + rec.row0 + min(r, rec.nrows));
                }
            }
            rows += rec.nrows;
            while (d < rr && (rr - d >= kStages || send[d % kStages] - a.npl < endp + rec.nload - a.S ||
                              rows - srow[d % kStages] > kRowsAhead)) {
                const int want = stask[d % kStages];
                bool ok = false;
                for (int t = 0; t < kDrainPolls; ++t) {
                    ok = __all_sync(0xffffffffu, ld_acquire(&finished[d % kStages]) - want >= 0) != 0;
                    if (ok || ended()) break;
                    __nanosleep(50);
                }
                if (!ok) {
                    give_up();
                    live = false;
                    break;
                }
                ++d;
            }
            if (!live) break;
            const int st = rr % kStages;
            const unsigned fb = full + 8 * st;
            const bool pairs = kPaired<CB> && a.pairs;
            bool async = false;  // planes by asynchronous copies
            if (rec.nload > 0) {
                const int z0 = rec.oz + a.npl - rec.nload;
                if (a.use_tma && rec.ox >= 0 && rec.oy >= 0 && rec.ox + a.P0 <= a.K[0] && rec.oy + a.P1 <= a.K[1]) {
                    if (pw == 0 && lane == 0) {
                        mbar_expect_bytes(fb, (unsigned)rec.nload * (unsigned)(a.P0 * a.P1) * SLOT);
                        // the slots may last have been written by ordinary copies (the
                        // fence waits for every copy in flight, so only then)
                        if (copied) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        int sl = slot;
                        for (int t = 0; t < rec.nload; ++t) {
                            const int z = a.small ? ring_wrap(z0 + t, a.K[2]) : near_wrap(z0 + t, a.K[2]);
                            const unsigned dst = ring + (unsigned)sl * pbytes;
                            if (kPaired<CB>) tma_load_4d(dst, &tmap, 2 * a.c0, rec.ox, rec.oy, z, fb);
                            else tma_load_3d(dst, &tmap, 2 * a.nc * rec.ox, rec.oy, z, fb);
                            if (++sl == a.S) sl = 0;
                        }
                    }
                    copied = false;
                } else if constexpr (ROWS) {
                    load_rows<CB>(a, ring, pbytes, slot, rec.ox, rec.oy, z0, rec.nload, lane, fb);
                } else {
                    copied = true;
                    async = pairs;
                    const int t = pw * 32 + lane;
                    if (rec.ox != col_x || rec.oy != col_y) {
                        col_x = rec.ox;
                        col_y = rec.oy;
                        __syncwarp();
                        if (pairs) plane_offsets<kUnits<CB>>(a, poff, col_x, col_y, t, 32 * NPW);
                        else plane_offsets<1>(a, poff, col_x, col_y, t, 32 * NPW);
                        __syncwarp();
                    }
                    if constexpr (kPaired<CB>) {
                        if (pairs) copy_pairs<CB>(a, poff, ring, pbytes, slot, z0, rec.nload, t, 32 * NPW);
                    }
                    if (!pairs) copy_coils<CB, NPW>(a, poff, gsm, pbytes, slot, z0, rec.nload, pw, lane);
                }
                endp += rec.nload;
                slot += rec.nload;
                if (slot >= a.S) slot -= a.S;
            }
            if (pw == 0) {
                // the tasks' descriptors
#pragma unroll
                for (int i = 0; i < kRecRows / 32 + 1; ++i) {
                    const int r = lane + 32 * i, q = r / kTaskRows, k = r % kTaskRows;
                    if (r > kTaskRows * nt) continue;
                    if (q < nt) tasks[(ntasks + q) % kTasks].c[k] = gr[i];
                    if (k == 0 && q > 0) tasks[(ntasks + q - 1) % kTasks].c[kTaskRows] = gr[i];
                }
                if (lane < nt) {
                    const int s = lane * kTaskRows * kRow, first = slot - a.npl;
                    *reinterpret_cast<int4 *>(&tasks[(ntasks + lane) % kTasks]) =
                        make_int4(rec.s0 + s, rec.ns - s, (first < 0 ? first + a.S : first) * (int)pbytes,
                                  st);
                }
            }
            if (lane == 0) {
                send[st] = endp;
                if (pw == 0) {
                    ahead_of[st] = make_uint2(rec.chunk0, rec.nchunk);
                    tend[st] = ntasks + nt;
                }
                srow[st] = rows - rec.nrows;
                stask[st] = stask[st] + nt;
            }
            __syncwarp();
            ntasks += nt;
            if (pw == 0 && lane == 0) st_release(&nrec[0], rr + 1);
            // (the bulk copies' bytes are expected beside the arrivals)
            if (async) mbar_arrive_on_copies(fb);
            else mbar_arrive(fb);
            ++rr;
        }
        if (pw == 0 && lane == 0) {  // no more tasks
            st_release(&ctl[2], ntasks);
            st_release(&nrec[1], rr);
        }
        // the helper waits for the planes of every record issued: without this
        // warp's arrivals it would not see them land
        if (!live && pw > 0)
            for (const int n = records(); rr < n; ++rr) mbar_arrive(full + 8 * (rr % kStages));
        // no exit before this thread's copies have landed
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ------------------------------------------------------ consumers
        const int ph = lane & 7, grp = lane >> 3;
        unsigned ko[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) ko[k] = kPaired<CB> ? 16u * (unsigned)((ph & (NP - 1)) ^ k) : 8u * k;
        // the warp's current task: sample that this lane will hold after the
        // reduction (or -1), ring byte of the slab, chunks of this lane's row,
        // its entries in flight
        int si = -1, stage = 0;
        unsigned base = 0;
        uint32_t n = 0;
        const float4 *wp = nullptr;
        const uint32_t *ip = nullptr;
        float4 wb[DEPTH];
        unsigned ib[DEPTH];
        int task = lane == 0 ? atomicAdd(&ctl[1], 1) : 0;
        // Starts the loads of the warp's next task; false at the end.
        auto next_task = [&]() -> bool {
            const int t = __shfl_sync(0xffffffffu, task, 0);
            if (lane == 0) task = atomicAdd(&ctl[1], 1);
            bool ok = false, end = false;
            for (int i = 0; i < kDrainPolls; ++i) {
                ok = __all_sync(0xffffffffu, ld_acquire(&ctl[0]) > t) != 0;
                if (ok) break;
                end = __any_sync(0xffffffffu, ld_acquire(&ctl[2]) <= t || *ab != 0) != 0;
                if (end) break;
                __nanosleep(50);
            }
            if (!ok) {
                if (!end) give_up();  // expired
                return false;
            }
            const GatherTask &f = tasks[t % kTasks];
            const int4 g = *reinterpret_cast<const int4 *>(&f);
            stage = g.w;
            const int sl = kRow * grp + (ph >> 2);
            si = sl < g.y ? g.x + sl : -1;
            base = (unsigned)g.z;
            const uint32_t c = f.c[grp];
            n = f.c[grp + 1] - c;
            wp = a.gw + (size_t)c * 8 + ph;
            ip = a.gi + (size_t)c * 8 + ph;
#pragma unroll
            for (int j = 0; j < DEPTH; ++j) {
                wb[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                ib[j] = 0;
                if ((uint32_t)j < n) {
                    wb[j] = ld_stream4(wp + 8 * j);
                    ib[j] = ld_stream32(ip + 8 * j);
                }
            }
            return true;
        };
        bool more = next_task();
        while (more) {
            float2 acc[kRow][CB];
#pragma unroll
            for (int s = 0; s < kRow; ++s)
#pragma unroll
                for (int k = 0; k < CB; ++k) acc[s][k] = make_float2(0.f, 0.f);
            const uint32_t nmax = __reduce_max_sync(0xffffffffu, n), nmin = __reduce_min_sync(0xffffffffu, n);
            auto apply1 = [&](float w0, float w1, unsigned idx) {
                unsigned off = base + idx * SLOT;
                off -= off >= a.rbytes ? a.rbytes : 0u;
                const float2 a0 = make_float2(w0, w0), a1 = make_float2(w1, w1);
                if constexpr (kPaired<CB>) {
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        const float4 v = *reinterpret_cast<const float4 *>(gsm + off + ko[k]);
                        acc[0][2 * k] = __ffma2_rn(a0, make_float2(v.x, v.y), acc[0][2 * k]);
                        acc[0][2 * k + 1] = __ffma2_rn(a0, make_float2(v.z, v.w), acc[0][2 * k + 1]);
                        acc[1][2 * k] = __ffma2_rn(a1, make_float2(v.x, v.y), acc[1][2 * k]);
                        acc[1][2 * k + 1] = __ffma2_rn(a1, make_float2(v.z, v.w), acc[1][2 * k + 1]);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        const float2 v = *reinterpret_cast<const float2 *>(gsm + off + 8 * k);
                        acc[0][k] = __ffma2_rn(a0, v, acc[0][k]);
                        acc[1][k] = __ffma2_rn(a1, v, acc[1][k]);
                    }
                }
            };
            auto apply = [&](const float4 w, unsigned idx) {
                apply1(w.x, w.y, idx & 0xFFFFu);
                apply1(w.z, w.w, idx >> 16);
            };
            uint32_t k0 = 0;
            for (; k0 + 2 * DEPTH <= nmin; k0 += DEPTH) {  // every row has its next entries
#pragma unroll
                for (int j = 0; j < DEPTH; ++j) {
                    const float4 w = wb[j];
                    const unsigned idx = ib[j];
                    wb[j] = ld_stream4(wp + 8 * (DEPTH + j));
                    ib[j] = ld_stream32(ip + 8 * (DEPTH + j));
                    apply(w, idx);
                }
                wp += 8 * DEPTH;
                ip += 8 * DEPTH;
            }
            for (; k0 < nmax; k0 += DEPTH) {  // rows end; ended ones apply weight 0
#pragma unroll
                for (int j = 0; j < DEPTH; ++j) {
                    const float4 w = wb[j];
                    const unsigned idx = ib[j];
                    wb[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                    ib[j] = 0;
                    if (k0 + j + DEPTH < n) {
                        wb[j] = ld_stream4(wp + 8 * (DEPTH + j));
                        ib[j] = ld_stream32(ip + 8 * (DEPTH + j));
                    }
                    if (k0 + j < nmax) apply(w, idx);
                }
                wp += 8 * DEPTH;
                ip += 8 * DEPTH;
            }
            const int so = si;
            __syncwarp();  // every lane has read its planes
            if (lane == 0) add_release(&finished[stage], 1);
            more = next_task();  // its first entries load while this task is reduced
            // reduce over the phases: each step keeps the accumulators of the same
            // register numbers in every lane (see the rotations above)
#pragma unroll
            for (int k = 0; k < CB; ++k) {  // sample 0 of 2
                acc[0][k].x += __shfl_xor_sync(0xffffffffu, acc[1][k].x, 4);
                acc[0][k].y += __shfl_xor_sync(0xffffffffu, acc[1][k].y, 4);
            }
            if constexpr (kPaired<CB>) {
                constexpr int X2 = 2 & (NP - 1), X1 = 1 & (NP - 1);
#pragma unroll
                for (int k = 0; k < NP; k += 1 + X1)  // every second unit (a single one: both lanes keep it)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float2 g = acc[0][2 * (k ^ X1) + h];
                        acc[0][2 * k + h].x += __shfl_xor_sync(0xffffffffu, g.x, 1);
                        acc[0][2 * k + h].y += __shfl_xor_sync(0xffffffffu, g.y, 1);
                    }
#pragma unroll
                for (int h = 0; h < 2; ++h) {  // the first of the two left
                    const float2 g = acc[0][2 * X2 + h];
                    acc[0][h].x += __shfl_xor_sync(0xffffffffu, g.x, 2);
                    acc[0][h].y += __shfl_xor_sync(0xffffffffu, g.y, 2);
                }
                if (so >= 0 && (ph & 3) < NP) {
                    const int c2 = 2 * (ph & (NP - 1));
                    const float sc = a.wsample ? a.scale * __ldg(&a.wsample[so]) : a.scale;
                    float2 *o = a.ks + (size_t)so * a.nc + a.c0 + c2;
                    const float2 u = make_float2(acc[0][0].x * sc, acc[0][0].y * sc);
                    const float2 v = make_float2(acc[0][1].x * sc, acc[0][1].y * sc);
                    if (a.pairs) {
                        if (c2 < a.cb) *reinterpret_cast<float4 *>(o) = make_float4(u.x, u.y, v.x, v.y);
                    } else {
                        if (c2 < a.cb) o[0] = u;
                        if (c2 + 1 < a.cb) o[1] = v;
                    }
                }
            } else {
                // every lane of a sample's four gets all its coils; lane j writes coils j and j + 4
#pragma unroll
                for (int o = 1; o <= 2; o <<= 1)
#pragma unroll
                    for (int k = 0; k < CB; ++k) {
                        acc[0][k].x += __shfl_xor_sync(0xffffffffu, acc[0][k].x, o);
                        acc[0][k].y += __shfl_xor_sync(0xffffffffu, acc[0][k].y, o);
                    }
                if (so >= 0) {
                    const float sc = a.wsample ? a.scale * __ldg(&a.wsample[so]) : a.scale;
                    float2 *o = a.ks + (size_t)so * a.nc + a.c0;
#pragma unroll
                    for (int k = 0; k < CB; ++k)
                        if ((k & 3) == (ph & 3)) o[k] = make_float2(acc[0][k].x * sc, acc[0][k].y * sc);
                }
            }
        }
    }
    // the last block out clears the work counter for the next launch
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(a.work + 1, 1) == (int)gridDim.x - 1) {
            a.work[0] = 0;
            a.work[1] = 0;
        }
    }
}

// ------------------------------------------------------------------ build
struct GatherBuild {
    const float4 *samples;
    const GatherRec *recs;
    Geom g;
    KBParams kb;
    int PS, ts;  // plane stride, z cells of a slab
};

// Place of entry e of a row in its chunks: lane l's two entries, l and l + 8
// of the chunk, are neighbours.
__device__ __forceinline__ int place_of(int e) { return (e & ~15) | ((e & 7) << 1) | ((e >> 3) & 1); }

// Plan time, one block per record, one warp per row: counts (FILL = false) or
// writes (FILL = true) the row's entries, walking the bounding box of its
// samples' supports.
template <bool FILL>
__global__ void __launch_bounds__(256)
k_gather_build(const __grid_constant__ GatherBuild b, uint32_t *__restrict__ cnt, const uint32_t *__restrict__ grow,
               float2 *__restrict__ gw, uint16_t *__restrict__ gi)
{
    const GatherRec rec = b.recs[blockIdx.x];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const Geom &g = b.g;
    for (int row = threadIdx.x >> 5; row < rec.nrows; row += blockDim.x >> 5) {
        float fx[kRow], fy[kRow], fz[kRow];
        int lx[kRow], ly[kRow], lz[kRow];
        int x0 = 1 << 20, x1 = 0, y0 = 1 << 20, y1 = 0, z0 = 1 << 20, z1 = 0;
        const int ns = min(kRow, rec.ns - kRow * row);
#pragma unroll
        for (int q = 0; q < kRow; ++q) {
            // absent samples of the last row get the first one's place and no weight
            const float4 r = __ldg(&b.samples[rec.s0 + kRow * row + (q < ns ? q : 0)]);
            const int packed = __float_as_int(r.w);
            fx[q] = r.x;
            fy[q] = r.y;
            fz[q] = r.z;
            lx[q] = packed & 0xFF;
            ly[q] = (packed >> 8) & 0xFF;
            // plane of the slab: cells of a slab follow the halo planes
            lz[q] = (((packed >> 16) & 0xFF) - g.Ra[2]) % b.ts + g.Ra[2];
            x0 = min(x0, lx[q] - g.Ra[0]);
            x1 = max(x1, lx[q] + g.Ra[0]);
            y0 = min(y0, ly[q] - g.Ra[1]);
            y1 = max(y1, ly[q] + g.Ra[1]);
            z0 = min(z0, lz[q] - g.Ra[2]);
            z1 = max(z1, lz[q] + g.Ra[2]);
        }
        const int nx = x1 - x0 + 1, nxy = nx * (y1 - y0 + 1), n = nxy * (z1 - z0 + 1);
        auto visit = [&](int i, bool weights, float (&w)[kRow], int &pt) {
            const int z = i / nxy, y = (i - z * nxy) / nx, x = i - z * nxy - y * nx;
            bool any = false;
#pragma unroll
            for (int q = 0; q < kRow; ++q) {
                w[q] = 0.f;
                if (q >= ns) continue;
                const float ex = __fsub_rn((float)(x0 + x - lx[q]), fx[q]), ey = __fsub_rn((float)(y0 + y - ly[q]), fy[q]),
                            ez = __fsub_rn((float)(z0 + z - lz[q]), fz[q]);
                const TapDist t = tap_dist(ex, ey, ez);
                if (!tap_inside(t, b.kb, g.radial)) continue;
                any = true;
                if (weights) w[q] = tap_value(t, b.kb, g.radial);
            }
            pt = (z0 + z) * b.PS + (y0 + y) * g.P[0] + x0 + x;
            return any;
        };
        int E = 0, O = 0;  // entries at even and odd points
        for (int i0 = 0; i0 < n; i0 += 32) {
            float w[kRow];
            int pt = 0;
            const bool hit = i0 + lane < n && visit(i0 + lane, false, w, pt);
            const unsigned m = __ballot_sync(0xffffffffu, hit), mo = __ballot_sync(0xffffffffu, hit && (pt & 1));
            O += __popc(mo);
            E += __popc(m & ~mo);
        }
        if (!FILL) {
            if (lane == 0) cnt[rec.row0 + row] = (uint32_t)((E + O + kChunk - 1) / kChunk);
            continue;
        }
        const size_t base = (size_t)__ldg(&grow[rec.row0 + row]) * kChunk;
        const int len = (int)((size_t)__ldg(&grow[rec.row0 + row + 1]) * kChunk - base);
        const int F = min(E, O) >> 2;  // whole groups of four even and four odd points
        int ne = 0, no = 0;
        for (int i0 = 0; i0 < n; i0 += 32) {
            float w[kRow];
            int pt = 0;
            const bool hit = i0 + lane < n && visit(i0 + lane, true, w, pt);
            const unsigned m = __ballot_sync(0xffffffffu, hit), mo = __ballot_sync(0xffffffffu, hit && (pt & 1));
            if (hit) {
                const bool odd = pt & 1;
                const int k = odd ? no + __popc(mo & lt) : ne + __popc(m & ~mo & lt);
                // phases 0-3 of a chunk take even points, 4-7 odd ones
                int pos;
                if (k < 4 * F) pos = (k >> 2) * 8 + (odd ? 4 : 0) + (k & 3);
                else pos = 8 * F + (odd ? E - 4 * F : 0) + (k - 4 * F);
                if (pos < len) {
                    gw[base + place_of(pos)] = (pos & 4) ? make_float2(w[1], w[0]) : make_float2(w[0], w[1]);
                    gi[base + place_of(pos)] = (uint16_t)pt;
                }
            }
            no += __popc(mo);
            ne += __popc(m & ~mo);
        }
        for (int p = E + O + lane; p < len; p += 32) {
            gw[base + place_of(p)] = make_float2(0.f, 0.f);
            gi[base + place_of(p)] = 0;
        }
    }
}

// Plan time, one warp per record: the record's whole rows sorted by length,
// longest first (a warp works on four neighbouring rows at a time and takes as
// long as the longest): rows are moved with their samples.
__global__ void __launch_bounds__(32)
k_gather_sort(const GatherRec *__restrict__ recs, uint32_t *__restrict__ cnt, float4 *__restrict__ samples,
              int32_t *__restrict__ perm, int32_t *__restrict__ inv)
{
    __shared__ uint32_t c[kRecRows];
    __shared__ float4 smp[kRecRows * kRow];
    __shared__ int32_t prm[kRecRows * kRow];
    const GatherRec r = recs[blockIdx.x];
    const int n = r.ns / kRow;  // whole rows
    for (int i = threadIdx.x; i < n; i += 32) c[i] = cnt[r.row0 + i];
    for (int i = threadIdx.x; i < n * kRow; i += 32) {
        smp[i] = samples[r.s0 + i];
        prm[i] = perm[r.s0 + i];
    }
    __syncwarp();
    for (int i = threadIdx.x; i < n; i += 32) {
        int rank = 0;
        for (int j = 0; j < n; ++j) rank += c[j] > c[i] || (c[j] == c[i] && j < i);
        cnt[r.row0 + rank] = c[i];
        for (int k = 0; k < kRow; ++k) {
            const int s = r.s0 + kRow * rank + k;
            samples[s] = smp[kRow * i + k];
            perm[s] = prm[kRow * i + k];
            inv[prm[kRow * i + k]] = s;
        }
    }
}

// The records' chunk ranges.
__global__ void k_gather_ranges(GatherRec *__restrict__ recs, int n, const uint32_t *__restrict__ grow)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    GatherRec &r = recs[i];
    r.chunk0 = grow[r.row0];
    r.nchunk = grow[r.row0 + r.nrows] - r.chunk0;
}

// ------------------------------------------------------------------- host
static int plane_stride(const Geom &g) { return (g.P[0] * g.P[1] + 15) & ~15; }  // whole 128-byte units for any CB

int slab_planes(const Geom &g) { return slab_cells(g) + 2 * g.Ra[2]; }

static void make_records(const nufft3d_plan *p, std::vector<GatherRec> &recs, uint32_t &nrows)
{
    const Geom &g = p->geom;
    const int spt = slabs_per_tile(g), ts = slab_cells(g), npl = slab_planes(g);
    int64_t s = 0;
    uint64_t row = 0;
    int prev_col = -1, prev_z = 0;
    for (size_t i = 0; i < p->slab_counts.size(); ++i) {
        const int cnt = p->slab_counts[i];
        if (cnt == 0) continue;
        const int t = (int)(i / spt), sl = (int)(i % spt);
        const int tz = t % g.nt[2], col = t / g.nt[2], tx = col % g.nt[0], ty = col / g.nt[0];
        const int z = tz * g.T[2] + sl * ts;
        int nload = col == prev_col ? std::min(npl, z - prev_z) : npl;
        for (int o = 0; o < cnt; o += kRow * kRecRows) {
            GatherRec r;
            r.ox = tx * g.T[0] + tile_shift(g) - g.Ra[0];
            r.oy = ty * g.T[1] - g.Ra[1];
            r.oz = z - g.Ra[2];
            r.nload = nload;
            r.chunk0 = r.nchunk = 0;
            r.row0 = (uint32_t)row;
            r.ns = std::min(kRow * kRecRows, cnt - o);
            r.nrows = (r.ns + kRow - 1) / kRow;
            r.s0 = (int)(s + o);
            recs.push_back(r);
            row += (uint64_t)r.nrows;
            nload = 0;
        }
        s += cnt;
        prev_col = col;
        prev_z = z;
    }
    nrows = (uint32_t)row;
}

// Record ranges: each about a sixth of what is left for each multiprocessor
// (rows, a loaded plane of 14 x 14 points counting as four, or 16 where the
// tile wraps around the grid edge and takes longer), so that the last ones are short,
// and at least 128 rows, below which the planes that a range loads anew
// outweigh its rows.
static std::vector<int2> make_chunks(const std::vector<GatherRec> &recs, const Geom &g, int sms)
{
    const int plane = std::max(1, plane_stride(g) / 196);  // planes of 14 x 14 points
    auto cost = [&](const GatherRec &r) {
        const bool inside = r.ox >= 0 && r.oy >= 0 && r.ox + g.P[0] <= g.K[0] && r.oy + g.P[1] <= g.K[1];
        return r.nrows + (inside ? 4 : 16) * r.nload * plane;
    };
    int64_t left = 0;
    for (auto &r : recs) left += cost(r);
    std::vector<int2> out;
    int64_t acc = 0;
    int lo = 0;
    for (int i = 0; i < (int)recs.size(); ++i) {
        acc += cost(recs[i]);
        if (acc >= std::max<int64_t>(128, left / ((int64_t)sms * 6)) || i + 1 == (int)recs.size()) {
            out.push_back(make_int2(lo, i + 1));
            lo = i + 1;
            left -= acc;
            acc = 0;
        }
    }
    return out;
}

// The stored H of the plan: records, rows, entries.  mode 0 = none, 1 =
// always, -1 = when it takes at most half of the free device memory.
int build_gather_table(nufft3d_plan *p, int mode, cudaStream_t s)
{
    if (mode == 0 || p->nnz == 0 || !tap_table_applies(p)) return NUFFT3D_SUCCESS;
    std::vector<GatherRec> recs;
    uint32_t nrows = 0;
    make_records(p, recs, nrows);
    const std::vector<int2> chunks = make_chunks(recs, p->geom, p->sm_count);
    struct Bufs {
        std::vector<void *> ptrs;
        ~Bufs()
        {
            NUFFT_DEVICE_LOCK;
            for (void *q : ptrs) cudaFree(q);
        }
    } tmp, keep;
    auto alloc = [&](auto **ptr, size_t n, Bufs &b) {
        NUFFT_DEVICE_LOCK;
        const cudaError_t e = cudaMalloc((void **)ptr, std::max<size_t>(n, 1) * sizeof(**ptr));
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(NUFFT3D_ERR_NOMEM, std::string("stored H: ") + cudaGetErrorString(e));
        }
        b.ptrs.push_back(*ptr);
        return NUFFT3D_SUCCESS;
    };
    auto none = [&](int st) {  // the kernels evaluate the weights instead
        if (mode > 0) return st;
        clear_error();
        return (int)NUFFT3D_SUCCESS;
    };
    GatherRec *drecs = nullptr;
    int2 *dchunks = nullptr;
    uint32_t *cnt = nullptr, *grow = nullptr;
    int st = alloc(&drecs, recs.size(), keep);
    if (st == NUFFT3D_SUCCESS) st = alloc(&dchunks, chunks.size(), keep);
    if (st == NUFFT3D_SUCCESS) st = alloc(&grow, (size_t)nrows + 1, keep);
    if (st == NUFFT3D_SUCCESS) st = alloc(&cnt, (size_t)nrows + 1, tmp);
    if (st != NUFFT3D_SUCCESS) return none(st);
    NUFFT_CUDA_TRY(cudaMemcpyAsync(drecs, recs.data(), sizeof(GatherRec) * recs.size(), cudaMemcpyHostToDevice, s));
    NUFFT_CUDA_TRY(cudaMemcpyAsync(dchunks, chunks.data(), sizeof(int2) * chunks.size(), cudaMemcpyHostToDevice, s));
    NUFFT_CUDA_TRY(cudaMemsetAsync(cnt + nrows, 0, sizeof(uint32_t), s));
    GatherBuild gb{p->samples, drecs, p->geom, p->kb, plane_stride(p->geom), slab_cells(p->geom)};
    k_gather_build<false><<<(unsigned)recs.size(), 256, 0, s>>>(gb, cnt, nullptr, nullptr, nullptr);
    NUFFT_CUDA_TRY(cudaGetLastError());
    k_gather_sort<<<(unsigned)recs.size(), 32, 0, s>>>(drecs, cnt, p->samples, p->perm, p->inv);
    NUFFT_CUDA_TRY(cudaGetLastError());
    size_t tb = 0;
    NUFFT_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, grow, (int64_t)nrows + 1, s));
    char *tstore = nullptr;
    if ((st = alloc(&tstore, tb, tmp)) != NUFFT3D_SUCCESS) return none(st);
    NUFFT_CUDA_TRY(cub::DeviceScan::ExclusiveSum(tstore, tb, cnt, grow, (int64_t)nrows + 1, s));
    uint32_t total = 0;
    NUFFT_CUDA_TRY(cudaMemcpyAsync(&total, grow + nrows, sizeof(total), cudaMemcpyDeviceToHost, s));
    NUFFT_CUDA_TRY(cudaStreamSynchronize(s));
    // chunk numbers are 32-bit: a row has at most kRow (2R+1)^3 points
    const int side = 2 * p->geom.R + 1;
    if ((uint64_t)nrows * (uint64_t)((kRow * side * side * (p->geom.is2d ? 1 : side) + kChunk - 1) / kChunk) >=
        0xffffffffull)
        return none(fail(NUFFT3D_ERR_SIZE, "too many samples for the stored H"));
    const size_t bytes = (size_t)total * kChunk * (sizeof(float2) + sizeof(uint16_t));
    if (mode < 0) {
        size_t fr = 0, to = 0;
        if (cudaMemGetInfo(&fr, &to) != cudaSuccess || bytes > fr / 2) {
            cudaGetLastError();
            return NUFFT3D_SUCCESS;
        }
    }
    float4 *gw = nullptr;
    uint32_t *gi = nullptr;
    st = alloc(&gw, (size_t)total * 8, keep);
    if (st == NUFFT3D_SUCCESS) st = alloc(&gi, (size_t)total * 8, keep);
    if (st != NUFFT3D_SUCCESS) return none(st);
    k_gather_build<true><<<(unsigned)recs.size(), 256, 0, s>>>(gb, nullptr, grow, reinterpret_cast<float2 *>(gw),
                                                              reinterpret_cast<uint16_t *>(gi));
    k_gather_ranges<<<(unsigned)((recs.size() + 255) / 256), 256, 0, s>>>(drecs, (int)recs.size(), grow);
    NUFFT_CUDA_TRY(cudaGetLastError());
    NUFFT_CUDA_TRY(cudaStreamSynchronize(s));
    p->grecs = drecs;
    p->gchunks = dchunks;
    p->n_gchunks = (int)chunks.size();
    p->grow = grow;
    p->gw = gw;
    p->gi = gi;
    p->tap_bytes = (int64_t)(bytes + sizeof(uint32_t) * ((size_t)nrows + 1) + sizeof(GatherRec) * recs.size() +
                             sizeof(int2) * chunks.size());
    p->table_bytes += p->tap_bytes;
    keep.ptrs.clear();
    return NUFFT3D_SUCCESS;
}

// Planes of the ring and its bytes for a coil width.
template <int CB>
static int ring_planes(const Geom &g, size_t *bytes)
{
    const size_t plane = (size_t)plane_stride(g) * CB * 8;
    const size_t room = (size_t)(227 * 1024) / GatherCfg<CB>::MINB - 8192 - (size_t)plane_stride(g) * sizeof(uint32_t);  // less the static part
    const int S = (int)std::min<size_t>(kRingPlanes, room / plane);
    *bytes = plane * S;
    return S;
}

template <int CB, int NPW, bool ROWS>
static int launch_rows(nufft3d_plan *p, GatherArgs &a, const CUtensorMap &m, cudaStream_t s)
{
    size_t smem = 0;
    a.S = ring_planes<CB>(p->geom, &smem);
    a.rbytes = (unsigned)smem;
    smem += (size_t)a.PS * sizeof(uint32_t);  // plane offsets
    if (a.S < a.npl) return fail(NUFFT3D_ERR_UNSUPPORTED, "stored H: plane ring too small");
    const int grid = std::min((a.nchunks + a.merge - 1) / a.merge, interp_grid_blocks(p, GatherCfg<CB>::MINB));
    k_gather_rows<CB, NPW, ROWS><<<grid, GatherCfg<CB>::WARPS * 32, smem, s>>>(a, m);
    NUFFT_CUDA_TRY(cudaGetLastError());
    return NUFFT3D_SUCCESS;
}

int launch_gather_tab(nufft3d_plan *p, const float2 *G, float2 *ks, int nc, int c0, int cb, float scale,
                      const float *ws, int merge, cudaStream_t s)
{
    const Geom &g = p->geom;
    GatherArgs a;
    std::memset(&a, 0, sizeof(a));
    a.G = G;
    a.ks = ks;
    a.nc = nc;
    a.c0 = c0;
    a.cb = std::min(cb, nc - c0);
    a.pairs = nc % 2 == 0 && c0 % 2 == 0;
    a.scale = scale;
    a.wsample = ws;
    a.recs = p->grecs;
    a.chunks = p->gchunks;
    a.nchunks = p->n_gchunks;
    a.merge = merge;
    a.grow = p->grow;
    a.gw = p->gw;
    a.gi = p->gi;
    for (int d = 0; d < 3; ++d) a.K[d] = g.K[d];
    a.P0 = g.P[0];
    a.P1 = g.P[1];
    a.rcpP0 = 65536 / g.P[0] + 1;
    a.small = g.P[0] > g.K[0] || g.P[1] > g.K[1] || g.P[2] > g.K[2];
    a.PS = plane_stride(g);
    a.npl = slab_planes(g);
    a.work = p->work + kWorkGatherTab;
    a.st = plan_status(p);
    alignas(64) CUtensorMap m;
    std::memset(&m, 0, sizeof(m));
    // an odd coil count in one pass: whole rows of points, every coil
    const bool odd = nc == a.cb && nc % 2 == 1 && nc < 8;
    if (odd) cb = nc;
    a.use_tma = p->use_tma && encode_plane_map(p, G, nc, cb, &m) ? 1 : 0;
    // Tiles that wrap around the grid edge are loaded row by row where a pass takes
    // every coil (gather of random samples in us, against copies by one and by
    // four producer warps: 8 coils at 96^3, 1000000 samples, 718, 824, 741, 65536 at
    // 64^3, J = 4, 212, 244, 228; 5 coils on 88 x 112 x 100 415, 657, 569; one coil at
    // 64^3, 262144, 100, 122, 148; radial samples, one coil at 48^3 51, 67, 61; a
    // bulk copy for each point of the other passes took 2 to 5 times as long as
    // the copies).  Eight coils on a grid of mostly outer tiles are left to the four
    // warps below: with a record of few rows the copies of all eight land sooner
    // (26^3, 49 % inner, radial / random 29 / 45 us row by row, 25 / 41; 48^3, 69 %, 62 /
    // 124, 66 / 119).
    const int inner = 100 * std::max(0, g.nt[0] - 2) * std::max(0, g.nt[1] - 2) / (g.nt[0] * g.nt[1]);
    if (p->use_tma && nc == cb && !a.small && (cb != 8 || g.is2d || inner >= 60)) {
        switch (cb) {
        case 1: return launch_rows<1, 1, true>(p, a, m, s);
        case 2: return launch_rows<2, 1, true>(p, a, m, s);
        case 3: return launch_rows<3, 1, true>(p, a, m, s);
        case 4: return launch_rows<4, 1, true>(p, a, m, s);
        case 5: return launch_rows<5, 1, true>(p, a, m, s);
        case 7: return launch_rows<7, 1, true>(p, a, m, s);
        default: return launch_rows<8, 1, true>(p, a, m, s);
        }
    }
    // Otherwise the producer warps copy them: four of them instead of one where
    // such tiles are common (percentage of inner tiles below the limit) gain on
    // the copies what the consumers lose in warps, the more the wider the pass.
    // One against four, radial / random samples, 8 coils: at 64^3 (76 % inner)
    // 174 / 315, 160 / 247 us, at 80^3 (81 %) 284 / 524, 292 / 459, at 96^3 (84 %)
    // 458 / 824, 501 / 741; 4 coils at 48^3 (69 %) 84 / 129, 79 / 113, at 64^3 144 / 225,
    // 150 / 230.  A 2-D plane is a whole tile of 38 x 38 points.  (An odd number of
    // coils takes this path without bulk copies, or on a grid of a tile or two.)
    const bool copies = !a.use_tma || g.is2d || inner < (cb == 8 ? 79 : cb == 4 ? 72 : 50);
    switch (cb) {
    case 1: return launch_rows<1, 4, false>(p, a, m, s);
    case 2: return copies ? launch_rows<2, 4, false>(p, a, m, s) : launch_rows<2, 1, false>(p, a, m, s);
    case 3: return launch_rows<3, 4, false>(p, a, m, s);
    case 4: return copies ? launch_rows<4, 4, false>(p, a, m, s) : launch_rows<4, 1, false>(p, a, m, s);
    case 5: return launch_rows<5, 4, false>(p, a, m, s);
    case 7: return launch_rows<7, 4, false>(p, a, m, s);
    default: return copies ? launch_rows<8, 4, false>(p, a, m, s) : launch_rows<8, 1, false>(p, a, m, s);
    }
}

template <int CB, int NPW, bool ROWS>
static int allow_rows()
{
    auto *k = k_gather_rows<CB, NPW, ROWS>;
    cudaFuncAttributes fa;
    NUFFT_CUDA_TRY(cudaFuncGetAttributes(&fa, k));
    NUFFT_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        227 * 1024 / GatherCfg<CB>::MINB - 1024 - (int)fa.sharedSizeBytes));
    return NUFFT3D_SUCCESS;
}

int configure_gather_tab_kernels()
{
    NUFFT_TRY((allow_rows<1, 1, true>()));
    NUFFT_TRY((allow_rows<2, 1, true>()));
    NUFFT_TRY((allow_rows<3, 1, true>()));
    NUFFT_TRY((allow_rows<4, 1, true>()));
    NUFFT_TRY((allow_rows<5, 1, true>()));
    NUFFT_TRY((allow_rows<7, 1, true>()));
    NUFFT_TRY((allow_rows<8, 1, true>()));
    NUFFT_TRY((allow_rows<1, 4, false>()));
    NUFFT_TRY((allow_rows<2, 1, false>()));
    NUFFT_TRY((allow_rows<2, 4, false>()));
    NUFFT_TRY((allow_rows<3, 4, false>()));
    NUFFT_TRY((allow_rows<4, 1, false>()));
    NUFFT_TRY((allow_rows<4, 4, false>()));
    NUFFT_TRY((allow_rows<5, 4, false>()));
    NUFFT_TRY((allow_rows<7, 4, false>()));
    NUFFT_TRY((allow_rows<8, 1, false>()));
    NUFFT_TRY((allow_rows<8, 4, false>()));
    return NUFFT3D_SUCCESS;
}

}  // namespace nufft3d
