// Spread (aNUFT's H' product, spmv_t of nufft_3d.m:274-282) from a stored
// transpose of H, for every coil width.
//
// The reference multiplies by the transpose of its sparse H through cuSPARSE
// (and on its CPU path keeps HT = H' as a matrix of its own, nufft_3d.m:218-219,
// so that the product reads a matrix laid out for it; this is that table for
// the GPU).  The on-the-fly spread (interp.cu) scatters each sample's taps into a tile
// with shared-memory integer reductions, which bounds it by instruction issue
// and the reduction pipe.  This form turns the product around: the samples of
// a piece are staged in shared memory, and the grid points of the piece's
// padded region are its rows, four at a time: a row owns a block of 2 x 2
// points (x, y) and holds an entry (four weights, sample) for every sample
// that reaches one of them.  A lane walks a row: one read of a sample's coils
// serves four points (44 reads a sample at J = 6 against 113 taps), the four
// points' coils accumulate in registers with FP32 FMAs, and the finished
// points are added to the grid with vector atomics (neighbouring pieces' halos
// overlap).  No shared-memory atomics, no kernel evaluation, and FP32
// accumulation throughout.
//
// Measured at 128^3 x 8 coils: 2.41 ms (a row a grid point: 2.81 ms), of which
// about 0.7 ms are the grid's atomics (a copy without them); no unit is above
// 52 % of its peak in a capture at 96^3, the warps wait at a piece's barriers
// (the runs end at different times) and on lines and atomics; 4 coils on 100 x 84 x 60 0.16 ms and one
// coil at 64^3 0.08 ms, where the spread evaluated the kernel before (0.46 and
// 0.24 ms).  A lane for a whole row (8 coils x 4 points: 64 accumulators, code
// that overflows the instruction cache when the loads are unrolled) took
// 3.9 ms, eight lines in flight instead of four 4.7 ms.
//
// A piece is a run of slabs of one tile column (the samples are sorted by
// column, slab and Hilbert position), at most kSpreadCap samples and kMaxExt
// cells of z; a slab with more samples than that is dealt to several pieces.
// Long runs in z keep the halo small (a piece adds (ext + 2R) / ext of its
// planes).
//
// Stored H' layout, per piece:
//   * the non-empty rows are sorted by length (longest first, ties by row) and
//     taken 16 at a time into bundles, so a warp walks 16 rows in lockstep (two
//     lanes a row) and every branch on the bundle structure is warp-uniform.  A
//     bundle is a run of lines, padded to whole steps of 4 lines; a line holds
//     one entry per row: a float4 of weights and the sample's slot (uint16) in
//     the staged samples (local index + 2; slots 0 and 1 stay zero and serve
//     as padding);
//   * the bundles are laid out in kBundleWarps runs of about equal length, one
//     per warp; a bundle that does not fit in what is left of a run is cut
//     into segments (both add their partial sums to the grid).  A segment has
//     its steps, one after the other, and a header: the grid indices of each
//     row's four points as int4 (-1 without a row) and the number of steps;
//   * the loads of a line's samples are free of bank conflicts while
//     neighbouring rows use different halves of the banks: odd rows read their
//     halves in the other order, and inside a row even-slot and odd-slot samples
//     alternate, starting with the parity of row / 2.  Leftovers of the larger
//     parity and padding (weight 0) follow.  Rows 2 and 3 of every four hold
//     their points in the order (x+1, x), see k_spread_rows.
// Inside a row each parity's samples keep the order in which the builder
// visits them, interleaved by a fixed rule (the fill is deterministic), so a
// row's FP32 sum does not depend on scheduling.
//
// The table is built from the samples (same weights and support test as the
// stored H) once per plan: a count pass gives each piece's steps and
// segments, the host scans them, and a fill pass writes the bundles.
#include <cub/block/block_radix_sort.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "async.h"
#include "internal.h"
#include "taps.h"

namespace nufft3d {

constexpr int kBundleWarps = 16;   // warps per block of the spread (512 threads)
constexpr int kRows = 16;          // rows of a bundle: two lanes each
constexpr int kLineBytes = kRows * (int)(sizeof(float4) + sizeof(uint16_t));
constexpr int kBundleDepth = 4;    // lines of a step: bodies are whole steps, which every lane keeps in flight
constexpr int kMaxExt = 48;        // z cells of a piece
// Lines of a warp's run that lane 0 asks L2 to fetch ahead of the register
// loads (kPrefetchAhead lines ahead, kPrefetchLines at a time), so that the
// loads wait on L2 rather than on DRAM.
constexpr int kPrefetchLines = 8;
constexpr int kPrefetchAhead = 24;

struct SpreadLines {
    const float4 *w;         // [line][16]: weights
    const uint16_t *x;       // [line][16]: sample slots
    const int4 *pts;         // [segment][16]: grid points
    const uint16_t *steps;   // [segment]: steps
};

__device__ __forceinline__ void prefetch_lines(const SpreadLines &t, uint32_t l, uint32_t l_hi)
{
    if (l >= l_hi) return;
    const uint32_t n = min((uint32_t)kPrefetchLines, l_hi - l);
    prefetch_l2(t.w + (size_t)l * kRows, n * (uint32_t)(kRows * sizeof(float4)));
    prefetch_l2(t.x + (size_t)l * kRows, n * (uint32_t)(kRows * sizeof(uint16_t)));
}

constexpr int kTabBuildThreads = 256;
constexpr int kTabBuildWarps = kTabBuildThreads / 32;
constexpr int kTabSortItems = 11;  // 256 x 11 >= 7 x 7 x (48 + 6) rows
constexpr int kMaxRows = kTabBuildThreads * kTabSortItems;
constexpr int kMaxBundles = (kMaxRows + kRows - 1) / kRows;

// A piece takes every stride-th sample from its first one on (y of the piece =
// count | stride << kCountBits; the stride is the number of pieces that share
// a slab, 1 for a run of slabs): samples of equal position follow one another
// in the sorted order (the centre of k-space, which every spoke of a radial
// trajectory samples), and an FP32 sum of many equal terms rounds the same way
// at every step.  Inside a piece the rows take the samples in a scattered order
// for the same reason.
constexpr int kCountBits = 11;
static_assert(kSpreadCap < (1 << kCountBits), "piece count");

__host__ __device__ __forceinline__ int piece_count(const int4 &pc) { return pc.y & ((1 << kCountBits) - 1); }
__host__ __device__ __forceinline__ int piece_stride(const int4 &pc) { return pc.y >> kCountBits; }

// A step coprime to n near n/phi: i -> i * step mod n visits 0..n-1 scattered.
__device__ __forceinline__ int scatter_step(int n)
{
    int g = max(1, (int)(0.618034f * (float)n));
    for (;; ++g) {
        int a = g, b = n;
        while (b) {
            const int t = a % b;
            a = b;
            b = t;
        }
        if (a == 1) return g;
    }
}

// Warp runs of a piece's bundles, of equal capacity in steps (a segment's
// header and flush counting as one): the bundles are laid out one after the
// other; a bundle that does not fit in what is left of a run is cut, and its
// rest continues in the next run, so every warp streams about as many steps as
// the others.
template <int MAXB>
struct RunLayout {
    uint16_t bl[MAXB];                          // steps of each bundle
    uint16_t fs[MAXB + 1];                      // first segment of each bundle
    uint16_t seg_i0[MAXB + 2 * kBundleWarps];   // a segment: steps [i0, i0 + n) of its bundle
    uint16_t seg_n[MAXB + 2 * kBundleWarps];
    uint32_t seg_step[MAXB + 2 * kBundleWarps];  // its first step in the piece
    uint32_t wstep[kBundleWarps + 1];           // first step and first segment of each warp's run
    uint32_t wseg[kBundleWarps + 1];
};

// Lays out nb bundles (bl set); one thread.
template <int MAXB>
__device__ void layout_runs(RunLayout<MAXB> &L, int nb)
{
    uint32_t T = 0;
    for (int k = 0; k < nb; ++k) T += 1u + L.bl[k];
    // (a cut adds a header of its own)
    const uint32_t C = (T + 3 * kBundleWarps - 1) / kBundleWarps;
    int w = 0, ns = 0;
    uint32_t used = 0, steps = 0;
    L.wstep[0] = L.wseg[0] = 0;
    for (int k = 0; k < nb; ++k) {
        L.fs[k] = (uint16_t)ns;
        uint32_t rem = L.bl[k], i0 = 0;
        while (rem > 0) {
            const uint32_t space = w < kBundleWarps - 1 ? C - min(used, C) : 0xFFFFFFFFu;  // the last run grows
            if (space < 2u) {
                ++w;
                L.wstep[w] = steps;
                L.wseg[w] = (uint32_t)ns;
                used = 0;
                continue;
            }
            // (a single step is not worth a header: the run grows by it)
            const uint32_t n = rem <= space ? rem : min(rem, space - 1u);
            L.seg_i0[ns] = (uint16_t)i0;
            L.seg_n[ns] = (uint16_t)n;
            L.seg_step[ns] = steps;
            ++ns;
            steps += n;
            used += 1u + n;
            rem -= n;
            i0 += n;
        }
    }
    L.fs[nb] = (uint16_t)ns;
    for (++w; w <= kBundleWarps; ++w) {
        L.wstep[w] = steps;
        L.wseg[w] = (uint32_t)ns;
    }
}

// Step of the piece that holds step i of bundle k.
template <int MAXB>
__device__ __forceinline__ uint32_t body_step(const RunLayout<MAXB> &L, int k, uint32_t i)
{
    int sg = L.fs[k];
    while (sg + 1 < (int)L.fs[k + 1] && i >= (uint32_t)L.seg_i0[sg] + L.seg_n[sg]) ++sg;
    return L.seg_step[sg] + (i - L.seg_i0[sg]);
}

using TabSort = cub::BlockRadixSort<uint32_t, kTabBuildThreads, kTabSortItems>;

struct TabBuildSmem {
    typename TabSort::TempStorage sort;
    RunLayout<kMaxBundles> L;
    uint16_t srow[kMaxRows];  // sorted rows
    int slab[kMaxExt / 2 + 2];  // first sample of each slab of the piece
    int nrows, step;
};

struct SpreadBuild {
    const int4 *pieces;       // (first sample, count | stride, first step, first slab)
    const uint32_t *seg0;     // first segment of each piece
    const int *ext;           // slabs of each piece
    const int *slab_start;    // first sample of each slab
    const float4 *samples;
    Geom g;
    KBParams kb;
    int ts, spt;              // z cells of a slab, slabs of a tile
};

// Plan time, one block per piece.  FILL = false: writes the piece's counts of
// steps and segments to size_out[b].  FILL = true: writes the piece's bundles
// from step pieces[b].z and segment seg0[b] on and the warps' first steps and
// segments to wstart.
// Dynamic shared memory: per-warp packed counts [warps][rows] (even-slot count
// | odd-slot count << 16), the row totals [rows] and each row's rank [rows].
// Warp w takes a contiguous run of the piece's scattered sample order, one
// sample at a time: its lanes take the candidate rows (the (R+1)^2 (2R+1)
// blocks of 2 x 2 points that the support can reach), which are distinct.
template <bool FILL>
__global__ void __launch_bounds__(kTabBuildThreads)
k_spread_tab_build(const __grid_constant__ SpreadBuild sb, uint2 *__restrict__ size_out,
                   uint2 *__restrict__ wstart, float4 *__restrict__ ent, uint16_t *__restrict__ idx,
                   int4 *__restrict__ seg_pts, uint16_t *__restrict__ seg_n)
{
    extern __shared__ uint32_t sm[];
    __shared__ TabBuildSmem ss;
    const Geom &g = sb.g;
    const int4 pc = sb.pieces[blockIdx.x];
    const int nslab = sb.ext[blockIdx.x];
    const int RX = g.P[0] / 2, RY = g.P[1] / 2, RZ = nslab * sb.ts + 2 * g.Ra[2];
    const int P = RX * RY * RZ;
    uint32_t *hist = sm;
    uint32_t *tot = sm + kTabBuildWarps * P;
    uint32_t *rank = tot + P;  // rank of row p (sorted order), or ~0u
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int np = piece_count(pc), stride = piece_stride(pc);
    for (int i = tid; i < kTabBuildWarps * P; i += blockDim.x) hist[i] = 0;
    for (int i = tid; i < nslab; i += blockDim.x) ss.slab[i] = sb.slab_start[pc.w + i];
    if (tid == 0) {
        ss.step = scatter_step(np);
        ss.nrows = 0;
    }
    __syncthreads();
    const int step = ss.step;
    const int i_lo = (np * warp) / kTabBuildWarps, i_hi = (np * (warp + 1)) / kTabBuildWarps;
    uint32_t *h = hist + (size_t)warp * P;
    // this lane's candidates: block offsets (ca, cb) and plane cc
    constexpr int kCand = 4;
    const int side = g.R + 1, ncand = side * side * (2 * g.Ra[2] + 1);
    int ca[kCand], cb[kCand], cc[kCand];
#pragma unroll
    for (int k = 0; k < kCand; ++k) {
        const int i = lane + 32 * k;
        cc[k] = i < ncand ? i / (side * side) : -1;
        const int r = i % (side * side);
        cb[k] = r / side;
        ca[k] = r - cb[k] * side;
    }
    // visits the rows that sample i of the scattered order reaches:
    // f(row, slot, weights), weights only when FILL
    auto visit = [&](int i, bool weights, auto &&f) {
        const int sl = (int)((long long)i * step % np), s = pc.x + sl * stride;
        const float4 rec = __ldg(&sb.samples[s]);
        const int packed = __float_as_int(rec.w);
        const int lx = packed & 0xFF, ly = (packed >> 8) & 0xFF;
        const unsigned below = __ballot_sync(0xffffffffu, lane < nslab && ss.slab[lane] <= s);
        const int zs = 32 - __clz(below) - 1;  // its slab
        const int z = zs * sb.ts + (((packed >> 16) & 0xFF) - g.Ra[2]) % sb.ts + g.Ra[2];
        const int bx = (lx - g.Ra[0]) >> 1, by = (ly - g.Ra[1]) >> 1;
#pragma unroll
        for (int k = 0; k < kCand; ++k) {
            if (cc[k] < 0) continue;
            const int qx = bx + ca[k], qy = by + cb[k], zz = z - g.Ra[2] + cc[k];
            const float ez = __fsub_rn((float)(zz - z), rec.z);
            float w[4];
            bool any = false;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const TapDist t = tap_dist(__fsub_rn((float)(2 * qx + (q & 1) - lx), rec.x),
                                           __fsub_rn((float)(2 * qy + (q >> 1) - ly), rec.y), ez);
                const bool in = tap_inside(t, sb.kb, g.radial);
                any |= in;
                w[q] = weights && in ? tap_value(t, sb.kb, g.radial) : 0.f;
            }
            if (any) f((zz * RY + qy) * RX + qx, sl, make_float4(w[0], w[1], w[2], w[3]));
        }
        __syncwarp();
    };
    for (int i = i_lo; i < i_hi; ++i)
        visit(i, false, [&](int p, int sl, float4) { h[p] += (sl & 1) ? 0x10000u : 1u; });
    __syncthreads();
    // per row: exclusive prefix over the warps and the row's total
    for (int p = tid; p < P; p += blockDim.x) {
        uint32_t acc = 0;
        for (int w = 0; w < kTabBuildWarps; ++w) {
            const uint32_t v = hist[(size_t)w * P + p];
            hist[(size_t)w * P + p] = acc;
            acc += v;
        }
        tot[p] = acc;
    }
    __syncthreads();
    // rows by length, longest first, ties by row: key (4095 - L) << 12 | p
    uint32_t key[kTabSortItems];
#pragma unroll
    for (int i = 0; i < kTabSortItems; ++i) {
        const int p = tid * kTabSortItems + i;
        uint32_t k = 0xFFFFFFFFu;
        if (p < P) {
            const uint32_t a = tot[p], L = (a & 0xFFFFu) + (a >> 16);
            k = ((4095u - L) << 12) | (uint32_t)p;
        }
        key[i] = k;
    }
    __syncthreads();
    TabSort(ss.sort).Sort(key, 0, 24);
    // blocked arrangement: thread t holds sorted positions t*items + i; the
    // rows with entries come first
#pragma unroll
    for (int i = 0; i < kTabSortItems; ++i) {
        const uint32_t k = key[i];
        if (k == 0xFFFFFFFFu) continue;
        const bool row = (k >> 12) != 4095u;
        rank[k & 0xFFFu] = row ? (uint32_t)(tid * kTabSortItems + i) : 0xFFFFFFFFu;
        if (row) {
            ss.srow[tid * kTabSortItems + i] = (uint16_t)(k & 0xFFFu);
            atomicAdd(&ss.nrows, 1);
        }
    }
    __syncthreads();
    const int nr = ss.nrows, nb = (nr + kRows - 1) / kRows;
    // bundle lengths: a bundle's first row is its longest
    for (int p = tid; p < P; p += blockDim.x) {
        const uint32_t r = rank[p];
        if (r != 0xFFFFFFFFu && r % kRows == 0) {
            const uint32_t a = tot[p];
            ss.L.bl[r / kRows] = (uint16_t)(((a & 0xFFFFu) + (a >> 16) + kBundleDepth - 1) / kBundleDepth);  // steps
        }
    }
    __syncthreads();
    if (tid == 0) layout_runs(ss.L, nb);
    __syncthreads();
    if (!FILL) {
        if (tid == 0) size_out[blockIdx.x] = make_uint2(ss.L.wstep[kBundleWarps], ss.L.wseg[kBundleWarps]);
        return;
    }
    const uint32_t base = (uint32_t)pc.z, seg0 = sb.seg0[blockIdx.x];
    if (tid <= kBundleWarps)
        wstart[(size_t)blockIdx.x * (kBundleWarps + 1) + tid] = make_uint2(base + ss.L.wstep[tid], seg0 + ss.L.wseg[tid]);
    // entry j of row r of bundle k lies in one of the bundle's segments
    auto at = [&](int k, int r, uint32_t j) -> size_t {
        const uint32_t step = base + body_step(ss.L, k, j / kBundleDepth);
        return ((size_t)step * kBundleDepth + j % kBundleDepth) * kRows + (size_t)r;
    };
    // headers of every segment and the padding of the rows up to their bundle's length
    const int tile = pc.w / sb.spt, tz = tile % g.nt[2], tx = tile / g.nt[2] % g.nt[0], ty = tile / (g.nt[2] * g.nt[0]);
    const int ox = tx * g.T[0] + tile_shift(g) - g.Ra[0], oy = ty * g.T[1] - g.Ra[1];
    const int oz = tz * g.T[2] + pc.w % sb.spt * sb.ts - g.Ra[2];
    auto wrap = [](int x, int K) {
        x %= K;
        return x < 0 ? x + K : x;
    };
    for (int i = tid; i < nb * kRows; i += blockDim.x) {
        const int k = i / kRows, r = i % kRows;
        int4 hd = make_int4(-1, -1, -1, -1);
        uint32_t L = 0;
        if (i < nr) {
            const int p = ss.srow[i];
            const uint32_t a = tot[p];
            L = (a & 0xFFFFu) + (a >> 16);
            const int x = ox + 2 * (p % RX), y = oy + 2 * (p / RX % RY), z = oz + p / (RX * RY);
            const long long zr = (long long)wrap(z, g.K[2]) * g.K[1];
            const int x0 = wrap(x, g.K[0]), x1 = wrap(x + 1, g.K[0]);
            const long long y0 = (zr + wrap(y, g.K[1])) * g.K[0], y1 = (zr + wrap(y + 1, g.K[1])) * g.K[0];
            hd = make_int4((int)(y0 + x0), (int)(y0 + x1), (int)(y1 + x0), (int)(y1 + x1));
            if (r & 2) hd = make_int4(hd.y, hd.x, hd.w, hd.z);
        }
        for (int sg = ss.L.fs[k]; sg < (int)ss.L.fs[k + 1]; ++sg) {
            seg_pts[((size_t)seg0 + sg) * kRows + r] = hd;
            if (r == 0) seg_n[(size_t)seg0 + sg] = ss.L.seg_n[sg];
        }
        for (uint32_t j = L; j < (uint32_t)ss.L.bl[k] * kBundleDepth; ++j) {  // weight 0, alternating zero slots
            const size_t o = at(k, r, j);
            ent[o] = make_float4(0.f, 0.f, 0.f, 0.f);
            idx[o] = (uint16_t)((j + (r >> 1)) & 1u);
        }
    }
    // the entries: row r starts with parity (r / 2) & 1, then alternates while
    // both parities last; leftovers follow in the visiting order
    for (int i = i_lo; i < i_hi; ++i)
        visit(i, true, [&](int p, int sl, const float4 &w) {
            const int par = sl & 1;
            const uint32_t hv = h[p];
            h[p] = hv + (par ? 0x10000u : 1u);
            const uint32_t rk = par ? hv >> 16 : hv & 0xFFFFu;
            const uint32_t a = tot[p], m = min(a & 0xFFFFu, a >> 16);
            const uint32_t rr = rank[p];
            const int k = (int)(rr / kRows), r = (int)(rr % kRows);
            const uint32_t j = rk < m ? 2u * rk + (uint32_t)(par != ((r >> 1) & 1)) : 2u * m + (rk - m);
            const size_t o = at(k, r, j);
            ent[o] = r & 2 ? make_float4(w.y, w.x, w.w, w.z) : w;
            idx[o] = (uint16_t)(sl + 2);
        });
}

// Blocks per SM by coil width.
template <int CB>
struct SpreadCfg;
template <> struct SpreadCfg<8> { static constexpr int MINB = 1; };
template <> struct SpreadCfg<4> { static constexpr int MINB = 1; };
template <> struct SpreadCfg<2> { static constexpr int MINB = 1; };
template <> struct SpreadCfg<1> { static constexpr int MINB = 2; };

// Stage the samples of a piece into one of the two sample buffers (slot
// 2 + i holds the piece's sample i) with asynchronous copies; the caller
// waits for them (cp.async.wait_all) and synchronises before reading.
template <int CB>
__device__ __forceinline__ void stage_samples(const float2 *__restrict__ ks, int nc, int c0, int cb, bool pairs,
                                              const int4 pc, unsigned buf_sa)
{
    const int first = pc.x, n = piece_count(pc), stride = piece_stride(pc);
    if (CB >= 2 && pairs) {
        constexpr int U = CB >= 2 ? CB / 2 : 1;
        for (int i = threadIdx.x; i < n * U; i += blockDim.x) {
            const int sl = i / U, u = i % U;
            if (2 * u < cb)
                copy_async16(buf_sa + (unsigned)((sl + 2) * (CB * 8) + u * 16),
                             ks + (size_t)(first + sl * stride) * nc + c0 + 2 * u);
        }
    } else {
        for (int i = threadIdx.x; i < n * CB; i += blockDim.x) {
            const int sl = i / CB, c = i % CB;
            if (c < cb)
                copy_async8(buf_sa + (unsigned)((sl + 2) * (CB * 8) + c * 8),
                            ks + (size_t)(first + sl * stride) * nc + c0 + c);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The spread.  Persistent blocks take pieces from a work counter, one piece
// ahead: while a piece is applied from one sample buffer, the next piece's
// samples land in the other, and each warp's first lines of the next piece are
// loaded into its pipeline before the piece barrier.  Warp w streams its run of
// lines, segment by segment: lane (r, h) = (lane / 2, lane % 2) applies row r's entry of each
// line; 8 and 4 coils are split between a row's two lanes by coil pair, 2 coils
// and 1 by point (x parity).  After a segment's last step the finished points
// are added to the grid.  The lines end with a spare step, so the loads that run
// ahead need no bounds test.
//
// The vector atomics leave the chip at about 50 G requests a second (timed by
// themselves), whatever their width (a request is what one warp instruction adds to one
// 128-byte line), so the four rows of eight lanes exchange their 16-byte parts
// first and each instruction adds whole points: two neighbouring points of 8
// coils, 128 bytes, a request.
template <int CB>
__global__ void __launch_bounds__(kBundleWarps * 32, SpreadCfg<CB>::MINB)
k_spread_rows(const float2 *__restrict__ ks, float2 *__restrict__ G, int nc, int c0, int cb,
              const int4 *__restrict__ pieces, int npieces, int cap, int *__restrict__ work,
              const uint2 *__restrict__ wstart, SpreadLines t)
{
    constexpr int D = kBundleDepth, SLOT = CB * 8;
    constexpr int NU = CB == 8 ? 2 : 1;   // 16-byte units of a lane (8 bytes for a single coil)
    constexpr int NQ = CB >= 4 ? 4 : 2;   // points of a lane
    constexpr int NV = CB >= 2 ? 2 : 1;   // coils of a unit
    extern __shared__ __align__(16) unsigned char ysm[];  // two buffers of cap + 2 slots; slots 0 and 1 stay zero
    __shared__ int next;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = lane >> 1, h = lane & 1, rho = row & 3;
    const unsigned bufb = (unsigned)(cap + 2) * SLOT;
    const bool pairs = nc % 2 == 0 && c0 % 2 == 0;
    if (tid < 2 * CB) {
        reinterpret_cast<float2 *>(ysm)[tid] = make_float2(0.f, 0.f);
        reinterpret_cast<float2 *>(ysm + bufb)[tid] = make_float2(0.f, 0.f);
    }
    const unsigned ys_sa = (unsigned)__cvta_generic_to_shared(ysm);
    // byte offsets of this lane's units: of 8 coils, units h and h + 2, the
    // second one first in odd rows
    const unsigned u0 = CB == 8 ? 16u * (unsigned)(h + 2 * (rho & 1)) : CB == 4 ? 16u * h : 0u;
    const unsigned u1 = CB == 8 ? 16u * (unsigned)(h + 2 * (1 - (rho & 1))) : 0u;
    const float4 *lw = t.w + row;
    const uint16_t *lx = t.x + row;
    if (tid == 0) next = atomicAdd(work, 1);
    __syncthreads();
    int b = next;
    float4 e[D];
    unsigned x[D];
    uint32_t l_lo = 0, l_hi = 0, s_lo = 0, s_hi = 0;  // lines and segments of this warp's run
    unsigned n_next = 0;                               // steps of its next segment
    auto first_lines = [&](int piece) {
        const uint2 lo = __ldg(&wstart[(size_t)piece * (kBundleWarps + 1) + warp]);
        const uint2 hi = __ldg(&wstart[(size_t)piece * (kBundleWarps + 1) + warp + 1]);
        l_lo = lo.x * D;
        l_hi = hi.x * D;
        s_lo = lo.y;
        s_hi = hi.y;
        n_next = __ldg(t.steps + s_lo);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            e[k] = ld_stream4(lw + (size_t)(l_lo + k) * kRows);
            x[k] = ld_stream16(lx + (size_t)(l_lo + k) * kRows);
        }
    };
    if (b < npieces) {
        stage_samples<CB>(ks, nc, c0, cb, pairs, pieces[b], ys_sa);
        first_lines(b);
    }
    int buf = 0;
    while (b < npieces) {
        __syncthreads();  // every thread has read `next`
        if (tid == 0) next = atomicAdd(work, 1);
        if (lane == 0)
            for (int k = 0; k < kPrefetchAhead + kPrefetchLines; k += kPrefetchLines)
                prefetch_lines(t, l_lo + D + k, l_hi);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();  // this piece's samples are in, `next` is set
        const int bn = next;
        if (bn < npieces) stage_samples<CB>(ks, nc, c0, cb, pairs, pieces[bn], ys_sa + (buf ? 0u : bufb));
        const unsigned char *ys = ysm + (buf ? bufb : 0u);
        float2 acc[NQ][NU * NV];
        auto clear = [&]() {
#pragma unroll
            for (int q = 0; q < NQ; ++q)
#pragma unroll
                for (int c = 0; c < NU * NV; ++c) acc[q][c] = make_float2(0.f, 0.f);
        };
        clear();
        int4 gp;  // this row's grid points
        auto add4 = [&](int g, unsigned unit, const float4 v) {  // a coil pair of grid point g
            if (g >= 0 && 2 * (int)unit < cb) atomicAdd(reinterpret_cast<float4 *>(G + (size_t)g * nc + c0 + 2 * unit), v);
        };
        auto swap4 = [&](const float4 v, int m) {
            return make_float4(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m),
                               __shfl_xor_sync(0xffffffffu, v.z, m), __shfl_xor_sync(0xffffffffu, v.w, m));
        };
        auto part = [&](int q, int k) {  // unit register k of point register q
            return make_float4(acc[q][2 * k].x, acc[q][2 * k].y, acc[q][2 * k + 1].x, acc[q][2 * k + 1].y);
        };
        auto either = [&](bool c, const float4 x, const float4 y) {
            return make_float4(c ? x.x : y.x, c ? x.y : y.y, c ? x.z : y.z, c ? x.w : y.w);
        };
        auto add_points = [&]() {
            const int gi[4] = {gp.x, gp.y, gp.z, gp.w};
            if constexpr (CB == 8) {
                if (pairs) {
#pragma unroll
                    for (int q = 0; q < 4; q += 2) {
                        // Of a row's two points and a lane's two units, register
                        // part j (unit bit 0, point bit 1) is part j ^ rho of the
                        // row: giving part s to the row rho ^ s leaves every lane
                        // with part rho of four rows, t[s] of row rho ^ s.
                        float4 t[4];
                        t[0] = part(q, 0);
                        t[1] = swap4(part(q, 1), 2);
                        t[2] = swap4(part(q + 1, 0), 4);
                        t[3] = swap4(part(q + 1, 1), 6);
                        const int p0 = rho & 2 ? gi[q + 1] : gi[q], p1 = rho & 2 ? gi[q] : gi[q + 1];
#pragma unroll
                        for (int R = 0; R < 4; ++R) {
                            // row R of the four: t[rho ^ R]
                            const float4 v = either(((rho ^ R) & 2) != 0, either((rho ^ R) & 1, t[3], t[2]),
                                                    either((rho ^ R) & 1, t[1], t[0]));
                            const int src = (lane & 24) + 2 * R;
                            const int g0 = __shfl_sync(0xffffffffu, p0, src), g1 = __shfl_sync(0xffffffffu, p1, src);
                            add4(rho & 2 ? g1 : g0, u0 / 16, v);
                        }
                    }
                    return;
                }
            }
            if (CB == 4 && pairs) {
                // rows r and r ^ 2 exchange one of two neighbouring points (they
                // hold them in opposite order): 64 bytes of one row, then of the other
                const bool up = rho & 2;
#pragma unroll
                for (int q = 0; q < 4; q += 2) {
                    const float4 mine = part(q, 0), other = swap4(part(q + 1, 0), 4);
                    const int go = __shfl_xor_sync(0xffffffffu, gi[q + 1], 4);
                    add4(up ? go : gi[q], u0 / 16, either(up, other, mine));
                    add4(up ? gi[q] : go, u0 / 16, either(up, mine, other));
                }
            } else if constexpr (CB >= 4) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (gi[q] < 0) continue;
                    float2 *o = G + (size_t)gi[q] * nc + c0;
#pragma unroll
                    for (int k = 0; k < NU; ++k) {
                        const int c = (int)(k == 0 ? u0 : u1) / 8;
                        if (c < cb) atomicAdd(o + c, acc[q][2 * k]);
                        if (c + 1 < cb) atomicAdd(o + c + 1, acc[q][2 * k + 1]);
                    }
                }
            } else {
                const int ga = h ? gp.y : gp.x, gb = h ? gp.w : gp.z;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int g1 = q ? gb : ga;
                    if constexpr (CB == 2) {
                        if (pairs) {
                            add4(g1, 0, part(q, 0));
                            continue;
                        }
                    }
                    if (g1 < 0) continue;
                    atomicAdd(G + (size_t)g1 * nc + c0, acc[q][0]);
                    if constexpr (CB == 2)
                        if (cb > 1) atomicAdd(G + (size_t)g1 * nc + c0 + 1, acc[q][1]);
                }
            }
        };
        // A step's lines are summed by themselves: a quarter of the additions to
        // the long sums, whose rounding grows with their number (64^3 koosh
        // ball, 8 coils: error against FP64 1.65e-7 -> 1.32e-7, the time as before).
        float2 sum4[NQ][NU * NV];
        auto line = [&](const float4 w, unsigned sx, bool first) {
            auto mad = [&](float2 x, float2 y, float2 c) { return first ? __fmul2_rn(x, y) : __ffma2_rn(x, y, c); };
            const unsigned char *y = ys + sx * SLOT;
            const float ws[4] = {w.x, w.y, w.z, w.w};
            if constexpr (CB >= 4) {
                float4 v[NU];
                v[0] = *reinterpret_cast<const float4 *>(y + u0);
                if constexpr (NU == 2) v[1] = *reinterpret_cast<const float4 *>(y + u1);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 ww = make_float2(ws[q], ws[q]);
#pragma unroll
                    for (int k = 0; k < NU; ++k) {
                        sum4[q][2 * k] = mad(ww, make_float2(v[k].x, v[k].y), sum4[q][2 * k]);
                        sum4[q][2 * k + 1] = mad(ww, make_float2(v[k].z, v[k].w), sum4[q][2 * k + 1]);
                    }
                }
            } else {
                const float wa = h ? w.y : w.x, wb = h ? w.w : w.z;
                if constexpr (CB == 2) {
                    const float4 v = *reinterpret_cast<const float4 *>(y);
                    sum4[0][0] = mad(make_float2(wa, wa), make_float2(v.x, v.y), sum4[0][0]);
                    sum4[0][1] = mad(make_float2(wa, wa), make_float2(v.z, v.w), sum4[0][1]);
                    sum4[1][0] = mad(make_float2(wb, wb), make_float2(v.x, v.y), sum4[1][0]);
                    sum4[1][1] = mad(make_float2(wb, wb), make_float2(v.z, v.w), sum4[1][1]);
                } else {
                    const float2 v = *reinterpret_cast<const float2 *>(y);
                    sum4[0][0] = mad(make_float2(wa, wa), v, sum4[0][0]);
                    sum4[1][0] = mad(make_float2(wb, wb), v, sum4[1][0]);
                }
            }
        };
        uint32_t l = l_lo, pf = l_lo + D + kPrefetchAhead + kPrefetchLines;  // next line, next one to prefetch
        for (uint32_t sg = s_lo; sg < s_hi; ++sg) {
            const unsigned n = n_next;
            n_next = __ldg(t.steps + sg + 1);
            gp = __ldg(t.pts + (size_t)sg * kRows + row);
            for (unsigned i = 0; i < n; ++i, l += D) {
                if (lane == 0 && l + D + kPrefetchAhead >= pf) {
                    prefetch_lines(t, pf, l_hi);
                    pf += kPrefetchLines;
                }
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const float4 w = e[k];
                    const unsigned sx = x[k];
                    e[k] = ld_stream4(lw + (size_t)(l + k + D) * kRows);
                    x[k] = ld_stream16(lx + (size_t)(l + k + D) * kRows);
                    line(w, sx, k == 0);
                }
#pragma unroll
                for (int q = 0; q < NQ; ++q)
#pragma unroll
                    for (int c = 0; c < NU * NV; ++c) acc[q][c] = __fadd2_rn(acc[q][c], sum4[q][c]);
            }
            add_points();
            clear();
        }
        // the next piece's first lines, while the others finish this piece
        if (bn < npieces) first_lines(bn);
        __syncthreads();  // this buffer is free: the piece after next lands in it
        buf ^= 1;
        b = bn;
    }
    // the last block out clears the work counter for the next launch
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(work + 1, 1) == (int)gridDim.x - 1) {
            work[0] = 0;
            work[1] = 0;
        }
    }
}

// ---------------------------------------------------------------- host

template <int CB>
static size_t spread_smem(int cap)
{
    return (size_t)2 * (cap + 2) * CB * 8;
}

template <int CB>
static int launch_rows(nufft3d_plan *p, const float2 *ks, float2 *G, int nc, int c0, cudaStream_t s)
{
    const size_t smem = spread_smem<CB>(p->spread_cap);
    const int64_t grid = std::min<int64_t>(p->n_spread_pieces, (int64_t)interp_grid_blocks(p, SpreadCfg<CB>::MINB));
    k_spread_rows<CB><<<(unsigned)grid, kBundleWarps * 32, smem, s>>>(
        ks, G, nc, c0, std::min(CB, nc - c0), p->spread_pieces, (int)p->n_spread_pieces, p->spread_cap,
        p->work + kWorkSpreadTab, p->spread_wstart,
        SpreadLines{p->spread_ent, p->spread_idx, p->spread_pts, p->spread_steps});
    NUFFT_CUDA_TRY(cudaGetLastError());
    return NUFFT3D_SUCCESS;
}

int launch_spread_tab(nufft3d_plan *p, const float2 *ks, float2 *G, int nc, int c0, int cb, cudaStream_t s)
{
    if (p->n_spread_pieces == 0) return NUFFT3D_SUCCESS;
    switch (cb) {
    case 1: return launch_rows<1>(p, ks, G, nc, c0, s);
    case 2: return launch_rows<2>(p, ks, G, nc, c0, s);
    case 4: return launch_rows<4>(p, ks, G, nc, c0, s);
    default: return launch_rows<8>(p, ks, G, nc, c0, s);
    }
}

template <int CB>
static int allow_rows()
{
    NUFFT_CUDA_TRY(cudaFuncSetAttribute(k_spread_rows<CB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)spread_smem<CB>(kSpreadCap)));
    return NUFFT3D_SUCCESS;
}

int configure_spread_tab_kernels()
{
    NUFFT_TRY(allow_rows<1>());
    NUFFT_TRY(allow_rows<2>());
    NUFFT_TRY(allow_rows<4>());
    NUFFT_TRY(allow_rows<8>());
    for (auto k : {k_spread_tab_build<false>, k_spread_tab_build<true>}) {
        cudaFuncAttributes fa;
        NUFFT_CUDA_TRY(cudaFuncGetAttributes(&fa, k));
        NUFFT_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            227 * 1024 - (int)fa.sharedSizeBytes));
    }
    return NUFFT3D_SUCCESS;
}

// Pieces of at most cap samples: runs of slabs of one column, or shares of a
// larger slab; most samples first (the heavy centre of radial k-space starts
// early).  ext: slabs of each piece.  A larger slab is dealt to pieces of up to
// twice cap: every one of them adds to the same few points of the grid, and the
// rounding of those sums grows with their number, while a larger share holds
// up the block that takes it (64^3 koosh ball, 262144 samples, cap 431; error
// against FP64 of 8 coils and adjoint of one coil: shares of 431 1.9e-7, 124 us,
// of 862 1.3e-7, 123 us, of 1664 1.2e-7, 129 us).
static void make_spread_pieces(const nufft3d_plan *p, int cap, std::vector<int4> &pcs, std::vector<int> &ext)
{
    const Geom &g = p->geom;
    const int spt = slabs_per_tile(g), col_slabs = spt * g.nt[2];
    const int max_slabs = std::max(1, kMaxExt / slab_cells(g));
    struct Run {
        int4 pc;
        int ext;
    };
    std::vector<Run> runs;
    int64_t off = 0;
    int first = 0, start = -1, count = 0;  // the open run: first sample, first slab (-1: none), samples
    auto close = [&](int end) {
        if (start >= 0) runs.push_back({make_int4(first, count | 1 << kCountBits, 0, start), end - start});
        start = -1;
    };
    int last = -1;  // last non-empty slab of the open run
    for (int i = 0; i < (int)p->slab_counts.size(); ++i) {
        const int c = p->slab_counts[i];
        if (c == 0) continue;
        if (start >= 0 && (i / col_slabs != start / col_slabs || i - start >= max_slabs || count + c > cap)) close(last + 1);
        if (c > cap) {
            const int share = std::min(kSpreadCap, 2 * cap), nb = (c + share - 1) / share;
            for (int b = 0; b < nb; ++b)
                runs.push_back({make_int4((int)(off + b), (c - b + nb - 1) / nb | nb << kCountBits, 0, i), 1});
        } else {
            if (start < 0) {
                start = i;
                first = (int)off;
                count = 0;
            }
            count += c;
            last = i;
        }
        off += c;
    }
    close(last + 1);
    std::stable_sort(runs.begin(), runs.end(),
                     [](const Run &a, const Run &b) { return piece_count(a.pc) > piece_count(b.pc); });
    for (auto &r : runs) {
        pcs.push_back(r.pc);
        ext.push_back(r.ext);
    }
}

static size_t build_smem(const Geom &g, int cells)
{
    return (size_t)(kTabBuildWarps + 2) * (g.P[0] / 2) * (g.P[1] / 2) * (cells + 2 * g.Ra[2]) * sizeof(uint32_t);
}

// The stored H' (with the stored H).  mode 0 = none, 1 = always, -1 = when it
// takes at most half of the free device memory.
int build_spread_table(nufft3d_plan *p, int mode, cudaStream_t s)
{
    if (mode == 0 || p->gw == nullptr || p->nnz == 0) return NUFFT3D_SUCCESS;
    const Geom &g = p->geom;
    // Runs for about four pieces a multiprocessor where the samples are few (64^3
    // x 1 coil, 262144 samples: 80 us, with the largest pieces 99 us).  A 2-D piece holds
    // a whole tile of 38 x 38 points however few its samples are, so there
    // smaller pieces only add points (256^2 x 8 coils: 27 us, four a
    // multiprocessor 41 us).
    const int cap = g.is2d ? kSpreadCap
                           : (int)std::max<int64_t>(128, std::min<int64_t>(kSpreadCap, p->nnz / ((int64_t)p->sm_count * 4)));
    std::vector<int4> pcs;
    std::vector<int> ext;
    make_spread_pieces(p, cap, pcs, ext);
    const int64_t np = (int64_t)pcs.size();
    int cells = 0;
    for (int e : ext) cells = std::max(cells, e * slab_cells(g));
    const size_t smem = build_smem(g, cells);
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
            return fail(NUFFT3D_ERR_NOMEM, std::string("stored H': ") + cudaGetErrorString(e));
        }
        b.ptrs.push_back(*ptr);
        return NUFFT3D_SUCCESS;
    };
    auto none = [&](int st) {  // the spread evaluates the kernel instead
        if (mode > 0) return st;
        clear_error();
        return (int)NUFFT3D_SUCCESS;
    };
    std::vector<int> starts(p->slab_counts.size() + 1, 0);
    for (size_t i = 0; i < p->slab_counts.size(); ++i) starts[i + 1] = starts[i] + p->slab_counts[i];
    int4 *pieces = nullptr;
    int *dext = nullptr, *dstart = nullptr;
    uint2 *dl = nullptr, *wst = nullptr;
    uint32_t *dseg = nullptr;
    int st = alloc(&pieces, (size_t)np, keep);
    if (st == NUFFT3D_SUCCESS) st = alloc(&wst, (size_t)np * (kBundleWarps + 1), keep);
    if (st == NUFFT3D_SUCCESS) st = alloc(&dext, (size_t)np, tmp);
    if (st == NUFFT3D_SUCCESS) st = alloc(&dstart, starts.size(), tmp);
    if (st == NUFFT3D_SUCCESS) st = alloc(&dl, (size_t)np, tmp);
    if (st == NUFFT3D_SUCCESS) st = alloc(&dseg, (size_t)np, tmp);
    if (st != NUFFT3D_SUCCESS) return none(st);
    NUFFT_CUDA_TRY(cudaMemcpyAsync(pieces, pcs.data(), sizeof(int4) * np, cudaMemcpyHostToDevice, s));
    NUFFT_CUDA_TRY(cudaMemcpyAsync(dext, ext.data(), sizeof(int) * np, cudaMemcpyHostToDevice, s));
    NUFFT_CUDA_TRY(cudaMemcpyAsync(dstart, starts.data(), sizeof(int) * starts.size(), cudaMemcpyHostToDevice, s));
    const SpreadBuild sb{pieces, dseg, dext, dstart, p->samples, g, p->kb, slab_cells(g), slabs_per_tile(g)};
    k_spread_tab_build<false><<<(unsigned)np, kTabBuildThreads, smem, s>>>(sb, dl, nullptr, nullptr, nullptr, nullptr,
                                                                           nullptr);
    NUFFT_CUDA_TRY(cudaGetLastError());
    std::vector<uint2> nl((size_t)np);
    NUFFT_CUDA_TRY(cudaMemcpyAsync(nl.data(), dl, sizeof(uint2) * np, cudaMemcpyDeviceToHost, s));
    NUFFT_CUDA_TRY(cudaStreamSynchronize(s));
    uint64_t total = 0, segs = 0;  // steps, segments
    std::vector<uint32_t> seg0((size_t)np);
    for (int64_t b = 0; b < np; ++b) {
        pcs[(size_t)b].z = (int)(uint32_t)total;
        seg0[(size_t)b] = (uint32_t)segs;
        total += nl[(size_t)b].x;
        segs += nl[(size_t)b].y;
        if ((total + 1) * kBundleDepth >= 0xffffffffull)  // line indices are 32-bit
            return none(fail(NUFFT3D_ERR_SIZE, "too many entries for the stored H'"));
    }
    const size_t lines = (size_t)(total + 1) * kBundleDepth;  // a spare step for the pipeline's overrun
    const size_t sbytes = (size_t)(segs + 1) * (kRows * sizeof(int4) + sizeof(uint16_t));
    const size_t bytes = lines * kLineBytes, wbytes = sbytes + sizeof(uint2) * (size_t)np * (kBundleWarps + 1);
    if (mode < 0) {
        size_t fr = 0, to = 0;
        if (cudaMemGetInfo(&fr, &to) != cudaSuccess || bytes + wbytes > fr / 2) {
            cudaGetLastError();
            return NUFFT3D_SUCCESS;  // the spread evaluates the kernel instead
        }
    }
    float4 *ent = nullptr;
    uint16_t *idx = nullptr, *steps = nullptr;
    int4 *pts = nullptr;
    st = alloc(&ent, lines * kRows, keep);
    if (st == NUFFT3D_SUCCESS) st = alloc(&idx, lines * kRows, keep);
    if (st == NUFFT3D_SUCCESS) st = alloc(&pts, (size_t)(segs + 1) * kRows, keep);
    if (st == NUFFT3D_SUCCESS) st = alloc(&steps, (size_t)segs + 1, keep);
    if (st != NUFFT3D_SUCCESS) return none(st);
    NUFFT_CUDA_TRY(cudaMemsetAsync(ent + (size_t)total * kBundleDepth * kRows, 0, kBundleDepth * kRows * sizeof(float4), s));
    NUFFT_CUDA_TRY(cudaMemsetAsync(idx + (size_t)total * kBundleDepth * kRows, 0, kBundleDepth * kRows * sizeof(uint16_t), s));
    NUFFT_CUDA_TRY(cudaMemsetAsync(steps + segs, 0, sizeof(uint16_t), s));
    NUFFT_CUDA_TRY(cudaMemcpyAsync(dseg, seg0.data(), sizeof(uint32_t) * np, cudaMemcpyHostToDevice, s));
    NUFFT_CUDA_TRY(cudaMemcpyAsync(pieces, pcs.data(), sizeof(int4) * np, cudaMemcpyHostToDevice, s));
    k_spread_tab_build<true><<<(unsigned)np, kTabBuildThreads, smem, s>>>(sb, nullptr, wst, ent, idx, pts, steps);
    NUFFT_CUDA_TRY(cudaGetLastError());
    NUFFT_CUDA_TRY(cudaStreamSynchronize(s));
    p->spread_ent = ent;
    p->spread_idx = idx;
    p->spread_pts = pts;
    p->spread_steps = steps;
    p->spread_pieces = pieces;
    p->spread_wstart = wst;
    p->n_spread_pieces = np;
    p->spread_cap = 0;
    for (auto &pc : pcs) p->spread_cap = std::max(p->spread_cap, piece_count(pc));
    p->spread_bytes = (int64_t)(bytes + wbytes + sizeof(int4) * np);
    p->table_bytes += p->spread_bytes;
    keep.ptrs.clear();
    return NUFFT3D_SUCCESS;
}

}  // namespace nufft3d
