// deposit.cu -- CIC mass assignment (the GPU counterpart of fieldize.cpp:46-113).
//
// A deposit pass over n particles sorts them into cell tiles and then
// accumulates one tile per CTA in shared memory:
//
//   k_bin_sort        up to 8192 tiles (a binned pass): each CTA sorts chunks of
//                     up to 12288 consecutive particles by tile in shared
//                     memory -- cell (two-product split, split_q28), shared
//                     counters, a scan, the packed records (tile-local cell +
//                     28-bit fraction per axis + mass bits) to their places --
//                     and writes the chunk's records and its header of tile
//                     offsets.  Positions are read from memory once.
//   k_sort_hist,      more tiles (a counting sort over the pass): tile counts,
//   k_sort_scatter    scanned by the last CTA, then every record to a slot of
//                     its tile's range.  (Grids with more tiles than a shared
//                     histogram holds count and claim in global memory.)
//   k_tile_deposit    one CTA per tile: each particle adds its eight CIC
//                     weights, rounded to integers of 2^-s mass units, to a
//                     (T+1)^3 block of 64-bit shared accumulators.  Integer
//                     sums are exact and independent of order, so the deposit
//                     is bit-reproducible.  Cells strictly inside the tile are
//                     final: (sum - mean) is converted to FP32 once and stored.
//                     The tile's low faces and its +1 halo layer go to scratch
//                     as 64-bit sums.
//   k_face_gather     per tile: every low-face cell adds the halo sums the
//                     (up to 7) lower neighbours hold for it, in a fixed order,
//                     and stores (sum - mean) as FP32; it also ends the pass
//                     (corner mode, running sums).
//
// The line between the two sorts is where a chunk's counters and its staging
// area fill an SM's shared memory.  On both sides of it, ms of the sort and tile
// kernels, uniform random particles: binned against the earlier counting sort
// 0.55 and 0.98 (27 M on 256^3, 4096 tiles), 0.066 and 0.098 (2.1 M on 128^3,
// 512 tiles); the counting sort 1.06 (30 M on 384^3, 13824 tiles; 1.43 before).
//
// A grouped pass runs the same kernels once for several boxes of one grid size
// (a batch of uneven boxes): the sort CTAs are shared out over the boxes'
// particles, the tile kernels take the box from their grid.  Record slots are
// global across the boxes (box b's begin at its first record).
//
// No global float atomics are involved and no grid memset is needed: every real
// cell is written exactly once per pass.  Subtracting the pass mean (in fixed
// point, before the single rounding) keeps the FP32 r2c accurate; it changes
// only the excluded k = 0 mode.  The mean is rounded to 24 significant bits so
// that an empty cell holds exactly -mean in FP32 and reads back as exactly 0.
#include "bulk.cuh"
#include "common.cuh"
#include "internal.h"
#include "launch.cuh"

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <utility>

namespace genpk {

cudaError_t ensure_dynamic_smem(const void *func, size_t bytes)
{
    // the limit is kept per device (a process may drive several GPUs)
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess)
        return err;
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, size_t> limit;
    std::lock_guard<std::mutex> lock(mu);
    size_t &cur = limit[std::make_pair(dev, func)];
    if (bytes <= cur)
        return cudaSuccess;
    err = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (err == cudaSuccess)
        cur = bytes;
    return err;
}

GridGeom make_grid_geom(int dims)
{
    GridGeom g;
    g.dims = dims;
    g.half = dims / 2;
    g.hc = dims / 2 + 1;
    g.row = 2 * g.hc;
    g.plane = (int64_t)g.row * dims;
    g.nfloat = g.plane * dims;
    return g;
}

namespace {

struct SortParams {
    const float *pos;
    const float *masses;
    int64_t n;
    int dims;
    int ctas;        // sort CTAs of this box: CTA k takes chunks k, k + ctas, ...
    float uh, ul;
    int lx, ly, lz;  // log2 of the tile edges
    int nty, ntz;
    int ntiles;
    float umass;     // uniform mass when masses == nullptr
    int corner;      // accumulate the exact (N/2,N/2,N/2) mode (even grids)
};

// Where a sort CTA's particles come from: the one box of a pass, or the boxes
// of a grouped pass (CTAs [cta0[b], cta0[b+1]) read box b).  Both are passed
// by value in the kernel parameters.
struct OneBox {
    SortParams p;
    __device__ __forceinline__ int box_of(int) const { return 0; }
    __device__ __forceinline__ SortParams params(int) const { return p; }
    __device__ __forceinline__ int first_cta(int) const { return 0; }
};

struct BoxGroup {
    int nbox;
    int cta0[kMaxGroupBoxes + 1];
    SortParams p[kMaxGroupBoxes];
    __device__ __forceinline__ int box_of(int blk) const
    {
        int b = 0;
        while (b + 1 < nbox && blk >= cta0[b + 1])
            b++;
        return b;
    }
    __device__ __forceinline__ SortParams params(int b) const { return p[b]; }
    __device__ __forceinline__ int first_cta(int b) const { return cta0[b]; }
};

// What the scan at the end of the histogram kernel needs per box: the first
// sort CTA (its mass partials), mass kind, uniform mass and first record.
struct ScanBoxes {
    int first[kMaxGroupBoxes + 1];
    int var[kMaxGroupBoxes];  // the particles carry masses
    double umass[kMaxGroupBoxes];
    long long rec0[kMaxGroupBoxes];
};

// The scatter's cursors lie a 128-byte line apart (a word apart where the
// tiles are too many for that): atomics on one line queue in one L2 slice.
constexpr int kCursorStride = 32;

struct ScanOut {
    uint32_t *totals;      // [ntiles] per box; zero between passes
    uint32_t *tile_start;  // [ntiles + 1] per box
    uint32_t *cursor;      // [ntiles] per box: the scatter's next free slot per tile
    int cursor_stride;     // words between them
    uint32_t *ticket;      // one per box; zero between passes
    double *mass_part;     // [sort CTAs]
    double inv_cells;
    bool clean;
    double *field_mass, *field_sub;
};

// Sort CTAs walk chunks of kSortChunk consecutive particles, kSortUnroll per
// thread (thread t takes base + t + kSortThreads * u: coalesced).
constexpr int kSortThreads = kSortChunkParticles / 8;
constexpr int kSortUnroll = 8;
constexpr uint32_t kNoTile = 0xffffffffu;

// A particle outside the fast split's range: the general split, and the test
// for particles that must be skipped (false).
__device__ __noinline__ bool split3_general(float x, float y, float z, float uh, float ul, int dims,
                                            AxisQ *a)
{
    if (!finite3(x, y, z))
        return false;
    const float lim = 1.0e9f;
    if (fabsf(x * uh) > lim || fabsf(y * uh) > lim || fabsf(z * uh) > lim)
        return false;
    a[0] = split_q28(x, uh, ul, dims);
    a[1] = split_q28(y, uh, ul, dims);
    a[2] = split_q28(z, uh, ul, dims);
    return true;
}

// Cell, 28-bit fraction and tile of one particle (split_q28, as the window
// engine splits it); kNoTile for a particle that must be skipped.
template <bool CORNER>
__device__ __forceinline__ uint32_t particle_cell(const SortParams &p, float x, float y, float z,
                                                  float m, AxisQ a[3])
{
    bool ok = split3_fast<CORNER>(x, y, z, p.uh, p.ul, p.dims, a);
    if (!ok) {
        AxisQ b[3];
        ok = split3_general(x, y, z, p.uh, p.ul, p.dims, b);
        a[0] = b[0];
        a[1] = b[1];
        a[2] = b[2];
    }
    if (!ok || !(fabsf(m) <= 3.4028235e38f))
        return kNoTile;
    return ((uint32_t)(a[0].cell >> p.lx) * (uint32_t)p.nty + (uint32_t)(a[1].cell >> p.ly)) *
               (uint32_t)p.ntz +
           (uint32_t)(a[2].cell >> p.lz);
}

// Per-CTA mass sum (FP64) and max |mass| (float bits) after the particle loop.
__device__ __forceinline__ void block_mass(float msum, float mc, float mmax, double *mass_part,
                                           DeviceStatus *st)
{
    __shared__ double sh_mass[32];
    __shared__ float sh_max[32];
    double md = warp_sum_d((double)msum - (double)mc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        mmax = fmaxf(mmax, __shfl_xor_sync(0xffffffffu, mmax, o));
    if ((threadIdx.x & 31) == 0) {
        sh_mass[threadIdx.x >> 5] = md;
        sh_max[threadIdx.x >> 5] = mmax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        float mx = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            s += sh_mass[w];
            mx = fmaxf(mx, sh_max[w]);
        }
        mass_part[blockIdx.x] = s;
        if (mx > 0.f)
            atomicMax(&st->max_mass_bits, __float_as_uint(mx));
    }
}

// True when some lane's tile equals the previous lane's (a run of particles in
// one tile, as spatially ordered input gives).  Without one, the lanes take
// their tile slots with one shared atomic each: __match_any_sync over 32
// distinct tiles (random order, the sorted engine's usual input) costs more
// than it merges.  Slots within a tile may then come in any order; the tile
// sums are exact integers, so the grid does not depend on it.
__device__ __forceinline__ bool warp_has_tile_runs(uint32_t t)
{
    const int lane = threadIdx.x & 31;
    const uint32_t prev = __shfl_up_sync(0xffffffffu, t, 1);
    return __any_sync(0xffffffffu, lane > 0 && t != kNoTile && t == prev);
}

// One slot of counts[t] per lane with a tile; lanes of one tile share an
// atomic where the order has runs.
__device__ __forceinline__ uint32_t claim_slot(uint32_t *counts, uint32_t t)
{
    uint32_t slot = 0;
    if (!warp_has_tile_runs(t)) {
        if (t != kNoTile)
            slot = atomicAdd(&counts[t], 1u);
    } else {
        const int lane = threadIdx.x & 31;
        const unsigned peers = __match_any_sync(0xffffffffu, t);
        const int leader = __ffs(peers) - 1;
        uint32_t slot0 = 0;
        if (t != kNoTile && lane == leader)
            slot0 = atomicAdd(&counts[t], (uint32_t)__popc(peers));
        slot = __shfl_sync(0xffffffffu, slot0, leader) + __popc(peers & ((1u << lane) - 1u));
    }
    return slot;
}

struct Pos3 {
    float x, y, z;
};

// kSortUnroll / 2 particles of a chunk, their loads in flight together.
__device__ __forceinline__ void load_half(const SortParams &p, int64_t i0, Pos3 (&v)[kSortUnroll / 2])
{
#pragma unroll
    for (int u = 0; u < kSortUnroll / 2; u++) {
        const int64_t i = i0 + kSortThreads * u;
        v[u] = Pos3{0.f, 0.f, 0.f};
        if (i < p.n) {
            v[u].x = __ldg(p.pos + 3 * i);
            v[u].y = __ldg(p.pos + 3 * i + 1);
            v[u].z = __ldg(p.pos + 3 * i + 2);
        }
    }
}

// A pass's constants into the status words and the grid's running sums, by one
// thread.
__device__ __forceinline__ void store_pass_consts(const PassConsts &k, bool clean,
                                                  double *field_mass, double *field_sub,
                                                  DeviceStatus *st)
{
    st->pass_mass = k.mass;
    st->fx_shift = k.fx_shift;
    st->mean_fixed = k.mean_fixed;
    add_pass_sums(k, clean, field_mass, field_sub);
}

// Exclusive scan of box `box`'s tile totals and its per-pass constants, by the
// box's last sort CTA.  A box's tile starts begin at its first record.  Unless
// the box's particles carry masses, every one weighs its uniform mass (of
// either sign).  The totals and the ticket are zero again afterwards.
__device__ __forceinline__ void scan_box(const ScanOut &o, const ScanBoxes &boxes, int box,
                                         int ntiles, DeviceStatus *st)
{
    constexpr int kWarps = kSortThreads / 32;
    constexpr int kItems = 8;  // tiles per thread and round
    __shared__ uint32_t warp_tot[kWarps];
    __shared__ double sh_m[kWarps];
    const uint32_t rec0 = (uint32_t)boxes.rec0[box];
    uint32_t *totals = o.totals + (size_t)box * ntiles;
    uint32_t *start = o.tile_start + (size_t)box * (ntiles + 1);
    uint32_t *cursor = o.cursor + (size_t)box * ntiles * o.cursor_stride;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t carry = rec0;
    for (int base = 0; base < ntiles; base += kSortThreads * kItems) {
        const int t0 = base + threadIdx.x * kItems;
        uint32_t v[kItems], sum = 0;
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            v[k] = t0 + k < ntiles ? __ldcg(totals + t0 + k) : 0u;
            sum += v[k];
        }
        uint32_t x = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d)
                x += y;
        }
        if (lane == 31)
            warp_tot[wid] = x;
        __syncthreads();
        uint32_t before = carry, all = 0;
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            const uint32_t y = warp_tot[w];
            before += w < wid ? y : 0u;
            all += y;
        }
        uint32_t run = before + x - sum;
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            if (t0 + k < ntiles) {
                start[t0 + k] = run;
                cursor[(size_t)(t0 + k) * o.cursor_stride] = run;
                totals[t0 + k] = 0u;
            }
            run += v[k];
        }
        carry += all;
        __syncthreads();
    }
    double m = 0.0;
    if (boxes.var[box]) {
        const int first = boxes.first[box], nsort = boxes.first[box + 1] - first;
        for (int c = threadIdx.x; c < nsort; c += blockDim.x)
            m += __ldcg(o.mass_part + first + c);
        m = warp_sum_d(m);
        if (lane == 0)
            sh_m[wid] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int w = 0; w < kWarps; w++)
                s += sh_m[w];
            m = s;
        }
    } else {
        m = (double)(carry - rec0) * boxes.umass[box];
    }
    if (threadIdx.x == 0) {
        start[ntiles] = carry;
        const float mref = !boxes.var[box] ? (float)fabs(boxes.umass[box])
                                           : __uint_as_float(__ldcg(&st->max_mass_bits));
        st->max_mass_bits = 0u;  // read: zero again for the next pass
        store_pass_consts(pass_consts(m, mref, o.inv_cells), o.clean, o.field_mass + box,
                          o.field_sub + box, st);
        o.ticket[box] = 0u;
    }
}

// Tile counts of every particle, summed per CTA in a shared histogram and
// added to the box's totals (GLOBAL = false), or counted straight into the
// totals (GLOBAL = true, for grids with more tiles than a shared histogram
// holds).  The last CTA of a box to finish scans its totals (scan_box), so the
// counts, the tile starts and the pass constants take one launch.
template <bool GLOBAL, class Src>
__global__ void __launch_bounds__(kSortThreads)
    k_sort_hist(const __grid_constant__ Src src, const __grid_constant__ ScanOut out,
                const __grid_constant__ ScanBoxes boxes, DeviceStatus *st)
{
    extern __shared__ uint32_t sh_hist[];
    __shared__ int last;
    const int box = src.box_of(blockIdx.x);
    const SortParams p = src.params(box);
    const int cta = blockIdx.x - src.first_cta(box);
    st += box;
    uint32_t *totals = out.totals + (size_t)box * p.ntiles;
    if (!GLOBAL) {
        for (int i = threadIdx.x; i < p.ntiles; i += blockDim.x)
            sh_hist[i] = 0u;
        __syncthreads();
    }
    uint32_t *counts = GLOBAL ? totals : sh_hist;
    wait_previous();
    float msum = 0.f, mc = 0.f, mmax = 0.f;
    unsigned bad = 0;
    for (int64_t c0 = (int64_t)cta * kSortChunkParticles; c0 < p.n;
         c0 += (int64_t)p.ctas * kSortChunkParticles) {
#pragma unroll 1
        for (int half = 0; half < 2; half++) {
            const int64_t i0 = c0 + half * (kSortChunkParticles / 2) + threadIdx.x;
            Pos3 v[kSortUnroll / 2];
            load_half(p, i0, v);
#pragma unroll
            for (int u = 0; u < kSortUnroll / 2; u++) {
                const int64_t i = i0 + kSortThreads * u;
                uint32_t t = kNoTile;
                if (i < p.n) {
                    AxisQ a[3];
                    const float m = p.masses ? __ldg(p.masses + i) : 0.f;
                    t = particle_cell<false>(p, v[u].x, v[u].y, v[u].z, m, a);
                    if (t == kNoTile) {
                        bad++;
                    } else if (p.masses) {
                        const float y = m - mc;  // Kahan-compensated FP32 sum of masses
                        const float s = msum + y;
                        mc = (s - msum) - y;
                        msum = s;
                        mmax = fmaxf(mmax, fabsf(m));
                    }
                }
                if (!warp_has_tile_runs(t)) {
                    if (t != kNoTile)
                        atomicAdd(&counts[t], 1u);
                } else {
                    const unsigned peers = __match_any_sync(0xffffffffu, t);
                    if (t != kNoTile && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
                        atomicAdd(&counts[t], (uint32_t)__popc(peers));
                }
            }
        }
    }
    __syncthreads();
    if (!GLOBAL) {
        for (int i = threadIdx.x; i < p.ntiles; i += blockDim.x) {
            const uint32_t v = sh_hist[i];
            if (v)
                atomicAdd(totals + i, v);
        }
    }
    if (p.masses)
        block_mass(msum, mc, mmax, out.mass_part, st);
    if (bad)
        atomicAdd(&st->bad_particles, (unsigned long long)bad);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        last = atomicAdd(out.ticket + box, 1u) == (uint32_t)p.ctas - 1u;
    __syncthreads();
    if (last) {
        __threadfence();
        scan_box(out, boxes, box, p.ntiles, st);
    }
}

// ---- binned passes: chunks sorted in shared memory ---------------------------

constexpr int kBinThreads = 1024;
constexpr int kBinPer = 12;                      // particles per thread and chunk, at most
constexpr int kBinMax = kBinThreads * kBinPer;   // 12288: a 192 KB staging area
constexpr int kBinMaxTiles = 8192;               // 32 KB of counters beside it

struct BinBox {
    SortParams s;
    int len;        // particles per chunk (a multiple of kBinThreads)
    int nchunks;
    uint32_t rec0;  // the box's first record
    uint32_t hdr0;  // the box's first header row
};

struct OneBin {
    BinBox b;
    __device__ __forceinline__ int box_of(int) const { return 0; }
    __device__ __forceinline__ const BinBox &box(int) const { return b; }
    __device__ __forceinline__ int first_cta(int) const { return 0; }
};

struct BinGroup {
    int nbox;
    int cta0[kMaxGroupBoxes + 1];
    BinBox b[kMaxGroupBoxes];
    __device__ __forceinline__ int box_of(int blk) const
    {
        int k = 0;
        while (k + 1 < nbox && blk >= cta0[k + 1])
            k++;
        return k;
    }
    __device__ __forceinline__ const BinBox &box(int k) const { return b[k]; }
    __device__ __forceinline__ int first_cta(int k) const { return cta0[k]; }
};

struct BinOut {
    uint4 *sorted;
    uint16_t *hdr;        // [chunk][stride]: a chunk's records of tile t are [hdr[t], hdr[t+1])
    int stride;
    double *mass_part;    // per sort CTA: the mass of its particles (boxes with masses)
    double *corner_part;  // per sort CTA: its share of the corner mode (over a uniform mass)
    uint32_t *ticket;     // one per box; zero between passes
    double inv_cells;
    bool clean;
    double *field_mass, *field_sub;
};

__device__ __forceinline__ void bulk_store(void *dst, const void *src, unsigned bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"(smem_addr(src)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// Sum over the CTA of one double per thread, in a fixed order (the result in
// warp 0).  sh: one double per warp.
__device__ __forceinline__ double block_sum_d(double v, double *sh)
{
    v = warp_sum_d(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32)
        v = warp_sum_d(threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0);
    return v;
}

// Packed particle: per axis (tile-local cell << 28) | 28-bit fraction (tiles
// of at most 16 cells per edge), then the mass bits.
__device__ __forceinline__ uint32_t pack_axis(const AxisQ &a, uint32_t mask)
{
    return (((uint32_t)a.cell & mask) << kFracBits) | a.q;
}

// A binned pass's first kernel.  A CTA takes a chunk of up to 12288 consecutive
// particles at a time and sorts its records by tile in shared memory:
//   1. every particle's tile, and its rank within (chunk, tile) from a shared
//      counter;
//   2. an exclusive scan of the counters: the tiles' places within the chunk,
//      also written out as the chunk's header row (16-bit offsets);
//   3. the particles again (from the L2), split in full: the packed record goes
//      to its place in the staging area, and its corner-mode term into a sum;
//   4. one bulk copy of the staging area to the chunk's record range.
// The records thus leave in whole lines, and no pass-wide counts are needed
// first: positions come from memory once, against twice for a counting sort
// over the whole pass, whose 16-byte records went to memory in pieces besides
// (644 MB read and 655 MB written for 432 MB of records; 27 M particles on 256^3).
// The tile kernels then read, per tile, its run in every chunk.  A box whose
// particles carry masses gets its pass constants from its last CTA to finish; a
// uniform mass's come from the host.
//
// The corner mode k = (N/2, N/2, N/2) of the CIC density (even grids) is summed
// exactly: that DFT coefficient is sum over particles of
// m (-1)^(x+y+z) prod_a (1 - 2 d_a) with (x, y, z) the particle's cell and d_a
// its fractions.  Each term is formed from the full two-product position in
// float-pair arithmetic and summed per thread in float pairs (a uniform mass
// factored out, others scaled to the chunk's largest), per CTA in FP64, and
// over the CTAs by the face kernel, in a fixed order.  The last log-k bin holds only this mode, so its value must not carry
// the FP32 grid's rounding noise.
template <class Src>
__global__ void __launch_bounds__(kBinThreads, 1)
    k_bin_sort(const __grid_constant__ Src src, const __grid_constant__ BinOut out, int stage_len,
               DeviceStatus *st)
{
    extern __shared__ __align__(128) unsigned char bin_smem[];
    uint4 *stage = reinterpret_cast<uint4 *>(bin_smem);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(stage + stage_len);  // [ntiles rounded up to 4]
    __shared__ uint32_t warp_tot[kBinThreads / 32];
    __shared__ double sh_d[kBinThreads / 32];
    __shared__ uint32_t chunk_max;  // |mass| as float bits
    __shared__ int last;
    const int box = src.box_of(blockIdx.x);
    const BinBox &bb = src.box(box);
    const SortParams p = bb.s;
    const int cta = blockIdx.x - src.first_cta(box);
    st += box;
    const uint32_t mx = (1u << p.lx) - 1u, my = (1u << p.ly) - 1u, mz = (1u << p.lz) - 1u;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nt4 = (p.ntiles + 3) >> 2;
    const bool var = p.masses != nullptr;
    wait_previous();

    f2sum alt = {0.f, 0.f};
    double corner = 0.0;
    float msum = 0.f, mc = 0.f;  // Kahan-compensated sum of this thread's masses
    uint32_t mmax = 0u, bad = 0u;
    for (int c = cta; c < bb.nchunks; c += p.ctas) {
        const int64_t first = (int64_t)c * bb.len;
        const int len = (int)min((int64_t)bb.len, p.n - first);
        for (int i = threadIdx.x; i < nt4; i += kBinThreads)
            reinterpret_cast<uint4 *>(cnt)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (threadIdx.x == 0)
            chunk_max = 0u;
        __syncthreads();

        uint32_t key[kBinPer];  // tile << 14 | rank
        uint32_t cmax = 0u;     // this thread's largest |mass| of the chunk
#pragma unroll
        for (int q = 0; q < kBinPer; q += 4) {
            if (q * kBinThreads < len) {
                Pos3 v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int j = threadIdx.x + kBinThreads * (q + u);
                    v[u] = Pos3{0.f, 0.f, 0.f};
                    if (j < len) {
                        const float *s = p.pos + 3 * (first + j);
                        v[u] = Pos3{__ldg(s), __ldg(s + 1), __ldg(s + 2)};
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int j = threadIdx.x + kBinThreads * (q + u);
                    uint32_t t = kNoTile;
                    if (j < len) {
                        AxisQ a[3];
                        const float m = var ? __ldg(p.masses + first + j) : 0.f;
                        t = particle_cell<false>(p, v[u].x, v[u].y, v[u].z, m, a);
                        if (t == kNoTile) {
                            bad++;
                        } else if (var) {
                            const float y = m - mc;
                            const float s = msum + y;
                            mc = (s - msum) - y;
                            msum = s;
                            cmax = max(cmax, __float_as_uint(fabsf(m)));
                        }
                    }
                    const uint32_t r = claim_slot(cnt, t);
                    key[q + u] = t == kNoTile ? kNoTile : (t << 14) | r;
                }
            } else {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    key[q + u] = kNoTile;
            }
        }
        if (var) {
            cmax = __reduce_max_sync(0xffffffffu, cmax);
            if (lane == 0)
                atomicMax(&chunk_max, cmax);
            mmax = max(mmax, cmax);
        }
        __syncthreads();

        // exclusive scan of the counters, four per thread and round; the
        // chunk's header row
        uint16_t *hdr = out.hdr + (size_t)(bb.hdr0 + (uint32_t)c) * (size_t)out.stride;
        uint32_t carry = 0u;
        for (int b0 = 0; b0 < nt4; b0 += kBinThreads) {
            const int i = b0 + threadIdx.x;
            uint4 v = i < nt4 ? reinterpret_cast<uint4 *>(cnt)[i] : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t sum = v.x + v.y + v.z + v.w;
            uint32_t x = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d)
                    x += y;
            }
            if (lane == 31)
                warp_tot[wid] = x;
            __syncthreads();
            const uint32_t w = warp_tot[lane];
            const uint32_t before = __reduce_add_sync(0xffffffffu, lane < wid ? w : 0u);
            const uint32_t all = __reduce_add_sync(0xffffffffu, w);
            const uint32_t e = carry + before + x - sum;
            if (i < nt4) {
                const uint4 o = make_uint4(e, e + v.x, e + v.x + v.y, e + v.x + v.y + v.z);
                reinterpret_cast<uint4 *>(cnt)[i] = o;
                reinterpret_cast<ushort4 *>(hdr)[i] =
                    make_ushort4((unsigned short)o.x, (unsigned short)o.y, (unsigned short)o.z,
                                 (unsigned short)o.w);
            }
            carry += all;
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            hdr[p.ntiles] = (uint16_t)carry;
            // the previous chunk's records have left the staging area
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
        __syncthreads();

        // (a mass of the chunk's largest exponent scales into [2^27, 2^28))
        const int ce = (int)(chunk_max >> 23);
        const int cs = max(-126, min(127, 154 - ce));
        const float mscale = __uint_as_float((uint32_t)(127 + cs) << 23);
#pragma unroll
        for (int q = 0; q < kBinPer; q += 4) {
            if (q * kBinThreads >= len)
                break;
            Pos3 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float *s = p.pos + 3 * (first + threadIdx.x + kBinThreads * (q + u));
                v[u] = Pos3{0.f, 0.f, 0.f};
                if (key[q + u] != kNoTile)
                    v[u] = Pos3{__ldg(s), __ldg(s + 1), __ldg(s + 2)};
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (key[q + u] == kNoTile)
                    continue;
                const int64_t i = first + threadIdx.x + kBinThreads * (q + u);
                AxisQ a[3];
                const float m = var ? __ldg(p.masses + i) : p.umass;
                particle_cell<true>(p, v[u].x, v[u].y, v[u].z, m, a);
                if (p.corner) {
                    f2sum w = corner_factor_q(a[0], a[1], a[2]);
                    if (var) {
                        const float mm = m * mscale;
                        const float h = __fmul_rn(w.hi, mm);
                        w = f2sum{h, fmaf(w.hi, mm, -h) + w.lo * mm};
                    }
                    f2_accumulate(alt, f2_signed(w, a[0].cell ^ a[1].cell ^ a[2].cell));
                }
                stage[cnt[key[q + u] >> 14] + (key[q + u] & 0x3fffu)] =
                    make_uint4(pack_axis(a[0], mx), pack_axis(a[1], my), pack_axis(a[2], mz),
                               __float_as_uint(m));
            }
        }
        if (var) {  // this chunk's share, out of its scale
            corner += ((double)alt.hi + (double)alt.lo) *
                      __longlong_as_double((long long)(1023 - cs) << 52);
            alt = f2sum{0.f, 0.f};
        }
        fence_proxy_async();
        __syncthreads();
        if (threadIdx.x == 0 && carry > 0u)
            bulk_store(out.sorted + bb.rec0 + (uint32_t)first, stage, carry * 16u);
    }
    if (!var)
        corner = (double)alt.hi + (double)alt.lo;

    corner = block_sum_d(corner, sh_d);
    if (threadIdx.x == 0)
        out.corner_part[blockIdx.x] = corner;
    bad = __reduce_add_sync(0xffffffffu, bad);
    if (lane == 0 && bad) {
        atomicAdd(&st->bad_particles, (unsigned long long)bad);
        atomicAdd(&st->pass_bad, (unsigned long long)bad);
    }
    if (!var) {
        if (threadIdx.x == 0)  // the staging area must outlive its copies
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        return;
    }
    // The CTA's mass; the last CTA of the box adds the masses up in order.
    const double part = block_sum_d((double)msum - (double)mc, sh_d);
    if (threadIdx.x == 0)
        out.mass_part[blockIdx.x] = part;
    if (lane == 0 && mmax)
        atomicMax(&st->max_mass_bits, mmax);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(out.ticket + box, 1u) == (uint32_t)p.ctas - 1u;
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (!last)
        return;
    __threadfence();
    double m = 0.0;
    for (int c = threadIdx.x; c < p.ctas; c += kBinThreads)
        m += __ldcg(out.mass_part + src.first_cta(box) + c);
    m = block_sum_d(m, sh_d);
    if (threadIdx.x == 0) {
        const float mref = __uint_as_float(__ldcg(&st->max_mass_bits));
        st->max_mass_bits = 0u;  // read: zero again for the next pass
        store_pass_consts(pass_consts(m, mref, out.inv_cells), out.clean, out.field_mass + box,
                          out.field_sub + box, st);
        out.ticket[box] = 0u;
    }
}

// Writes every particle's packed record to a slot of its tile's range.  A CTA
// takes a chunk at a time: its particles claim ranks within (chunk, tile) in a
// shared histogram, the first of each tile claims that many slots of the tile
// with one global atomic on the tile's cursor, and all write their records at
// once (GLOBAL = true: every particle claims its slot from the cursor itself).
// All CTAs thus fill the same tiles' ranges front to back together, so that a
// 128-byte line of eight records is completed while it is still in the L2;
// with a range of its own per (CTA, tile) each line waited for one CTA to come
// by eight times and went to memory in pieces (644 MB read and 655 MB written
// for 432 MB of records, 27 M particles on 256^3).
//
// On even grids it also sums the corner mode k = (N/2, N/2, N/2) of the CIC
// density exactly: that DFT coefficient is sum over particles of
// m (-1)^(x+y+z) prod_a (1 - 2 d_a) with (x, y, z) the particle's cell and d_a
// its fractions.  Each term is formed from the full two-product position in
// float-pair arithmetic and summed per thread in float pairs; each warp's total
// is rounded to an integer of 2^-(s+4) mass units and summed in 64-bit integers
// (deterministic: fixed per-thread order, integer sums across warps).  The last log-k bin holds only
// this mode, so its value must not carry the FP32 grid's rounding noise.
template <bool GLOBAL, class Src>
__global__ void __launch_bounds__(kSortThreads, 2)
    k_sort_scatter(const __grid_constant__ Src src, uint32_t *__restrict__ cursor,
                   uint4 *__restrict__ sorted, DeviceStatus *st)
{
    extern __shared__ uint32_t sh_cur[];
    const int box = src.box_of(blockIdx.x);
    const SortParams p = src.params(box);
    const int cta = blockIdx.x - src.first_cta(box);
    st += box;
    constexpr int kStride = GLOBAL ? 1 : kCursorStride;
    cursor += (size_t)box * p.ntiles * kStride;
    if (!GLOBAL) {
        for (int i = threadIdx.x; i < p.ntiles; i += blockDim.x)
            sh_cur[i] = 0u;
        __syncthreads();
    }
    const uint32_t mx = (1u << p.lx) - 1u, my = (1u << p.ly) - 1u, mz = (1u << p.lz) - 1u;
    const int lane = threadIdx.x & 31;
    wait_previous();
    cursor = fresh(cursor);
    st = fresh(st);
    // Corner terms in 2^-(s+4) mass units (|term| < 2^32), summed per thread as
    // a float pair and converted to an integer once per warp.
    const float mscale = ldexpf(1.f, st->fx_shift + 4);
    f2sum alt = {0.f, 0.f};
    for (int64_t c0 = (int64_t)cta * kSortChunkParticles; c0 < p.n;
         c0 += (int64_t)p.ctas * kSortChunkParticles) {
        uint32_t wx[kSortUnroll], wy[kSortUnroll], wz[kSortUnroll];
        uint32_t key[kSortUnroll];  // tile << 13 | rank, or the slot (GLOBAL); kNoTile
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int64_t i0 = c0 + half * (kSortChunkParticles / 2) + threadIdx.x;
            Pos3 v[kSortUnroll / 2];
            load_half(p, i0, v);
#pragma unroll
            for (int u = 0; u < kSortUnroll / 2; u++) {
                const int e = half * (kSortUnroll / 2) + u;
                const int64_t i = i0 + kSortThreads * u;
                uint32_t t = kNoTile;
                if (i < p.n) {
                    AxisQ a[3];
                    const float m = p.masses ? __ldg(p.masses + i) : p.umass;
                    t = particle_cell<true>(p, v[u].x, v[u].y, v[u].z, m, a);
                    wx[e] = pack_axis(a[0], mx);
                    wy[e] = pack_axis(a[1], my);
                    wz[e] = pack_axis(a[2], mz);
                    if (p.corner && t != kNoTile) {
                        const float mm = m * mscale;
                        f2sum w = corner_factor_q(a[0], a[1], a[2]);
                        const float h = __fmul_rn(w.hi, mm);
                        w = f2sum{h, fmaf(w.hi, mm, -h) + w.lo * mm};
                        f2_accumulate(alt, f2_signed(w, a[0].cell ^ a[1].cell ^ a[2].cell));
                    }
                }
                const uint32_t r = claim_slot(GLOBAL ? cursor : sh_cur, t);
                key[e] = t == kNoTile ? kNoTile : GLOBAL ? r : (t << 13) | r;
            }
        }
        if (!GLOBAL) {
            __syncthreads();
            uint32_t base[kSortUnroll];
#pragma unroll
            for (int e = 0; e < kSortUnroll; e++)
                if (key[e] != kNoTile && (key[e] & 0x1fffu) == 0u)
                    base[e] = atomicAdd(cursor + (key[e] >> 13) * kStride, sh_cur[key[e] >> 13]);
#pragma unroll
            for (int e = 0; e < kSortUnroll; e++)
                if (key[e] != kNoTile && (key[e] & 0x1fffu) == 0u)
                    sh_cur[key[e] >> 13] = base[e];
            __syncthreads();
        }
#pragma unroll
        for (int e = 0; e < kSortUnroll; e++) {
            if (key[e] != kNoTile) {
                const uint32_t slot = GLOBAL ? key[e] : sh_cur[key[e] >> 13] + (key[e] & 0x1fffu);
                const int64_t i = c0 + threadIdx.x + (int64_t)kSortThreads * e;
                // (the mass word carries a uniform mass too, for grouped passes)
                const float m = p.masses ? __ldg(p.masses + i) : p.umass;
                sorted[slot] = make_uint4(wx[e], wy[e], wz[e], __float_as_uint(m));
            }
        }
        if (!GLOBAL) {
            __syncthreads();
#pragma unroll
            for (int e = 0; e < kSortUnroll; e++)
                if (key[e] != kNoTile && (key[e] & 0x1fffu) == 0u)
                    sh_cur[key[e] >> 13] = 0u;
            __syncthreads();
        }
    }
    if (p.corner) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const f2sum other = {__shfl_xor_sync(0xffffffffu, alt.hi, o),
                                 __shfl_xor_sync(0xffffffffu, alt.lo, o)};
            alt = f2_add2(alt, other);
        }
        if (lane == 0) {
            const long long w = __float2ll_rn(alt.hi) + __float2ll_rn(alt.lo);
            if (w != 0)
                atomicAdd((unsigned long long *)&st->alt_sum, (unsigned long long)w);
        }
    }
}

// Halo layer of one tile (the cells at local x = ext_x, y = ext_y or z = ext_z),
// stored as 64-bit sums.  S* = T* + 1.
//   X face (x = ext_x):              e = y*SZ + z                   y<=ext_y, z<=ext_z
//   Y face (y = ext_y, x < ext_x):   e = NX + x*SZ + z              z<=ext_z
//   Z face (z = ext_z, x, y inside): e = NX + NY + x*TY + y
// Low faces of one tile (local x = 0, y = 0 or z = 0), 64-bit sums, each plane
// whole (edge cells appear in two planes, the corner cell in three):
//   A (x = 0):   e = y*TZ + z
//   B (y = 0):   e = TY*TZ + x*TZ + z
//   C (z = 0):   e = TY*TZ + TX*TZ + x*TY + y
template <int TX, int TY, int TZ>
struct TileLayout {
    static constexpr int SX = TX + 1, SY = TY + 1, SZ = TZ + 1;
    static constexpr int NACC = SX * SY * SZ;
    static constexpr int NX = SY * SZ, NY = TX * SZ, NZ = TX * TY;
    static constexpr int NHALO = NX + NY + NZ;
    static constexpr int NFACE = TY * TZ + TX * TZ + TX * TY;

    __device__ __forceinline__ static int acc_index(int x, int y, int z)
    {
        return (x * SY + y) * SZ + z;
    }

    // Halo entry of a cell on the halo layer.
    __device__ __forceinline__ static int halo_encode(int x, int y, int z, int ex, int ey)
    {
        if (x == ex)
            return y * SZ + z;
        if (y == ey)
            return NX + x * SZ + z;
        return NX + NY + x * TY + y;
    }
};

struct TileParams {
    int dims;
    int64_t plane;
    int row;
    int ntx, nty, ntz;
};

constexpr int kTileThreads = 512;

__device__ __forceinline__ float fixed_to_float(long long v, float inv_scale)
{
    // One rounding (int64 -> float), then an exact power-of-two scaling.
    return i64_to_f32_rn(v) * inv_scale;
}

// The tiles of a launch grid of (ntz, nty, ntx * boxes) blocks from slice z0 on.
struct TileOfBlock {
    int box, t, tx, ty, tz;
};

__device__ __forceinline__ TileOfBlock tile_of_block(const TileParams &p, int z0)
{
    TileOfBlock b;
    const int z = (int)blockIdx.z - z0;
    b.box = (int)gridDim.z - z0 == p.ntx ? 0 : z / p.ntx;
    b.tx = z - b.box * p.ntx;
    b.ty = (int)blockIdx.y;
    b.tz = (int)blockIdx.x;
    b.t = (b.tx * p.nty + b.ty) * p.ntz + b.tz;
    return b;
}

// 2^-s for a pass's fixed-point shift s (|s| <= 100).
__device__ __forceinline__ float inv_scale_of(int s)
{
    return __uint_as_float((uint32_t)(127 - s) << 23);
}

// 64-bit cell sum kept as two 32-bit shared words: lo takes each weight with a
// native 32-bit atomic, and the rare carry out of it (weights are < 2^28, so at
// most one add in 2^4 carries) goes to hi.  Exact and order-independent.
// A positive weight is added whatever its value (testing for zero, a particle
// on a cell face, cost more than the rare empty add: 0.218 -> 0.213 ms for
// 27 M particles on 256^3); a negative one skips zero, since its high-word
// term assumes w > 0.  (Testing the eight words returned for a particle together, by
// their maximum, took 11 % longer: eight results live at once cost a CTA per SM.)
__device__ __forceinline__ void acc_add(unsigned *lo, unsigned *hi, int idx, unsigned w, bool neg)
{
    if (neg && w == 0u)
        return;
    if (!neg) {
        const unsigned old = atomicAdd(&lo[idx], w);
        if (old + w < old)
            atomicAdd(&hi[idx], 1u);
    } else {  // adding -w: lo += 2^32 - w, hi += carry - 1
        const unsigned wl = 0u - w;
        const unsigned old = atomicAdd(&lo[idx], wl);
        if (!(old + wl < old))
            atomicAdd(&hi[idx], 0xffffffffu);
    }
}

__device__ __forceinline__ long long acc_get(const unsigned *lo, const unsigned *hi, int idx)
{
    return (long long)(((unsigned long long)hi[idx] << 32) | lo[idx]);
}

// Where a tile's records lie: one range (a counting sort over the pass), or a
// run in every chunk of the box (a binned pass).
struct RangeRecords {
    const uint32_t *tile_start;
};
struct ChunkRecords {
    const uint16_t *hdr;
    int stride;
    int len[kMaxGroupBoxes], nchunks[kMaxGroupBoxes];
    int group[kMaxGroupBoxes];  // runs a warp of the tile kernel takes at a time
    uint32_t rec0[kMaxGroupBoxes], hdr0[kMaxGroupBoxes];
};

// A pass's constants as its tile kernels take them.  host[b] != 0: box b's
// particles weigh a uniform mass, and its constants come from the host, for all
// n[b] particles (where some were skipped, st->pass_bad of them, the mean is
// formed again from the rest), and the box's first tile puts them in the status
// words and the running sums.  Else the sort kernel's last CTA did.  umass is the
// uniform mass either way.
struct TileConsts {
    int host[kMaxGroupBoxes];
    int fx_shift[kMaxGroupBoxes];
    long long mean_fixed[kMaxGroupBoxes];
    double umass[kMaxGroupBoxes];
    long long n[kMaxGroupBoxes];
    double inv_cells;
    double *field_mass, *field_sub;
};

__device__ __forceinline__ PassConsts box_consts(const TileConsts &k, int box,
                                                 const DeviceStatus *st)
{
    if (!k.host[box])
        return {st->pass_mass, st->fx_shift, st->mean_fixed};
    const unsigned long long bad = st->pass_bad;
    if (bad == 0)
        return {(double)k.n[box] * k.umass[box], k.fx_shift[box], k.mean_fixed[box]};
    return pass_consts((double)(k.n[box] - (long long)bad) * k.umass[box],
                       (float)fabs(k.umass[box]), k.inv_cells);
}

// Walks the records of tile t: begin() issues the first loads, walk() calls
// f(record) for every record (one lane each).
struct RangeWalk {
    uint32_t s0, s1;
    __device__ __forceinline__ void begin(const RangeRecords &r, int box, int ntiles, int t)
    {
        const uint32_t *start = fresh(r.tile_start) + (size_t)box * (ntiles + 1);
        s0 = start[t];
        s1 = start[t + 1];
    }
    template <class F>
    __device__ __forceinline__ void walk(const uint4 *__restrict__ sorted, F &&f) const
    {
        for (uint32_t i = s0 + threadIdx.x; i < s1; i += blockDim.x)
            f(sorted[i]);
    }
};

// A warp takes up to 32 chunks' runs at a time, lane l holding run l, and walks
// their records 32 at a time: a lane finds its record's run by bisection of the
// runs' inclusive scan (five shuffles).  Runs of any length keep all lanes
// busy, and no barrier is needed.  The next runs' bounds are loaded meanwhile.
struct ChunkWalk {
    const uint16_t *hdr;  // this lane's column of the box's headers
    int stride, len, nchunks, group, c;
    uint32_t rec0, lo, hi;  // run bounds within chunk c
    __device__ __forceinline__ void load()
    {
        lo = hi = 0u;
        if ((int)(threadIdx.x & 31) < group && c < nchunks) {
            const uint16_t *h = hdr + (size_t)c * (size_t)stride;
            lo = __ldg(h);
            hi = __ldg(h + 1);
        }
    }
    __device__ __forceinline__ void begin(const ChunkRecords &r, int box, int, int t)
    {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        stride = r.stride;
        len = r.len[box];
        nchunks = r.nchunks[box];
        rec0 = r.rec0[box];
        hdr = fresh(r.hdr) + (size_t)r.hdr0[box] * (size_t)stride + t;
        group = r.group[box];
        c = wid * group + lane;
        load();
    }
    template <class F>
    __device__ __forceinline__ void walk(const uint4 *__restrict__ sorted, F &&f)
    {
        const int lane = threadIdx.x & 31;
        for (; c - lane < nchunks;) {
            const uint32_t n = hi - lo;
            uint32_t incl = n;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d)
                    incl += y;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            const uint32_t delta = rec0 + (uint32_t)c * (uint32_t)len + lo - (incl - n);
            c += (int)(blockDim.x >> 5) * group;
            load();
            for (uint32_t j0 = 0; j0 < total; j0 += 32) {
                const uint32_t j = j0 + lane;
                int s = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, incl, s + step - 1) <= j)
                        s += step;
                const uint32_t i = __shfl_sync(0xffffffffu, delta, s) + j;
                if (j < total)
                    f(sorted[i]);
            }
        }
    }
};
template <class Records>
struct WalkOf {
    typedef RangeWalk T;
};
template <>
struct WalkOf<ChunkRecords> {
    typedef ChunkWalk T;
};

// One tile of one box (grid_stride floats between the boxes' grids).
template <int TX, int TY, int TZ, bool VARMASS, bool CLEAN, class Records>
__global__ void __launch_bounds__(kTileThreads, 4)
    k_tile_deposit(TileParams p, const uint4 *__restrict__ sorted,
                   const __grid_constant__ Records records,
                   const __grid_constant__ TileConsts consts, DeviceStatus *st, float *__restrict__ grid, long long *__restrict__ faces,
                   long long *__restrict__ halo, int64_t grid_stride)
{
    using L = TileLayout<TX, TY, TZ>;
    extern __shared__ __align__(16) unsigned acc_words[];
    unsigned *lo = acc_words, *hi = acc_words + L::NACC;
    const TileOfBlock tb = tile_of_block(p, 0);
    const int ntiles = p.ntx * p.nty * p.ntz;
    st += tb.box;
    grid += (size_t)tb.box * (size_t)grid_stride;
    const size_t slot = (size_t)tb.box * ntiles + tb.t;
    const int x0 = tb.tx * TX, y0 = tb.ty * TY, z0 = tb.tz * TZ;
    const int ex = min(TX, p.dims - x0), ey = min(TY, p.dims - y0), ez = min(TZ, p.dims - z0);
    for (int i = threadIdx.x; i < (2 * L::NACC + 3) / 4; i += blockDim.x)
        reinterpret_cast<uint4 *>(acc_words)[i] = make_uint4(0u, 0u, 0u, 0u);
    wait_previous();
    sorted = fresh(sorted);
    st = fresh(st);
    typename WalkOf<Records>::T records_walk;
    records_walk.begin(records, tb.box, ntiles, tb.t);
    __syncthreads();

    const int s = consts.host[tb.box] ? consts.fx_shift[tb.box] : st->fx_shift;
    const float inv_scale = inv_scale_of(s);
    // Weights in 2^-s mass units with s = 154 - emax (common.cuh pair_w / z_mass /
    // corner_w, as the window engine computes them).
    const int emax = 154 - s;
    const unsigned ubits = __float_as_uint((float)consts.umass[tb.box]);  // (it was a float)
    const unsigned umant = (ubits & 0x7fffffu) | 0x800000u;
    const int uef = (int)((ubits >> 23) & 0xffu);
    const bool uneg = (ubits >> 31) != 0u;
    records_walk.walk(sorted, [&](const uint4 w) {
        unsigned mant = umant;
        int ef = uef;
        bool neg = uneg;
        if (VARMASS) {
            const unsigned mb = w.w;
            ef = (int)((mb >> 23) & 0xffu);
            mant = (mb & 0x7fffffu) | 0x800000u;
            neg = (mb >> 31) != 0u;
        }
        if (ef == 0)  // zero or subnormal mass deposits nothing
            return;
        const int dsh = max(emax - ef, 0);
        const uint32_t qx = w.x & (kFracOne - 1u), qy = w.y & (kFracOne - 1u),
                       qz = w.z & (kFracOne - 1u);
        const uint32_t rx = kFracOne - qx, ry = kFracOne - qy, rz = kFracOne - qz;
        const int base = L::acc_index((int)(w.x >> kFracBits), (int)(w.y >> kFracBits),
                                      (int)(w.z >> kFracBits));
        constexpr int DX = L::SY * L::SZ, DY = L::SZ;
        const uint32_t p00 = pair_w(rx, ry), p10 = pair_w(qx, ry), p01 = pair_w(rx, qy),
                       p11 = pair_w(qx, qy);
        const uint32_t z0 = z_mass(rz, mant, dsh), z1 = z_mass(qz, mant, dsh);
        acc_add(lo, hi, base, corner_w(p00, z0), neg);
        acc_add(lo, hi, base + DX, corner_w(p10, z0), neg);
        acc_add(lo, hi, base + DY, corner_w(p01, z0), neg);
        acc_add(lo, hi, base + DX + DY, corner_w(p11, z0), neg);
        acc_add(lo, hi, base + 1, corner_w(p00, z1), neg);
        acc_add(lo, hi, base + DX + 1, corner_w(p10, z1), neg);
        acc_add(lo, hi, base + DY + 1, corner_w(p01, z1), neg);
        acc_add(lo, hi, base + DX + DY + 1, corner_w(p11, z1), neg);
    });
    __syncthreads();

    // Cells strictly inside the tile (no low face): final value.  A thread keeps
    // its (y, z) and steps through x.
    {
        constexpr int NXP = kTileThreads / (TY * TZ);  // x planes per step
        const PassConsts pc = box_consts(consts, tb.box, st);
        const long long mean = pc.mean_fixed;
        if (consts.host[tb.box] && tb.t == 0 && threadIdx.x == 0)
            store_pass_consts(pc, CLEAN, consts.field_mass + tb.box, consts.field_sub + tb.box,
                              st);
        const int z = threadIdx.x % TZ, y = (threadIdx.x / TZ) % TY;
        int x = threadIdx.x / (TY * TZ);
        x += x == 0 ? NXP : 0;
        if (y >= 1 && z >= 1 && y < ey && z < ez) {
            float *dst = grid + cell_index(p.plane, p.row, x0 + x, y0 + y, z0 + z);
            int idx = L::acc_index(x, y, z);
            for (; x < ex; x += NXP) {
                const float v = fixed_to_float(acc_get(lo, hi, idx) - mean, inv_scale);
                if (CLEAN)
                    *dst = v;
                else
                    *dst += v;
                dst += NXP * p.plane;
                idx += NXP * L::SY * L::SZ;
            }
        }
    }
    // The low faces (entries beyond a partial tile's extent are not read) ...
    long long *f = faces + slot * L::NFACE;
    for (int e = threadIdx.x; e < TY * TZ; e += kTileThreads)
        f[e] = acc_get(lo, hi, L::acc_index(0, e / TZ, e % TZ));
    for (int e = threadIdx.x; e < TX * TZ; e += kTileThreads)
        f[TY * TZ + e] = acc_get(lo, hi, L::acc_index(e / TZ, 0, e % TZ));
    for (int e = threadIdx.x; e < TX * TY; e += kTileThreads)
        f[TY * TZ + TX * TZ + e] = acc_get(lo, hi, L::acc_index(e / TY, e % TY, 0));
    // ... and the halo layer: a warp per row, lanes along it
    long long *h = halo + slot * L::NHALO;
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < L::SY + TX + TX; r += kTileThreads / 32) {
        if (r < L::SY) {
            if (lane < L::SZ && r <= ey)
                h[r * L::SZ + lane] = acc_get(lo, hi, L::acc_index(ex, r, lane));
        } else if (r < L::SY + TX) {
            const int x = r - L::SY;
            if (lane < L::SZ && x < ex)
                h[L::NX + x * L::SZ + lane] = acc_get(lo, hi, L::acc_index(x, ey, lane));
        } else {
            const int x = r - L::SY - TX;
            if (lane < TY && x < ex)
                h[L::NX + L::NY + x * TY + lane] = acc_get(lo, hi, L::acc_index(x, lane, ez));
        }
    }
}

// Extent of tile index ti along an axis of `dims` cells with tiles of T.
__device__ __forceinline__ int tile_ext(int ti, int T, int dims)
{
    return min(T, dims - ti * T);
}

// Low-face cells of one tile of one box: the tile's own sum of a cell and the
// shares that the halo layers of its lower neighbours hold.  A cell on one low
// face has one such neighbour, one on an edge three, the corner cell seven.
// The first slice of blocks ends the boxes' passes instead (beside the others: as
// part of a tile's block it cost 6 us).  The corner mode
// k = (N/2, N/2, N/2) of an even grid is sum (-1)^(x+y+z) rho(x): this pass's
// exact share, from the sort's partial sums, joins the grid's running value (the
// subtracted mean contributes nothing: the signs balance on an even grid).  The
// sums that a pass accumulates are zeroed for the next one; a grouped pass also
// hands each box's count of skipped particles to bad_out and zeroes it.
struct PassEnd {
    const double *corner_part;       // binned passes: one per sort CTA, else null
    int first[kMaxGroupBoxes + 1];   // each box's partials
    double unit_mass[kMaxGroupBoxes];  // what they are in units of
    double *field_corner;
    bool clean;  // the grid's first pass: its sums start here
    unsigned long long *bad_out;
};

__device__ __forceinline__ void end_pass(const PassEnd &e, int box, DeviceStatus *st)
{
    __shared__ double sh[8];
    double corner = 0.0;
    if (e.corner_part) {
        for (int i = e.first[box] + threadIdx.x; i < e.first[box + 1]; i += blockDim.x)
            corner += fresh(e.corner_part)[i];
        corner = block_sum_d(corner, sh) * e.unit_mass[box];
    }
    if (threadIdx.x != 0)
        return;
    st->pass_bad = 0;
    if (!e.corner_part) {
        corner = ldexp((double)st->alt_sum, -(st->fx_shift + 4));
        st->alt_sum = 0;
    }
    e.field_corner[box] = (e.clean ? 0.0 : e.field_corner[box]) + corner;
    if (e.bad_out) {
        e.bad_out[box] = st->bad_particles;
        st->bad_particles = 0;
    }
}

template <int TX, int TY, int TZ, bool CLEAN>
__global__ void __launch_bounds__(256)
    k_face_gather(TileParams p, const long long *__restrict__ faces,
                  const long long *__restrict__ halo, const __grid_constant__ PassEnd end,
                  DeviceStatus *st, float *__restrict__ grid, int64_t grid_stride)
{
    using L = TileLayout<TX, TY, TZ>;
    wait_previous();
    faces = fresh(faces);
    halo = fresh(halo);
    st = fresh(st);
    if (blockIdx.z == 0) {
        const int nbox = ((int)gridDim.z - 1) / p.ntx;
        for (int b = blockIdx.y * gridDim.x + blockIdx.x; b < nbox; b += gridDim.x * gridDim.y)
            end_pass(end, b, st + b);
        return;
    }
    const TileOfBlock tb = tile_of_block(p, 1);
    const int ntiles = p.ntx * p.nty * p.ntz;
    st += tb.box;
    const int x0 = tb.tx * TX, y0 = tb.ty * TY, z0 = tb.tz * TZ;
    const int ex = min(TX, p.dims - x0), ey = min(TY, p.dims - y0), ez = min(TZ, p.dims - z0);
    // Lower neighbour along each axis (periodic) and its extent.
    const int txm = tb.tx ? tb.tx - 1 : p.ntx - 1;
    const int tym = tb.ty ? tb.ty - 1 : p.nty - 1;
    const int tzm = tb.tz ? tb.tz - 1 : p.ntz - 1;
    const int exm = tile_ext(txm, TX, p.dims), eym = tile_ext(tym, TY, p.dims),
              ezm = tile_ext(tzm, TZ, p.dims);
    const float inv_scale = inv_scale_of(st->fx_shift);
    const long long mean = st->mean_fixed;
    const long long *f = faces + ((size_t)tb.box * ntiles + tb.t) * L::NFACE;
    halo += (size_t)tb.box * ntiles * L::NHALO;
    float *g0 = grid + (size_t)tb.box * (size_t)grid_stride +
                cell_index(p.plane, p.row, x0, y0, z0);
    auto halo_of = [&](int sx, int sy, int sz) {
        return halo + (size_t)((sx * p.nty + sy) * p.ntz + sz) * L::NHALO;
    };
    auto put = [&](int a, int b, int c, long long sum) {
        float *dst = g0 + (int64_t)a * p.plane + b * p.row + c;
        const float v = fixed_to_float(sum - mean, inv_scale);
        if (CLEAN)
            *dst = v;
        else
            *dst += v;
    };
    {
        const long long *h = halo_of(txm, tb.ty, tb.tz);
        for (int e = threadIdx.x; e < TY * TZ; e += 256) {
            const int y = e / TZ, z = e % TZ;
            if (y >= 1 && z >= 1 && y < ey && z < ez)
                put(0, y, z, f[e] + h[y * L::SZ + z]);
        }
    }
    {
        const long long *h = halo_of(tb.tx, tym, tb.tz) + L::NX;
        for (int e = threadIdx.x; e < TX * TZ; e += 256) {
            const int x = e / TZ, z = e % TZ;
            if (x >= 1 && z >= 1 && x < ex && z < ez)
                put(x, 0, z, f[TY * TZ + e] + h[x * L::SZ + z]);
        }
    }
    {
        const long long *h = halo_of(tb.tx, tb.ty, tzm) + L::NX + L::NY;
        for (int e = threadIdx.x; e < TX * TY; e += 256) {
            const int x = e / TY, y = e % TY;
            if (x >= 1 && y >= 1 && x < ex && y < ey)
                put(x, y, 0, f[TY * TZ + TX * TZ + e] + h[e]);
        }
    }
    // Edges and the corner: every non-empty subset of the axes on which the
    // cell sits on the low face names one lower neighbour.
    const int e = threadIdx.x;
    if (e >= TX + TY + TZ)
        return;
    const int a = e < TY + TZ ? 0 : e - TY - TZ;
    const int b = e < TZ ? 0 : e < TY + TZ ? e - TZ : 0;
    const int c = e < TZ ? e : 0;
    if (a >= ex || b >= ey || c >= ez || (e == TZ) || (e == TY + TZ))
        return;
    long long sum = a == 0 ? f[b * TZ + c] : f[TY * TZ + a * TZ + c];
    const int zmask = (a == 0 ? 1 : 0) | (b == 0 ? 2 : 0) | (c == 0 ? 4 : 0);
    for (int mask = 1; mask < 8; mask++) {
        if (mask & ~zmask)
            continue;
        const int sx = (mask & 1) ? txm : tb.tx, sy = (mask & 2) ? tym : tb.ty,
                  sz = (mask & 4) ? tzm : tb.tz;
        const int sex = (mask & 1) ? exm : ex, sey = (mask & 2) ? eym : ey;
        const int xs = (mask & 1) ? exm : a, ys = (mask & 2) ? eym : b, zs = (mask & 4) ? ezm : c;
        sum += halo_of(sx, sy, sz)[L::halo_encode(xs, ys, zs, sex, sey)];
    }
    put(a, b, c, sum);
}

int ilog2(int v)
{
    int l = 0;
    while ((1 << l) < v)
        l++;
    return l;
}

// What the tile kernels of a pass write: nbox grids from `grid` on, with
// their corner sums and (grouped passes) skipped-particle counts.
struct TileTarget {
    float *grid;
    int64_t grid_stride;
    int nbox;
    bool var;    // weights from the records' masses, else from the boxes' uniform masses
    bool clean;
    TileConsts consts;
    PassEnd end;
};

template <int TX, int TY, int TZ, class Records>
cudaError_t launch_tile_kernels(const DepositGeom &g, const TileTarget &a, const Records &records,
                                DepositScratch &s,
                                DeviceStatus *dstat, cudaStream_t stream, int64_t *launches,
                                StageHook hook, void *hook_user)
{
    using L = TileLayout<TX, TY, TZ>;
    TileParams tp;
    tp.dims = g.grid.dims;
    tp.plane = g.grid.plane;
    tp.row = g.grid.row;
    tp.ntx = g.ntx;
    tp.nty = g.nty;
    tp.ntz = g.ntz;
    const size_t smem = sizeof(uint4) * ((2 * L::NACC + 3) / 4);
    const bool var = a.var;
    const dim3 tiles((unsigned)g.ntz, (unsigned)g.nty, (unsigned)(g.ntx * a.nbox));
    const dim3 slices(tiles.x, tiles.y, tiles.z + 1);
    cudaError_t err;
#define GENPK_TILE_LAUNCH(V, C)                                                                \
    do {                                                                                       \
        auto kern = k_tile_deposit<TX, TY, TZ, V, C, Records>;                                 \
        err = ensure_dynamic_smem(kern, smem);                                                 \
        if (err != cudaSuccess)                                                                \
            return err;                                                                        \
        err = launch_after(kern, tiles, kTileThreads, smem, stream, tp, s.sorted, records,     \
                           a.consts, dstat, a.grid, s.faces, s.halo, a.grid_stride);           \
    } while (0)
    if (var && a.clean)
        GENPK_TILE_LAUNCH(true, true);
    else if (var)
        GENPK_TILE_LAUNCH(true, false);
    else if (a.clean)
        GENPK_TILE_LAUNCH(false, true);
    else
        GENPK_TILE_LAUNCH(false, false);
#undef GENPK_TILE_LAUNCH
    (*launches)++;
    if (hook)
        hook(hook_user, "dep_tile");
    if (err != cudaSuccess)
        return err;
    auto face = a.clean ? k_face_gather<TX, TY, TZ, true> : k_face_gather<TX, TY, TZ, false>;
    err = launch_after(face, slices, 256, 0, stream, tp, s.faces, s.halo, a.end, dstat, a.grid,
                       a.grid_stride);
    (*launches)++;
    if (hook)
        hook(hook_user, "dep_faces");
    return err;
}

template <class Records>
cudaError_t launch_tile_pass(const DepositGeom &g, const TileTarget &t, const Records &r,
                             DepositScratch &s, DeviceStatus *dstat, cudaStream_t stream, int64_t *launches,
                             StageHook hook, void *hook_user)
{
    if (g.tx == 8)
        return launch_tile_kernels<8, 8, 8>(g, t, r, s, dstat, stream, launches, hook, hook_user);
    if (g.tz == 8)
        return launch_tile_kernels<16, 16, 8>(g, t, r, s, dstat, stream, launches, hook, hook_user);
    return launch_tile_kernels<16, 16, 16>(g, t, r, s, dstat, stream, launches, hook, hook_user);
}

SortParams sort_params(const DepositGeom &g, const float *pos, const float *masses, float mass,
                       int64_t n, float uh, float ul, int ctas)
{
    SortParams sp;
    sp.pos = pos;
    sp.masses = masses;
    sp.n = n;
    sp.ctas = ctas;
    sp.dims = g.grid.dims;
    sp.uh = uh;
    sp.ul = ul;
    sp.lx = ilog2(g.tx);
    sp.ly = ilog2(g.ty);
    sp.lz = ilog2(g.tz);
    sp.nty = g.nty;
    sp.ntz = g.ntz;
    sp.ntiles = g.ntiles;
    sp.umass = mass;
    sp.corner = (g.grid.dims % 2 == 0) ? 1 : 0;
    return sp;
}

// The histogram (and scan) and scatter launches of a pass over `ctas` sort CTAs.
template <class Src>
cudaError_t launch_sort(const DepositGeom &g, const Src &src, const ScanBoxes &sb, DepositScratch &s,
                        const TileTarget &t, DeviceStatus *dstat, int ctas, cudaStream_t stream,
                        int64_t *launches, StageHook hook, void *hook_user)
{
    auto mark = [&](const char *name) {
        (*launches)++;
        if (hook)
            hook(hook_user, name);
    };
    ScanOut out;
    out.totals = s.totals;
    out.tile_start = s.tile_start;
    out.cursor = s.cursor;
    out.cursor_stride = deposit_shared_hist(g) ? kCursorStride : 1;
    out.ticket = s.ticket;
    out.mass_part = s.mass_part;
    out.inv_cells = t.consts.inv_cells;
    out.clean = t.clean;
    out.field_mass = t.consts.field_mass;
    out.field_sub = t.consts.field_sub;
    // (max_mass_bits and alt_sum are zero here: the pass that used them last
    // zeroed them, in scan_box / k_window_prep and the finishing kernels)
    const bool shared_hist = deposit_shared_hist(g);
    const size_t hsmem = shared_hist ? deposit_hist_smem(g) : 0;
    auto hist = shared_hist ? k_sort_hist<false, Src> : k_sort_hist<true, Src>;
    auto scatter = shared_hist ? k_sort_scatter<false, Src> : k_sort_scatter<true, Src>;
    cudaError_t err;
    if ((err = ensure_dynamic_smem(hist, hsmem)) != cudaSuccess)
        return err;
    if ((err = launch_after(hist, ctas, kSortThreads, hsmem, stream, src, out, sb, dstat)) !=
        cudaSuccess)
        return err;
    mark("dep_hist");
    if ((err = ensure_dynamic_smem(scatter, hsmem)) != cudaSuccess)
        return err;
    err = launch_after(scatter, ctas, kSortThreads, hsmem, stream, src, s.cursor, s.sorted, dstat);
    mark("dep_scatter");
    return err;
}

// Chunk length and count of a binned pass over n particles on `ctas` CTAs:
// whole rounds of chunks, at most kBinMax particles each.
void bin_chunks(int64_t n, int ctas, int *len, int *nchunks)
{
    const int64_t rounds = std::max<int64_t>(1, (n + (int64_t)ctas * kBinMax - 1) / ((int64_t)ctas * kBinMax));
    int64_t l = (n + ctas * rounds - 1) / (ctas * rounds);
    l = std::max<int64_t>(1, (l + kBinThreads - 1) / kBinThreads) * kBinThreads;
    l = std::min<int64_t>(l, kBinMax);
    *len = (int)l;
    *nchunks = (int)((n + l - 1) / l);
}

// Runs a warp of the tile kernel takes at a time: whole rounds of the CTA's
// warps, at most 32 runs each, the last round spread over every warp.
int bin_group(int nchunks)
{
    const int warps = kTileThreads / 32;
    const int rounds = std::max(1, (nchunks + 32 * warps - 1) / (32 * warps));
    return std::max(1, (nchunks + rounds * warps - 1) / (rounds * warps));
}

int bin_stride(int ntiles)
{
    return (ntiles + 1 + 3) & ~3;  // rows of whole 8-byte groups
}

// Box b's constants from the host where its particles weigh a uniform mass.
void set_host_consts(TileConsts *k, int b, const float *masses, float mass, int64_t n)
{
    const PassConsts c = pass_consts((double)n * (double)mass, (float)std::fabs((double)mass),
                                     k->inv_cells);
    k->host[b] = masses ? 0 : 1;
    k->fx_shift[b] = c.fx_shift;
    k->mean_fixed[b] = c.mean_fixed;
    k->umass[b] = (double)mass;
    k->n[b] = (long long)n;
}

template <class Src>
cudaError_t launch_bins(const DepositGeom &g, const Src &src, const ChunkRecords &rec, int stage_len,
                        DepositScratch &s, const TileTarget &t, DeviceStatus *dstat, int ctas,
                        cudaStream_t stream, int64_t *launches, StageHook hook, void *hook_user)
{
    BinOut out;
    out.sorted = s.sorted;
    out.hdr = s.hdr;
    out.stride = rec.stride;
    out.mass_part = s.mass_part;
    out.corner_part = s.mass_part + ctas;
    out.ticket = s.ticket;
    out.inv_cells = t.consts.inv_cells;
    out.clean = t.clean;
    out.field_mass = t.consts.field_mass;
    out.field_sub = t.consts.field_sub;
    const size_t smem = sizeof(uint4) * (size_t)stage_len + 4 * (size_t)((g.ntiles + 3) & ~3);
    auto kern = k_bin_sort<Src>;
    cudaError_t err;
    if ((err = ensure_dynamic_smem(kern, smem)) != cudaSuccess)
        return err;
    err = launch_after(kern, ctas, kBinThreads, smem, stream, src, out, stage_len, dstat);
    (*launches)++;
    if (hook)
        hook(hook_user, "dep_bins");
    return err;
}

}  // namespace

bool deposit_binned(const DepositGeom &g)
{
    return g.ntiles <= kBinMaxTiles;
}

size_t deposit_header_words(const DepositGeom &g, int64_t n, int ctas)
{
    int len, nchunks;
    bin_chunks(n, std::max(ctas, 1), &len, &nchunks);
    return (size_t)nchunks * (size_t)bin_stride(g.ntiles);
}

// Tile edges of at most 16 cells: the packed record keeps 4 bits of tile-local
// cell beside each 28-bit fraction.
bool deposit_tile_supported(int tx, int ty, int tz)
{
    return (tx == 8 && ty == 8 && tz == 8) || (tx == 16 && ty == 16 && tz == 8) ||
           (tx == 16 && ty == 16 && tz == 16);
}

TileShape deposit_default_tile(int dims, int64_t n)
{
    (void)n;
    if (dims <= 64)
        return {8, 8, 8};
    return {16, 16, 16};
}

void deposit_scratch_sizes(const DepositGeom &g, size_t *face_elems, size_t *halo_elems)
{
    const int tx = g.tx, ty = g.ty, tz = g.tz;
    *face_elems = (size_t)g.ntiles * (size_t)(ty * tz + tx * tz + tx * ty);
    *halo_elems = (size_t)g.ntiles * (size_t)((ty + 1) * (tz + 1) + tx * (tz + 1) + tx * ty);
}

size_t deposit_cursor_words(const DepositGeom &g)
{
    return (size_t)g.ntiles * (deposit_shared_hist(g) ? kCursorStride : 1);
}

size_t deposit_hist_smem(const DepositGeom &g)
{
    return sizeof(uint32_t) * (size_t)g.ntiles;
}

bool deposit_shared_hist(const DepositGeom &g)
{
    return deposit_hist_smem(g) <= 160 * 1024;
}

int deposit_sort_ctas(const DepositGeom &g, int64_t n, int num_sms)
{
    if (deposit_binned(g))
        return (int)std::max<int64_t>(1, std::min<int64_t>(num_sms, (n + kBinThreads - 1) / kBinThreads));
    int per_sm = 2;
    if (deposit_shared_hist(g) && deposit_hist_smem(g) > 100 * 1024)
        per_sm = 1;
    const int64_t want = (n + kSortChunkParticles - 1) / kSortChunkParticles;
    return (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)num_sms * per_sm, want));
}

cudaError_t deposit_pass(const DepositGeom &g, const DepositArgs &a, DepositScratch &s,
                         DeviceStatus *dstat, int sort_ctas, cudaStream_t stream,
                         int64_t *launches, StageHook hook, void *hook_user)
{
    const OneBox src{sort_params(g, a.pos, a.masses, a.mass, a.n, g.units_hi, g.units_lo,
                                 sort_ctas)};
    TileTarget t{a.grid, 0, 1, a.masses != nullptr, a.clean, {}, {}};
    t.consts.inv_cells = 1.0 / ((double)g.grid.dims * g.grid.dims * g.grid.dims);
    t.consts.field_mass = a.field_mass;
    t.consts.field_sub = a.field_sub;
    t.end.field_corner = a.field_corner;
    t.end.clean = a.clean;
    t.consts.umass[0] = (double)a.mass;
    if (deposit_binned(g)) {
        OneBin one = {};
        one.b.s = src.p;
        bin_chunks(a.n, sort_ctas, &one.b.len, &one.b.nchunks);
        ChunkRecords rec = {};
        rec.hdr = s.hdr;
        rec.stride = bin_stride(g.ntiles);
        rec.len[0] = one.b.len;
        rec.nchunks[0] = one.b.nchunks;
        rec.group[0] = bin_group(one.b.nchunks);
        set_host_consts(&t.consts, 0, a.masses, a.mass, a.n);
        t.end.corner_part = s.mass_part + sort_ctas;
        t.end.first[1] = sort_ctas;
        t.end.unit_mass[0] = a.masses ? 1.0 : (double)a.mass;
        const cudaError_t e = launch_bins(g, one, rec, one.b.len, s, t, dstat, sort_ctas, stream,
                                          launches, hook, hook_user);
        if (e != cudaSuccess)
            return e;
        return launch_tile_pass(g, t, rec, s, dstat, stream, launches, hook, hook_user);
    }
    ScanBoxes sb = {};
    sb.first[1] = sort_ctas;
    sb.var[0] = a.masses ? 1 : 0;
    sb.umass[0] = (double)a.mass;
    cudaError_t err = launch_sort(g, src, sb, s, t, dstat, sort_ctas, stream, launches, hook,
                                  hook_user);
    if (err != cudaSuccess)
        return err;
    return launch_tile_pass(g, t, RangeRecords{s.tile_start}, s, dstat, stream, launches, hook, hook_user);
}

// (At most sort_ctas of them in all, unless there are more boxes: one more than
// the SMs hold at once would run alone after all the others.)
GroupLayout deposit_group_layout(int nbox, const GroupBox *boxes, int sort_ctas)
{
    GroupLayout lay = {};
    lay.nbox = nbox;
    int64_t total = 0;
    for (int b = 0; b < nbox; b++)
        total += boxes[b].n;
    int ctas[kMaxGroupBoxes], sum = 0;
    for (int b = 0; b < nbox; b++) {
        // (an empty box's one CTA sets its pass constants)
        const double share = total > 0 ? (double)sort_ctas * (double)boxes[b].n / (double)total : 0.0;
        ctas[b] = std::max(1, (int)share);
        sum += ctas[b];
    }
    auto chunks = [&](int b) { return (boxes[b].n + kBinThreads - 1) / kBinThreads; };
    for (; sum < sort_ctas; sum++) {  // the rest to the boxes whose CTAs have most to do
        int most = -1;
        for (int b = 0; b < nbox; b++)
            if (ctas[b] < chunks(b) &&
                (most < 0 || (double)boxes[b].n * ctas[most] > (double)boxes[most].n * ctas[b]))
                most = b;
        if (most < 0)
            break;
        ctas[most]++;
    }
    int c = 0;
    int64_t r = 0;
    for (int b = 0; b < nbox; b++) {
        lay.cta0[b] = c;
        lay.rec0[b] = r;
        c += (int)std::max<int64_t>(1, std::min<int64_t>(ctas[b], chunks(b)));
        r += boxes[b].n;
    }
    lay.cta0[nbox] = c;
    lay.rec0[nbox] = r;
    return lay;
}

cudaError_t deposit_group_pass(const DepositGeom &g, const GroupLayout &lay, const GroupBox *boxes,
                               float *grid0, int64_t grid_stride, double *field_mass0,
                               double *field_sub0, double *field_corner0, DepositScratch &s,
                               DeviceStatus *st0, unsigned long long *bad_out, cudaStream_t stream,
                               int64_t *launches)
{
    const int nbox = lay.nbox;
    if (nbox < 1 || nbox > kMaxGroupBoxes || !deposit_shared_hist(g) ||
        lay.rec0[nbox] > (int64_t)0xfffffffeLL)
        return cudaErrorInvalidValue;
    // Every box's records carry its mass bits, which the tile kernel reads where
    // some box's particles have masses of their own; else it takes the boxes'
    // uniform masses (six boxes of 105 M particles on 256^3: 0.87 -> 0.70 ms).
    bool var = false;
    for (int b = 0; b < nbox; b++)
        var = var || boxes[b].masses;
    TileTarget t{grid0, grid_stride, nbox, var, true, {}, {}};
    for (int b = 0; b < nbox; b++)
        t.consts.umass[b] = (double)boxes[b].mass;
    t.consts.inv_cells = 1.0 / ((double)g.grid.dims * g.grid.dims * g.grid.dims);
    t.consts.field_mass = field_mass0;
    t.consts.field_sub = field_sub0;
    t.end.field_corner = field_corner0;
    t.end.clean = true;
    t.end.bad_out = bad_out;
    if (deposit_binned(g)) {
        BinGroup src = {};
        ChunkRecords rec = {};
        rec.hdr = s.hdr;
        rec.stride = bin_stride(g.ntiles);
        src.nbox = nbox;
        uint32_t hdr0 = 0;
        int stage_len = 0;
        for (int b = 0; b <= nbox; b++)
            src.cta0[b] = lay.cta0[b];
        for (int b = 0; b < nbox; b++) {
            const GroupBox &x = boxes[b];
            BinBox &o = src.b[b];
            const int ctas = lay.cta0[b + 1] - lay.cta0[b];
            o.s = sort_params(g, x.pos, x.masses, x.mass, x.n, x.units_hi, x.units_lo, ctas);
            bin_chunks(x.n, ctas, &o.len, &o.nchunks);
            o.rec0 = (uint32_t)lay.rec0[b];
            o.hdr0 = hdr0;
            hdr0 += (uint32_t)o.nchunks;
            stage_len = std::max(stage_len, o.len);
            rec.len[b] = o.len;
            rec.nchunks[b] = o.nchunks;
            rec.group[b] = bin_group(o.nchunks);
            set_host_consts(&t.consts, b, x.masses, x.mass, x.n);
            t.end.first[b] = lay.cta0[b];
            t.end.first[b + 1] = lay.cta0[b + 1];
            t.end.unit_mass[b] = x.masses ? 1.0 : (double)x.mass;
            rec.rec0[b] = o.rec0;
            rec.hdr0[b] = o.hdr0;
        }
        t.end.corner_part = s.mass_part + lay.cta0[nbox];
        const cudaError_t e = launch_bins(g, src, rec, stage_len, s, t, st0, lay.cta0[nbox], stream,
                                          launches, nullptr, nullptr);
        if (e != cudaSuccess)
            return e;
        return launch_tile_pass(g, t, rec, s, st0, stream, launches, nullptr, nullptr);
    }
    BoxGroup src = {};
    ScanBoxes sb = {};
    src.nbox = nbox;
    for (int b = 0; b <= nbox; b++) {
        src.cta0[b] = lay.cta0[b];
        sb.first[b] = lay.cta0[b];
    }
    for (int b = 0; b < nbox; b++) {
        const GroupBox &x = boxes[b];
        src.p[b] = sort_params(g, x.pos, x.masses, x.mass, x.n, x.units_hi, x.units_lo,
                               lay.cta0[b + 1] - lay.cta0[b]);
        sb.var[b] = x.masses ? 1 : 0;
        sb.umass[b] = (double)x.mass;
        sb.rec0[b] = (long long)lay.rec0[b];
    }
    const cudaError_t err = launch_sort(g, src, sb, s, t, st0, lay.cta0[nbox], stream, launches,
                                        nullptr, nullptr);
    if (err != cudaSuccess)
        return err;
    return launch_tile_pass(g, t, RangeRecords{s.tile_start}, s, st0, stream, launches, nullptr,
                            nullptr);
}

}  // namespace genpk
