// bin_rows.cuh -- the row-binning kernel of spectrum.cu and its launch, for the
// files that instantiate it.
//
// Its twenty forms lie in bin_single.cu (one field) and bin_multi.cu: the first
// kernel of a file that a process launches loads the file's whole device code,
// and with all forms beside k_bin_finalize that cost every process's first
// spectrum 0.2 ms, also on the grids whose x pass bins (64^3: 4.19 -> 4.40 ms
// with the context's creation).
#pragma once

#include "common.cuh"
#include "internal.h"
#include "launch.cuh"

namespace genpk {

struct BinParams {
    const float2 *f[kMaxBinFields];
    const double *corner[kMaxBinFields];  // exact (N/2,N/2,N/2) value per field, or null
    int64_t corner_row;                   // row index i*N+j of that mode, -1 if none
    int np;          // pair sums per CTA partial: the instantiation's pair count
    int dims, hc, half;
    int nrbins;
    float bpu_half;  // 0.5 * binsperunit as float, for the first-guess bin
    int warps;       // warps per CTA
};

// One field's auto spectrum (bin_single.cu).
cudaError_t bin_rows_single(const BinParams &p, const BinDevice &d, double *partial, int ctas,
                            size_t smem, cudaStream_t stream);
// Two fields' cross spectrum (cross1), or every pair of nf = 2, 3 or 4 fields
// (bin_multi.cu).
cudaError_t bin_rows_multi(int nf, bool cross1, const BinParams &p, const BinDevice &d,
                           double *partial, int ctas, size_t smem, cudaStream_t stream);

namespace {

constexpr int kPromoteRows = 16;  // rows summed in FP32 before promotion to FP64

// Pairs an instantiation sums, with compile-time field indices: the single
// cross pair (0, 1) (CROSS1), or every pair a <= b of NF fields in the order
// (0,0), (0,1), ..., (0,NF-1), (1,1), ... (Re F_a F_b* is symmetric).
template <int NF, bool CROSS1>
struct PairSet {
    static constexpr int NP = CROSS1 ? 1 : NF * (NF + 1) / 2;
};

__host__ __device__ constexpr int pair_slot(int nf, int a, int b)
{
    return a * nf - a * (a - 1) / 2 + (b - a);
}

template <int NF, bool CROSS1>
__device__ __forceinline__ void add_pairs(const float2 (&fv)[NF], float w,
                                          float (&acc)[PairSet<NF, CROSS1>::NP])
{
    if (CROSS1) {
        acc[0] = fmaf(w, fmaf(fv[0].x, fv[NF - 1].x, fv[0].y * fv[NF - 1].y), acc[0]);
    } else {
#pragma unroll
        for (int a = 0; a < NF; a++)
#pragma unroll
            for (int b = a; b < NF; b++)
                acc[pair_slot(NF, a, b)] =
                    fmaf(w, fmaf(fv[a].x, fv[b].x, fv[a].y * fv[b].y), acc[pair_slot(NF, a, b)]);
    }
}

__device__ __forceinline__ int kval_dev(int i, int dims)
{
    return i <= dims / 2 ? i : i - dims;
}

// Bin of |k|^2 = kk2 >= 1: float first guess, then exact integer fix-up.
__device__ __forceinline__ int bin_lookup(uint32_t kk2, const uint32_t *thr, int nrbins,
                                          float bpu_half)
{
    int b = (int)(bpu_half * __logf((float)kk2));
    b = max(0, min(nrbins - 1, b));
    while (b + 1 < nrbins && kk2 >= thr[b + 1])
        b++;
    while (b > 0 && kk2 < thr[b])
        b--;
    return b;
}

// Shared layout (bytes, each block 16-byte aligned):
//   thr [nrbins+1] u32 | izc [hc] float2 {iw(kz), mode weight 1 or 2} |
//   per warp: whist [NP][nrbins] f64, rhist [NP][nrbins] f32, buf [NF][32*RP] float2
struct BinLayout {
    size_t izc, warps, whist, rhist, buf, per_warp;
};

__host__ __device__ inline size_t align16(size_t v)
{
    return (v + 15) & ~(size_t)15;
}

__host__ __device__ inline BinLayout bin_layout(int nrbins, int hc, int np, int nf, int rp)
{
    BinLayout L;
    L.izc = align16(sizeof(uint32_t) * (nrbins + 1));
    L.warps = L.izc + align16(sizeof(float2) * hc);
    L.whist = 0;
    L.rhist = align16(sizeof(double) * np * nrbins);
    L.buf = L.rhist + align16(sizeof(float) * np * nrbins);
    L.per_warp = L.buf + sizeof(float2) * nf * 32 * rp;
    return L;
}

// One piece of a row: 32*RP consecutive modes from kz = pb, field values into
// registers (coalesced loads; zero past the row's end).
template <int NF, int RP>
__device__ __forceinline__ void load_piece(const BinParams &p, int64_t r, int pb, int lane,
                                           float2 (&v)[NF][RP])
{
    const size_t rowoff = (size_t)r * p.hc;
#pragma unroll
    for (int t = 0; t < RP; t++) {
        const int m = pb + t * 32 + lane;
        const bool in = m < p.hc;
#pragma unroll
        for (int f = 0; f < NF; f++)
            v[f][t] = in ? __ldg(p.f[f] + rowoff + m) : make_float2(0.f, 0.f);
    }
}

// Registers -> the warp's staging buffer, with the two special modes fixed:
// (0,0,0) is skipped (zeroed) and the exact corner value replaces the
// transform's (N/2,N/2,N/2) mode.
template <int NF, int RP>
__device__ __forceinline__ void stage_piece(const BinParams &p, int64_t r, int pb, int lane,
                                            float2 (&v)[NF][RP], float2 *buf, int piece)
{
    if (r == 0 && pb == 0 && lane == 0) {
#pragma unroll
        for (int f = 0; f < NF; f++)
            v[f][0] = make_float2(0.f, 0.f);
    }
    if (r == p.corner_row) {
#pragma unroll
        for (int t = 0; t < RP; t++) {
            if (pb + t * 32 + lane == p.half) {
#pragma unroll
                for (int f = 0; f < NF; f++)
                    if (p.corner[f])
                        v[f][t] = make_float2((float)*p.corner[f], 0.f);
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < RP; t++) {
#pragma unroll
        for (int f = 0; f < NF; f++)
            buf[f * piece + t * 32 + lane] = v[f][t];
    }
    __syncwarp();
}

// Work split: each warp takes a contiguous block of (i, j) rows; a row is
// walked in pieces of 32*RP modes, the next piece's loads in flight while the
// current one is binned.  Lane l bins the contiguous run [l*RP, (l+1)*RP) of a
// piece (RP odd: conflict-free strided shared reads) with a running FP32 sum
// per spectrum pair.  Along a run |k|^2 grows, so the bin only moves up: the
// next threshold is kept in a register and a completed bin inside a run is
// added to the warp's FP32 histogram.  Two lanes never complete the same bin at
// the same place of their runs (by then the upper lane has been past it for
// RP - 1 >= 2 modes), so with the lanes in step the adds are plain ones; an FP32
// shared atomic is a loop, and six pairs' loops at nearly every mode of a row
// were half of its instructions (three fields, six pairs on 512^3: 0.52 -> 0.42
// ms).  One pair's single atomic costs less than keeping the lanes in step.  At the end of a piece the lanes' open sums
// are combined by a segmented warp scan over their (non-decreasing) bins and
// each bin's last lane adds the total without atomics.  Every kPromoteRows
// rows the touched FP32 bins are promoted into the warp's FP64 histogram.
//
// Bound by instruction issue and, on small grids, by its CTAs' start and end
// (five rows a warp at N = 200): the stream of modes is 5 us of memory time
// there.  RP is a template argument so that a lane's loads, stores and run
// are unrolled at their true count - as a run-time value of up to 9 the
// staging registers alone held a CTA to 3 per SM (68 registers; now 54, 4 per
// SM and exactly two waves of the 1216 CTAs) and the row cost 509
// instructions (now 410).  With k_bin_finalize: N = 200 40.3 -> 30.7 us,
// N = 160 28.7 -> 22.5, N = 384 124 -> 96.
template <int NF, bool CROSS1, int RP>
__global__ void __launch_bounds__(256, NF == 1 ? 4 : 2)
    k_bin(BinParams p, const uint32_t *__restrict__ thr_g, const float *__restrict__ iw_g,
          double *__restrict__ partial)
{
    constexpr int NP = PairSet<NF, CROSS1>::NP;
    extern __shared__ __align__(16) unsigned char smem[];
    const int nrb = p.nrbins;
    constexpr int piece = 32 * RP;
    constexpr bool kPlain = NP > 1;
    const BinLayout L = bin_layout(nrb, p.hc, NP, NF, RP);
    uint32_t *thr = (uint32_t *)smem;
    float2 *izc = (float2 *)(smem + L.izc);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char *wbase = smem + L.warps + L.per_warp * wid;
    double *whist = (double *)(wbase + L.whist);
    float *rhist = (float *)(wbase + L.rhist);
    float2 *buf = (float2 *)(wbase + L.buf);

    for (int i = threadIdx.x; i <= nrb; i += blockDim.x)
        thr[i] = thr_g[i];  // thr[nrb] = 0xffffffff: the bin never runs past nrb-1
    for (int i = threadIdx.x; i < p.hc; i += blockDim.x)
        izc[i] = make_float2(iw_g[i], (i == 0 || i == p.half) ? 1.f : 2.f);
    for (int i = lane; i < NP * nrb; i += 32) {
        whist[i] = 0.0;
        rhist[i] = 0.f;
    }
    wait_previous();
#pragma unroll
    for (int f = 0; f < NF; f++) {
        p.f[f] = fresh(p.f[f]);
        p.corner[f] = fresh(p.corner[f]);
    }
    __syncthreads();

    const int64_t nrows = (int64_t)p.dims * p.dims;
    const int64_t gw = (int64_t)blockIdx.x * p.warps + wid;
    const int64_t nw = (int64_t)gridDim.x * p.warps;
    const int64_t per = (nrows + nw - 1) / nw;
    const int64_t r_begin = min(nrows, gw * per), r_end = min(nrows, r_begin + per);
    int i = (int)(r_begin / p.dims), j = (int)(r_begin - (int64_t)i * p.dims);
    int bmin = nrb, bmax = -1;  // bins touched since the last FP64 promotion
    int rows_since = 0;
    float2 v[NF][RP];
    if (r_begin < r_end)
        load_piece<NF, RP>(p, r_begin, 0, lane, v);
    for (int64_t r = r_begin; r < r_end; r++) {
        const int ki = kval_dev(i, p.dims), kj = kval_dev(j, p.dims);
        const uint32_t r2 = (uint32_t)(ki * ki + kj * kj);
        const float pxy = __ldg(iw_g + i) * __ldg(iw_g + j);
        for (int pb = 0; pb < p.hc; pb += piece) {
            stage_piece<NF, RP>(p, r, pb, lane, v, buf, piece);
            // next piece (this row's, or the next row's first) in flight
            if (pb + piece < p.hc)
                load_piece<NF, RP>(p, r, pb + piece, lane, v);
            else if (r + 1 < r_end)
                load_piece<NF, RP>(p, r + 1, 0, lane, v);

            const int kz0 = pb + lane * RP;
            int cb = nrb;  // key of a lane without modes: sorts after every bin
            float acc[NP];
#pragma unroll
            for (int s = 0; s < NP; s++)
                acc[s] = 0.f;
            uint32_t kk2 = r2 + (uint32_t)(kz0 * kz0), nx = 0;
            const int lim = min(RP, p.hc - kz0);  // <= 0: none
            const float2 *bl = buf + lane * RP;
            auto bin_mode = [&](int t) {
                if (kk2 >= nx) {
#pragma unroll
                    for (int s = 0; s < NP; s++) {
                        if (kPlain)
                            rhist[s * nrb + cb] += acc[s];
                        else
                            atomicAdd(&rhist[s * nrb + cb], acc[s]);
                        acc[s] = 0.f;
                    }
                    do {
                        cb++;
                        nx = thr[cb + 1];
                    } while (kk2 >= nx);
                }
                const int kz = kz0 + t;
                const float2 ic = izc[kz];
                const float pz = pxy * ic.x;
                const float p2 = pz * pz;
                const float w = ic.y * (p2 * p2);
                float2 fv[NF];
#pragma unroll
                for (int f = 0; f < NF; f++)
                    fv[f] = bl[f * piece + t];
                add_pairs<NF, CROSS1>(fv, w, acc);
                kk2 += (uint32_t)(2 * kz + 1);
            };
            if (lim > 0) {
                cb = bin_lookup(kk2, thr, nrb, p.bpu_half);
                bmin = min(bmin, cb);
                nx = thr[cb + 1];
                if (!kPlain) {
#pragma unroll
                    for (int t = 0; t < RP; t++) {
                        if (t >= lim)
                            break;
                        bin_mode(t);
                    }
                }
            }
            if (kPlain) {
#pragma unroll
                for (int t = 0; t < RP; t++) {
                    if (t < lim)
                        bin_mode(t);
                    if (t > 0)
                        __syncwarp();
                }
            }
            if (lim > 0)
                bmax = max(bmax, cb);
            // Segmented inclusive scan over lanes with equal open bin.
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int ku = __shfl_up_sync(0xffffffffu, cb, o);
#pragma unroll
                for (int s = 0; s < NP; s++) {
                    const float x = __shfl_up_sync(0xffffffffu, acc[s], o);
                    if (lane >= o && ku == cb)
                        acc[s] += x;
                }
            }
            const int kd = __shfl_down_sync(0xffffffffu, cb, 1);
            if (cb < nrb && (lane == 31 || kd != cb)) {
#pragma unroll
                for (int s = 0; s < NP; s++)
                    rhist[s * nrb + cb] += acc[s];
            }
            __syncwarp();
        }
        if (++j == p.dims) {
            j = 0;
            i++;
        }
        if (++rows_since == kPromoteRows || r + 1 == r_end) {
            rows_since = 0;
            const int lo = (int)__reduce_min_sync(0xffffffffu, (unsigned)bmin);
            const int hi = (int)__reduce_max_sync(0xffffffffu, (unsigned)(bmax + 1)) - 1;
            for (int b = lo + lane; b <= hi; b += 32) {
#pragma unroll
                for (int s = 0; s < NP; s++) {
                    whist[s * nrb + b] += (double)rhist[s * nrb + b];
                    rhist[s * nrb + b] = 0.f;
                }
            }
            __syncwarp();
            bmin = nrb;
            bmax = -1;
        }
    }
    __syncthreads();
    // CTA reduction in warp order -> one partial histogram per CTA.
    for (int k = threadIdx.x; k < p.np * nrb; k += blockDim.x) {
        double s = 0.0;
        for (int w = 0; w < p.warps; w++) {
            const double *wh = (const double *)(smem + L.warps + L.per_warp * w + L.whist);
            s += wh[k];
        }
        partial[(size_t)blockIdx.x * p.np * nrb + k] = s;
    }
}

// Modes per lane per piece (odd) for rows of hc modes.
inline int bin_rp(int hc)
{
    return hc <= 32 ? 1 : hc <= 96 ? 3 : hc <= 160 ? 5 : 9;
}

template <int NF, bool CROSS1>
cudaError_t launch_bin_rows(const BinParams &p, const BinDevice &d, double *partial, int ctas,
                            size_t smem, cudaStream_t stream)
{
    const int rp = bin_rp(p.hc);
    auto kern = rp == 1   ? k_bin<NF, CROSS1, 1>
                : rp == 3 ? k_bin<NF, CROSS1, 3>
                : rp == 5 ? k_bin<NF, CROSS1, 5>
                          : k_bin<NF, CROSS1, 9>;
    const cudaError_t err = ensure_dynamic_smem(kern, smem);
    if (err != cudaSuccess)
        return err;
    return launch_after(kern, ctas, 32 * p.warps, smem, stream, p, d.thr, d.iw, partial);
}

}  // namespace

}  // namespace genpk
