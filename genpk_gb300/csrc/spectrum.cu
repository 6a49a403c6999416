// spectrum.cu -- fused CIC deconvolution + log-k shell binning over the
// half-complex spectrum (the GPU counterpart of powerspectrum.c:35-111).
//
// Work split (k_bin, in bin_rows.cuh): each warp takes a contiguous block of
// (i, j) rows of N/2+1 modes, walked in pieces of 32*RP modes with the next
// piece's loads in flight.  Every lane bins a contiguous run of RP modes; bins only grow along a
// run, so a lane keeps one FP32 running sum per spectrum pair and compares
// |k|^2 with the next threshold held in a register.  The lanes' open sums are
// combined at the end of a piece by a segmented warp scan over their bins (no
// atomics); a bin completed inside a run (only where bins are narrower than a
// run) goes to the warp's FP32 histogram: with a shared atomic for one spectrum,
// by a plain add with the lanes in step for several.  Every 16 rows
// the touched bins are promoted into the warp's FP64 histogram.  At the end
// the CTA sums its warps in a fixed order and writes one FP64 partial
// histogram; k_bin_finalize sums the partials of all CTAs in a fixed order and
// normalises, so results do not depend on scheduling.
//
// Per mode (powerspectrum.c:55-91): bin = max{b : thr[b] <= |k|^2} with the
// integer thresholds built on the host from the reference's own bin
// expression, weight c = 1 on the kz = 0 and kz = N/2 planes, 2 elsewhere,
// (0,0,0) skipped; value = c * Re(F_a F_b*) * p^4 where p = (iw_x*iw_y)*iw_z is
// the float product of the per-axis inverse windows (fieldize.cpp:129-132) and
// p^4 = invwindow^2.  Counts and mean |k| per bin are pure geometry and come
// from the host tables.
#include "bin_rows.cuh"

#include <algorithm>

namespace genpk {
namespace {

// ---- binning of a kz-major spectrum (the N = 1024 transform) --------------
//
// The spectrum is stored as S[kz][x][y] (kz = 0..N/2, planes of N x N complex
// values; xfft.cu k_zfft_t1024 + a batched 2-D C2C).  Each (kz, x) row of N
// modes along y is binned as two half-rows along which |k|^2 grows: y = 0..N/2
// (ky = y) and y = N-1 down to N/2+1 (ky = y - N, |ky| = 1..N/2-1).  The rest
// is k_bin's: lane runs of RP modes with a running FP32 sum and the next
// threshold in a register, a segmented warp scan of the lanes' open sums,
// FP64 promotion every kPromoteRows half-rows, one FP64 partial histogram per
// CTA, k_bin_finalize.  Per mode: weight c = 1 on the kz = 0 and kz = N/2
// planes, 2 elsewhere; value c * p^4 |F|^2 with p = (iw_x iw_y) iw_z, the
// float product order of k_bin; (0,0,0) skipped; the exact corner value at
// (N/2, N/2, N/2).  One spectrum (its auto pair).
constexpr int kKzMaxRP = 9;

struct BinKzParams {
    const float2 *f;
    const double *corner;  // exact (N/2, N/2, N/2) value, or null
    int dims, half, hc;
    int nrbins;
    float bpu_half;
    int rp;     // modes per lane per piece (odd)
    int warps;  // warps per CTA
    uint4 *zero;          // region to clear (16-byte units), or null
    int64_t zero_units;
    int64_t zero_per_row; // units cleared per half-row
};

// Half-row r (physical row r/2 = kz * N + x, half r & 1): piece loads.
__device__ __forceinline__ void load_piece_kz(const BinKzParams &p, int64_t r, int pb, int lane,
                                              float2 (&v)[kKzMaxRP])
{
    const int h = (int)(r & 1);
    const int len = h ? p.half - 1 : p.hc;
    const float2 *row = p.f + (size_t)(r >> 1) * (size_t)p.dims;
#pragma unroll
    for (int t = 0; t < kKzMaxRP; t++) {
        const int m = pb + t * 32 + lane;
        const bool in = t < p.rp && m < len;
        const int y = h ? p.dims - 1 - m : m;
        v[t] = in ? __ldg(row + y) : make_float2(0.f, 0.f);
    }
}

__global__ void __launch_bounds__(256)
    k_bin_kz(BinKzParams p, const uint32_t *__restrict__ thr_g, const float *__restrict__ iw_g,
             double *__restrict__ partial)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int nrb = p.nrbins;
    const int rp = p.rp, piece = 32 * rp;
    const BinLayout L = bin_layout(nrb, p.hc, 1, 1, rp);
    uint32_t *thr = (uint32_t *)smem;
    float *iwy = (float *)(smem + L.izc);  // [dims]: 4 dims bytes fit the layout's 8 hc
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char *wbase = smem + L.warps + L.per_warp * wid;
    double *whist = (double *)(wbase + L.whist);
    float *rhist = (float *)(wbase + L.rhist);
    float2 *buf = (float2 *)(wbase + L.buf);

    for (int i = threadIdx.x; i <= nrb; i += blockDim.x)
        thr[i] = thr_g[i];
    for (int i = threadIdx.x; i < p.dims; i += blockDim.x)
        iwy[i] = iw_g[i];
    for (int i = lane; i < nrb; i += 32) {
        whist[i] = 0.0;
        rhist[i] = 0.f;
    }
    wait_previous();
    p.f = fresh(p.f);
    p.corner = fresh(p.corner);
    __syncthreads();

    const int64_t nrows = (int64_t)2 * p.hc * p.dims;  // half-rows
    const int64_t gw = (int64_t)blockIdx.x * p.warps + wid;
    const int64_t nw = (int64_t)gridDim.x * p.warps;
    const int64_t per = (nrows + nw - 1) / nw;
    const int64_t r_begin = min(nrows, gw * per), r_end = min(nrows, r_begin + per);
    int bmin = nrb, bmax = -1;
    int rows_since = 0;
    float2 v[kKzMaxRP];
    if (r_begin < r_end)
        load_piece_kz(p, r_begin, 0, lane, v);
    for (int64_t r = r_begin; r < r_end; r++) {
        const int h = (int)(r & 1);
        const int64_t pr = r >> 1;
        const int kz = (int)(pr / p.dims), x = (int)(pr - (int64_t)kz * p.dims);
        const int kx = kval_dev(x, p.dims);
        const uint32_t r2 = (uint32_t)(kx * kx + kz * kz);
        const float cw = (kz == 0 || kz == p.half) ? 1.f : 2.f;
        const float iwx = iwy[x], iwz = iwy[kz];
        const int len = h ? p.half - 1 : p.hc;
        const bool origin = kz == 0 && x == 0 && h == 0;
        const bool corner = p.corner && kz == p.half && x == p.half && h == 0;
        if (p.zero) {  // this half-row's share of the clear (nothing waits on it)
            const int64_t a0 = r * p.zero_per_row;
            const int64_t e0 = min(a0 + p.zero_per_row, p.zero_units);
            for (int64_t u = a0 + lane; u < e0; u += 32)
                __stcs(p.zero + u, make_uint4(0u, 0u, 0u, 0u));
        }
        for (int pb = 0; pb < len; pb += piece) {
            if (origin && pb == 0 && lane == 0)
                v[0] = make_float2(0.f, 0.f);
            if (corner) {
#pragma unroll
                for (int t = 0; t < kKzMaxRP; t++)
                    if (pb + t * 32 + lane == p.half)
                        v[t] = make_float2((float)*p.corner, 0.f);
            }
            __syncwarp();
#pragma unroll
            for (int t = 0; t < kKzMaxRP; t++)
                if (t < rp)
                    buf[t * 32 + lane] = v[t];
            __syncwarp();
            if (pb + piece < len)
                load_piece_kz(p, r, pb + piece, lane, v);
            else if (r + 1 < r_end)
                load_piece_kz(p, r + 1, 0, lane, v);

            const int m0 = pb + lane * rp;
            int cb = nrb;
            float acc = 0.f;
            if (m0 < len) {
                int ky = m0 + h;  // |ky| of the run's first mode
                uint32_t kk2 = r2 + (uint32_t)(ky * ky);
                cb = bin_lookup(kk2, thr, nrb, p.bpu_half);
                bmin = min(bmin, cb);
                uint32_t nx = thr[cb + 1];
                const int lim = min(rp, len - m0);
                const float2 *bl = buf + lane * rp;
                for (int t = 0; t < lim; t++) {
                    if (kk2 >= nx) {
                        atomicAdd(&rhist[cb], acc);
                        acc = 0.f;
                        do {
                            cb++;
                            nx = thr[cb + 1];
                        } while (kk2 >= nx);
                    }
                    const int m = m0 + t;
                    const int y = h ? p.dims - 1 - m : m;
                    const float pz = (iwx * iwy[y]) * iwz;
                    const float p2 = pz * pz;
                    const float w = cw * (p2 * p2);
                    const float2 fv = bl[t];
                    acc = fmaf(w, fmaf(fv.x, fv.x, fv.y * fv.y), acc);
                    kk2 += (uint32_t)(2 * ky + 1);
                    ky++;
                }
                bmax = max(bmax, cb);
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int ku = __shfl_up_sync(0xffffffffu, cb, o);
                const float xo = __shfl_up_sync(0xffffffffu, acc, o);
                if (lane >= o && ku == cb)
                    acc += xo;
            }
            const int kd = __shfl_down_sync(0xffffffffu, cb, 1);
            if (cb < nrb && (lane == 31 || kd != cb))
                rhist[cb] += acc;
            __syncwarp();
        }
        if (++rows_since == kPromoteRows || r + 1 == r_end) {
            rows_since = 0;
            const int lo = (int)__reduce_min_sync(0xffffffffu, (unsigned)bmin);
            const int hi = (int)__reduce_max_sync(0xffffffffu, (unsigned)(bmax + 1)) - 1;
            for (int b = lo + lane; b <= hi; b += 32) {
                whist[b] += (double)rhist[b];
                rhist[b] = 0.f;
            }
            __syncwarp();
            bmin = nrb;
            bmax = -1;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nrb; k += blockDim.x) {
        double sum = 0.0;
        for (int w = 0; w < p.warps; w++) {
            const double *wh = (const double *)(smem + L.warps + L.per_warp * w + L.whist);
            sum += wh[k];
        }
        partial[(size_t)blockIdx.x * nrb + k] = sum;
    }
}

struct NormParams {
    double ma[kMaxBinPairs], mb[kMaxBinPairs];
    int src[kMaxBinPairs];  // the partials' pair slot of each reported pair
    int npc;                // pair slots per CTA partial
};

// One block per (pair, bin): strided sums over the CTA partials, then a
// fixed-order tree, so the result does not depend on scheduling.  Bound by
// latency: the loads of a thread are issued eight at a time and added in their
// order, and the tree's last five levels are shuffles (1216 partials of a
// N = 200 pass: 9.7 -> 7.6 us).
constexpr int kFinalizeThreads = 256;

__global__ void __launch_bounds__(kFinalizeThreads)
    k_bin_finalize(const double *__restrict__ partial, int ctas, int nrbins,
                   const double *__restrict__ count, NormParams mn, double *__restrict__ power,
                   const DeviceStatus *__restrict__ st_in, DeviceStatus *__restrict__ st_out)
{
    wait_previous();
    partial = fresh(partial);
    st_in = fresh(st_in);
    if (st_out && blockIdx.x == 0 && threadIdx.x == 0)
        *st_out = *st_in;  // the pass's status words, beside the results
    __shared__ double sh[kFinalizeThreads];
    const int k = blockIdx.x;
    const int s = k / nrbins, b = k - s * nrbins;
    const size_t src = (size_t)mn.src[s] * nrbins + b;
    const double cnt = count[b];
    double part = 0.0;
    constexpr int U = 8;  // loads in flight; added in the CTAs' order
    for (int c0 = threadIdx.x; c0 < ctas; c0 += U * kFinalizeThreads) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int c = c0 + u * kFinalizeThreads;
            v[u] = c < ctas ? partial[(size_t)c * mn.npc * nrbins + src] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c0 + u * kFinalizeThreads < ctas)
                part += v[u];
    }
    sh[threadIdx.x] = part;
    __syncthreads();
    for (int w = kFinalizeThreads / 2; w >= 32; w >>= 1) {
        if (threadIdx.x < w)
            sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x >= 32)
        return;
    double acc = sh[threadIdx.x];
#pragma unroll
    for (int w = 16; w > 0; w >>= 1)  // (the tree's last levels)
        acc += __shfl_down_sync(0xffffffffu, acc, w);
    if (threadIdx.x != 0)
        return;
    double out = 0.0;
    if (cnt > 0.0) {
        out = acc / (mn.ma[s] * mn.mb[s]);
        out /= cnt;
    }
    power[k] = out;
}

size_t bin_smem(int nrbins, int hc, int np, int nf, int warps)
{
    const BinLayout L = bin_layout(nrbins, hc, np, nf, bin_rp(hc));
    return L.warps + L.per_warp * warps;
}

// Instantiated shapes: one field (its auto pair); two fields and one pair
// (the cross pair alone); else every pair of 2, 3 or 4 fields.  A request's
// pairs are found among the shape's by pair_slot.
struct Shape {
    int nf, np;
    bool cross1;
};

Shape pick_shape(int nf, int np)
{
    if (nf == 1)
        return {1, 1, false};
    if (nf == 2 && np == 1)
        return {2, 1, true};
    if (nf >= 2 && nf <= kMaxBinFields)
        return {nf, nf * (nf + 1) / 2, false};
    return {0, 0, false};
}

}  // namespace

int bin_pair_slots(int nfields, int npairs)
{
    return pick_shape(nfields, npairs).np;
}

int bin_ctas(const GridGeom &g, int nrbins, int npairs, int nfields, int num_sms, int *warps,
             size_t *smem)
{
    const Shape s = pick_shape(nfields, npairs);
    if (s.nf == 0)
        return 0;
    int w = 8;
    while (w > 1 && bin_smem(nrbins, g.hc, s.np, s.nf, w) > 200 * 1024)
        w /= 2;
    const size_t sm = bin_smem(nrbins, g.hc, s.np, s.nf, w);
    if (sm > 220 * 1024)
        return 0;
    *warps = w;
    *smem = sm;
    const int per_sm = std::max(1, std::min(2048 / (32 * w), (int)((220 * 1024) / sm)));
    const int64_t rows = (int64_t)g.dims * g.dims;
    const int64_t want = (rows + w - 1) / w;
    return (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)num_sms * per_sm, want));
}

cudaError_t bin_spectra(const GridGeom &g, const BinTables &t, const BinDevice &d,
                        const BinLaunch &l, double *partial, double *out_power, int ctas,
                        int warps, size_t smem, cudaStream_t stream, int64_t *launches,
                        const DeviceStatus *st_in, DeviceStatus *st_out)
{
    const Shape s = pick_shape(l.nfields, l.npairs);
    BinParams p;
    for (int f = 0; f < kMaxBinFields; f++) {
        p.f[f] = l.fields[f < l.nfields ? f : 0];
        p.corner[f] = l.corner[f < l.nfields ? f : 0];
    }
    p.corner_row = (g.dims % 2 == 0) ? (int64_t)g.half * g.dims + g.half : -1;
    p.np = s.np;
    p.dims = g.dims;
    p.hc = g.hc;
    p.half = g.half;
    p.nrbins = t.nrbins;
    p.bpu_half = (float)(0.5 * t.binsperunit);
    p.warps = warps;
    const cudaError_t err =
        s.nf == 1 ? bin_rows_single(p, d, partial, ctas, smem, stream)
                  : bin_rows_multi(s.nf, s.cross1, p, d, partial, ctas, smem, stream);
    (*launches)++;
    if (err != cudaSuccess)
        return err;
    NormParams mn;
    mn.npc = s.np;
    for (int q = 0; q < kMaxBinPairs; q++) {
        mn.ma[q] = q < l.npairs ? l.pairs[q].mass_a : 1.0;
        mn.mb[q] = q < l.npairs ? l.pairs[q].mass_b : 1.0;
        const int a = q < l.npairs ? std::min(l.pairs[q].a, l.pairs[q].b) : 0;
        const int b = q < l.npairs ? std::max(l.pairs[q].a, l.pairs[q].b) : 0;
        mn.src[q] = s.cross1 ? 0 : pair_slot(s.nf, a, b);
    }
    const int k = l.npairs * t.nrbins;
    (*launches)++;
    return launch_after(k_bin_finalize, k, kFinalizeThreads, 0, stream, partial, ctas, t.nrbins,
                        d.count, mn, out_power, st_in, st_out);
}

int bin_kz_ctas(const GridGeom &g, int nrbins, int num_sms, int *warps, size_t *smem)
{
    int w = 8;
    while (w > 1 && bin_smem(nrbins, g.hc, 1, 1, w) > 200 * 1024)
        w /= 2;
    const size_t sm = bin_smem(nrbins, g.hc, 1, 1, w);
    if (sm > 220 * 1024 || (size_t)4 * g.dims > align16(sizeof(float2) * g.hc))
        return 0;
    *warps = w;
    *smem = sm;
    const int per_sm = std::max(1, std::min(2048 / (32 * w), (int)((220 * 1024) / sm)));
    const int64_t rows = (int64_t)2 * g.hc * g.dims;
    const int64_t want = (rows + w - 1) / w;
    return (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)num_sms * per_sm, want));
}

cudaError_t bin_spectrum_kz(const GridGeom &g, const BinTables &t, const BinDevice &d,
                            const float2 *spec, const double *corner, double *partial, int ctas,
                            int warps, size_t smem, void *zero, int64_t zero_bytes,
                            cudaStream_t stream, int64_t *launches)
{
    BinKzParams p;
    p.f = spec;
    p.corner = (g.dims % 2 == 0) ? corner : nullptr;
    p.dims = g.dims;
    p.half = g.half;
    p.hc = g.hc;
    p.nrbins = t.nrbins;
    p.bpu_half = (float)(0.5 * t.binsperunit);
    p.rp = bin_rp(g.hc);
    p.warps = warps;
    p.zero = reinterpret_cast<uint4 *>(zero);
    p.zero_units = zero ? zero_bytes / 16 : 0;
    const int64_t half_rows = (int64_t)2 * g.hc * g.dims;
    p.zero_per_row = (p.zero_units + half_rows - 1) / half_rows;
    cudaError_t err;
    if ((err = ensure_dynamic_smem(k_bin_kz, smem)) != cudaSuccess)
        return err;
    (*launches)++;
    return launch_after(k_bin_kz, ctas, 32 * warps, smem, stream, p, d.thr, d.iw, partial);
}

cudaError_t finalize_power(const double *partial, int ctas, int nrbins, const double *count,
                           double ma, double mb, double *out, cudaStream_t stream,
                           int64_t *launches, const DeviceStatus *st_in, DeviceStatus *st_out)
{
    NormParams mn;
    mn.npc = 1;
    for (int q = 0; q < kMaxBinPairs; q++) {
        mn.ma[q] = q == 0 ? ma : 1.0;
        mn.mb[q] = q == 0 ? mb : 1.0;
        mn.src[q] = 0;
    }
    (*launches)++;
    return launch_after(k_bin_finalize, nrbins, kFinalizeThreads, 0, stream, partial, ctas, nrbins,
                        count, mn, out, st_in, st_out);
}

cudaError_t finalize_powers(const double *partial, int ctas, int nrbins, int nfields,
                            const double *count, const double *mass, double *out,
                            cudaStream_t stream, int64_t *launches, const DeviceStatus *st_in,
                            DeviceStatus *st_out)
{
    for (int f0 = 0; f0 < nfields; f0 += kMaxBinPairs) {
        const int k = std::min(kMaxBinPairs, nfields - f0);
        NormParams mn;
        mn.npc = nfields;
        for (int q = 0; q < kMaxBinPairs; q++) {
            mn.ma[q] = mn.mb[q] = q < k ? mass[f0 + q] : 1.0;
            mn.src[q] = q < k ? f0 + q : 0;
        }
        const bool last = f0 + k >= nfields;
        (*launches)++;
        const cudaError_t err = launch_after(k_bin_finalize, k * nrbins, kFinalizeThreads, 0, stream,
                                             partial, ctas, nrbins, count, mn,
                                             out + (size_t)f0 * nrbins, st_in,
                                             last ? st_out : nullptr);
        if (err != cudaSuccess)
            return err;
    }
    return cudaSuccess;
}

namespace {

// Bound by the link that brought the doubles (17 MB at 128^3: 0.1-0.2 ms; this
// pass 6 us): conversions run on the small FP64 pipe, in the copy's shadow.
__global__ void __launch_bounds__(256)
    k_doubles_to_floats(const double2 *__restrict__ in, float2 *__restrict__ out, size_t pairs)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < pairs;
         i += (size_t)gridDim.x * blockDim.x) {
        const double2 v = __ldcs(in + i);
        out[i] = make_float2(__double2float_rn(v.x), __double2float_rn(v.y));
    }
}

}  // namespace

// (n is even: whole complex values, 16-byte aligned)
cudaError_t doubles_to_floats(const double *in, float *out, size_t n, int num_sms,
                              cudaStream_t stream, int64_t *launches)
{
    const size_t pairs = n / 2;
    const unsigned ctas = (unsigned)std::min<size_t>((pairs + 255) / 256, (size_t)num_sms * 8);
    k_doubles_to_floats<<<ctas, 256, 0, stream>>>(reinterpret_cast<const double2 *>(in),
                                                  reinterpret_cast<float2 *>(out), pairs);
    (*launches)++;
    return cudaGetLastError();
}

}  // namespace genpk
