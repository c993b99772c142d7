// sparc_tt.cu -- travel-time adjoint source on the device (ADJOINT_SOURCE_FILT,
// driver.f90:1758-2238), FP64, for a batch of sources.
//
// The reference, per ridge filter ("mode") and per measured receiver i, windows the time
// derivative of the filtered synthetic at x_i, transforms it, multiplies by the filter and by
// exp(-i k x_i), transforms the whole (x, t) plane back and adds the result, scaled by
// -tau_i / (sum ccdot^2 dt), time-reversed into the adjoint source: one 2-D transform per
// receiver.  The sum over receivers is linear, and exp(-2 pi i k (i-1)/nx) is the forward DFT
// kernel of a point at x_i, so it equals one transform per mode:
//     adj_mode = Re IDFT2( filter * DFT2(c) ),  c(x_i, t) = con_i w_i(t) ccdot(x_i, t),
// with c zero at unmeasured x.  A filter is real; an even one (filter(-f, -k) = filter(f, k), as every ridge is)
// keeps real records real:
//   - synthetic and data share one transform as real and imaginary part (the data times a power of two of
//     each source, which keeps the rounding of either relative to itself);
//   - per mode one inverse transform gives both filtered records; a second, of the synthetic's spectrum, the
//     time derivative ccdot and, as imaginary part, the Gizon-Birch derivative.  With an even record count the
//     middle frequency makes ccdot complex, and the two derivatives take a transform each;
//   - only Re c enters adj_mode, and the filtered spectra of all modes are summed: one inverse transform at the end;
//   - with any other filter the picks and travel times see the real part of the filtered records, which is that of
//     the filter's even part; ccdot is complex and enters adj_mode whole, and the two derivatives take a transform
//     each.  The spectra's kernel notes such a filter, and the mode is run again for it;
//   - only measured columns are transformed along t (their tiles of a few columns, listed on the host).
// Per mode 3 transforms along x and 3 along t of the measured columns, where 4 and 7 of every column were taken.
//
// Fields are complex [nb][nt][nx] (x fastest).  x transforms: the register transforms of sparc_wfft.cuh (nx in
// the FFT table).  t transforms: any nt (the record count, 240 or 241 for 3600 steps -- 241 is prime): Bluestein's
// chirp-z transform on two power-of-two FFTs of length M >= 2 nt - 1 (nt <= 512), a direct DFT over 16-column tiles
// above that.  FFTW's transforms are unnormalised, and so are these.  FP64 throughout: bound by the
// double-precision pipe.
#include <cmath>
#include <string>
#include <vector>

#include "sparc_gb300.h"
#include "sparc_wfft.cuh"

namespace sparc {
int report_error(int code, const std::string &msg);
}
using namespace sparc;

namespace {

constexpr int TT_THREADS = 256;
constexpr int TT_COLS = 16;      // columns per block of the t transform
constexpr int TT_XWPB = 2;       // rows (warps) per block of the x transform
constexpr double TT_PI = 3.141592653589793;

// x transform of complex rows in place, sign -1 forward, +1 inverse (unnormalised).
template <int N, bool INV>
__global__ void __launch_bounds__(TT_XWPB *WARP) tt_fft_x_kernel(double2 *data, long long nrows, const double *twr,
                                                                 const double *twi)
{
    using W = WFft<double, N, false>;
    constexpr int V = W::V, L = W::L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x % L, slot = threadIdx.x / L;
    const long long first = (long long)blockIdx.x * (W::rows(TT_XWPB)) + slot;
    const bool valid = first < nrows;
    const RowExchange<double, N, L> ex{reinterpret_cast<double *>(smem_raw) + (size_t)slot * W::REGION, slot};
    double2 *d = data + (valid ? first : nrows - 1) * N + t;
    double re[V], im[V];
#pragma unroll
    for (int m = 0; m < V; m++) {
        const double2 v = d[L * m];
        re[m] = v.x;
        im[m] = v.y;
    }
    wfft_stages<double, N, V, false, 0, 1, INV, 0>(re, im, ex, twr, twi, t);
    if (!valid) return;
#pragma unroll
    for (int m = 0; m < V; m++) d[L * m] = make_double2(re[m], im[m]);
}

// A tile of columns that a t transform covers: source b, columns x0 .. x0 + width - 1.
struct TTTile {
    int b, x0;
};

// t transform of complex columns in place: column (b, x) of length nt, stride nx.
// wt[m] = exp(-2 pi i m / nt); inverse uses the conjugate.
__global__ void __launch_bounds__(TT_THREADS) tt_dft_t_kernel(double2 *data, const TTTile *tiles, int nt, int nx,
                                                              const double2 *wt, int inverse)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *tile = reinterpret_cast<double2 *>(smem_raw);  // [nt][TT_COLS]
    double2 *w = tile + (size_t)nt * TT_COLS;                // [nt]
    const int x0 = tiles[blockIdx.x].x0;
    double2 *base = data + (size_t)tiles[blockIdx.x].b * nt * nx + x0;
    for (int idx = threadIdx.x; idx < nt * TT_COLS; idx += TT_THREADS) {
        const int t = idx / TT_COLS, c = idx % TT_COLS;
        tile[idx] = (x0 + c < nx) ? base[(size_t)t * nx + c] : make_double2(0.0, 0.0);
    }
    for (int m = threadIdx.x; m < nt; m += TT_THREADS) {
        double2 v = wt[m];
        if (inverse) v.y = -v.y;
        w[m] = v;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nt * TT_COLS; idx += TT_THREADS) {
        const int k = idx / TT_COLS, c = idx % TT_COLS;
        double sr = 0.0, si = 0.0;
        int m = 0;
        for (int t = 0; t < nt; t++) {
            const double2 a = tile[t * TT_COLS + c], b = w[m];
            sr += a.x * b.x - a.y * b.y;
            si += a.x * b.y + a.y * b.x;
            m += k;
            if (m >= nt) m -= nt;
        }
        if (x0 + c < nx) base[(size_t)k * nx + c] = make_double2(sr, si);
    }
}

// t transform by Bluestein's chirp-z algorithm: nk = (n^2 + k^2 - (k-n)^2) / 2 turns the length-nt
// DFT into a convolution with the chirp b_m = exp(+i pi m^2 / nt), evaluated with two power-of-two
// FFTs of length M >= 2 nt - 1 (Bluestein, IEEE Trans. Audio Electroacoust. 18 (1970) 451-455):
//   X_k = w_k IFFT_M( FFT_M(x_n w_n) * FFT_M(b) )_k / M,   w_n = exp(-i pi n^2 / nt).
// The inverse transform is the conjugate of the forward one of the conjugate.  A block takes the COLS consecutive
// columns of a tile, WFft<M>::L threads each: the tile [nt][COLS] is loaded and stored row-contiguously (COLS x 16
// bytes per record) through the columns' exchange regions.
template <int M, int COLS>
__global__ void __launch_bounds__(COLS *WFft<double, M, false>::L)
    tt_bluestein_t_kernel(double2 *data, const TTTile *tiles, int nt, int nx, const double2 *chirp, const double2 *bhat,
                          const double *twr, const double *twi, int inverse)
{
    using W = WFft<double, M, false>;
    constexpr int V = W::V, L = W::L, SW = W::REGION + 1;  // odd: the columns' equal elements on distinct banks
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sm = reinterpret_cast<double *>(smem_raw);
    const int t = threadIdx.x % L, col = threadIdx.x / L;
    const int x0 = tiles[blockIdx.x].x0;
    double2 *base = data + (size_t)tiles[blockIdx.x].b * nt * nx + x0;
    const double cs = inverse ? -1.0 : 1.0;  // conjugation of the input and output for the inverse
    for (int idx = threadIdx.x; idx < nt * COLS; idx += COLS * L) {
        const int k = idx / COLS, c = idx % COLS;
        const RowExchange<double, M, L> ex{sm + (size_t)c * SW};
        double2 v = (x0 + c < nx) ? base[(size_t)k * nx + c] : make_double2(0.0, 0.0);
        v.y *= cs;
        const double2 w = chirp[k];
        ex.put<0>(k, v.x * w.x - v.y * w.y, v.x * w.y + v.y * w.x);
    }
    __syncthreads();
    const RowExchange<double, M, L> ex{sm + (size_t)col * SW, col};
    double re[V], im[V];
#pragma unroll
    for (int m = 0; m < V; m++) {
        re[m] = im[m] = 0.0;
        if (t + L * m < nt) ex.get<0>(t + L * m, re[m], im[m]);
    }
    wfft_stages<double, M, V, false, 0, 1, false, 0>(re, im, ex, twr, twi, t);
#pragma unroll
    for (int m = 0; m < V; m++) {
        const double2 b = bhat[t + L * m];
        const double ar = re[m], ai = im[m];
        re[m] = ar * b.x - ai * b.y;
        im[m] = ar * b.y + ai * b.x;
    }
    wfft_stages<double, M, V, false, 0, 1, true, 0>(re, im, ex, twr, twi, t);
    ex.sync();  // the transform's last reads of the region are done
    const double inv_m = 1.0 / (double)M;
#pragma unroll
    for (int m = 0; m < V; m++) {  // X_k = w_k c_k / M, back into the column's region
        const int k = t + L * m;
        if (k < nt) {
            const double2 w = chirp[k];
            const double ar = re[m] * inv_m, ai = im[m] * inv_m;
            ex.put<0>(k, ar * w.x - ai * w.y, (ar * w.y + ai * w.x) * cs);
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nt * COLS; idx += COLS * L) {
        const int k = idx / COLS, c = idx % COLS;
        if (x0 + c >= nx) continue;
        const RowExchange<double, M, L> ec{sm + (size_t)c * SW};
        double2 v;
        ec.get<0>(k, v.x, v.y);
        base[(size_t)k * nx + c] = v;
    }
}

// Angular frequencies of spectral row t: of the time derivative of driver.f90:2015-2017 (freqnu = distmat(nt) /
// (nt dt 60): index 0 at 0, upper half negative) and of COMPUTE_TT_GIZONBIRCH's derivative (driver.f90:913-917: zero
// at q = nt/2 and its mirror).
__device__ __forceinline__ double tt_omega(int t, int nt, double dt_min)
{
    const int d = (t > nt - t) ? -(nt - t) : t;
    return 2.0 * TT_PI * ((double)d / ((double)nt * dt_min * 60.0));
}
__device__ __forceinline__ double tt_omega_gb(int t, int nt, double dt_min)
{
    const int h = nt / 2, q = t < h ? t : t > nt - h ? -(nt - t) : 0;
    return 2.0 * TT_PI * (double)q / ((double)nt * dt_min);
}

// Per source: the power of two that brings the data's largest value to the synthetic's binary exponent, its inverse,
// and what stands in the imaginary part.  A transform rounds relative to the larger of its two parts, so a part that
// separate transforms would keep exactly (zero, or equal to the other one) is not taken from it: a source without a
// synthetic or without data then has no travel time (0 / 0, or no correlation peak), and data equal to the synthetic
// have a shift of exactly zero.
enum { TT_PACKED = 0, TT_NOT_FINITE, TT_ZERO, TT_EQUAL };  // else alone: u NaN, u = 0, u = u0
struct TTScale {
    double s, inv;
    int kind, pad;
};
// Largest |value| of both planes as bit patterns, and whether any value differs.
struct TTTop {
    unsigned long long synth, data, differ;
};

__global__ void __launch_bounds__(TT_THREADS) tt_max_kernel(const double *synth, const double *data, TTTop *top,
                                                            long long plane)
{
    const int b = blockIdx.y;
    const unsigned long long MAG = 0x7fffffffffffffffull;
    unsigned long long ms = 0, md = 0;
    bool differ = false;
    for (long long i = (long long)blockIdx.x * TT_THREADS + threadIdx.x; i < plane; i += (long long)gridDim.x * TT_THREADS) {
        const unsigned long long u = (unsigned long long)__double_as_longlong(synth[b * plane + i]),
                                 v = (unsigned long long)__double_as_longlong(data[b * plane + i]);
        ms = max(ms, u & MAG);
        md = max(md, v & MAG);
        differ |= u != v;
    }
    for (int o = 16; o > 0; o >>= 1) {
        ms = max(ms, __shfl_xor_sync(0xffffffffu, ms, o));
        md = max(md, __shfl_xor_sync(0xffffffffu, md, o));
    }
    differ = __any_sync(0xffffffffu, differ);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&top[b].synth, ms);
        atomicMax(&top[b].data, md);
        if (differ) atomicMax(&top[b].differ, 1ull);
    }
}

// Biased binary exponent of |v| (bits, not zero), of a subnormal as if it were normalised.
__device__ __forceinline__ int tt_exponent(unsigned long long bits)
{
    const int e = (int)(bits >> 52);
    return e ? e : 12 - __clzll((long long)bits);
}

__global__ void tt_scale_kernel(const TTTop *top, TTScale *scale, int nb)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const unsigned long long ms = top[b].synth, md = top[b].data, INF = 0x7ffull << 52;
    const int kind = md >= INF ? TT_NOT_FINITE : ms == 0 || md == 0 ? TT_ZERO : !top[b].differ ? TT_EQUAL : TT_PACKED;
    const int d = kind == TT_PACKED && ms < INF ? max(-1000, min(1000, tt_exponent(ms) - tt_exponent(md))) : 0;
    scale[b] = TTScale{__hiloint2double((1023 + d) << 20, 0), __hiloint2double((1023 - d) << 20, 0), kind, 0};
}

// Real records into one complex plane: synthetic + i scale data, the synthetic alone where they are not packed.
__global__ void __launch_bounds__(TT_THREADS) tt_load_kernel(const double *synth, const double *data, double2 *out,
                                                             const TTScale *scale, long long n, long long plane)
{
    const long long stride = (long long)gridDim.x * TT_THREADS;
    for (long long i = (long long)blockIdx.x * TT_THREADS + threadIdx.x; i < n; i += stride) {
        const TTScale c = scale[i / plane];
        out[i] = make_double2(synth[i], c.kind == TT_PACKED ? data[i] * c.s : 0.0);
    }
}

// The data's value at an element z of the filtered records.
__device__ __forceinline__ double tt_data(const TTScale &sc, const double2 &z)
{
    return sc.kind == TT_PACKED ? z.y * sc.inv : sc.kind == TT_ZERO ? 0.0 : sc.kind == TT_EQUAL ? z.x : nan("");
}

// The spectra of one mode from Z = DFT2(synth + i data): acc = filter Z (both filtered records after the
// inverse), and of the synthetic's spectrum S(k) = (Z(k) + conj Z(-k)) / 2: ccd = filter (i om S - om_gb S / 64),
// whose inverse is ccdot + i u0dot / 64 where both are real (odd nt, even filter), or (u0d given) ccdot and u0dot
// apart.  (In minutes u0dot is 60 times ccdot: the power of two keeps the rounding of either relative to itself.)
// acc and u0dot take the filter's even part, (f + f) / 2 = f of an even one: the real parts of the records.  odd: set
// where the filter is not even (null: ccd and u0d are not wanted).  One block per spectral row: its two frequencies
// cost a division each.
constexpr double TT_GB_SCALE = 64.0;
__global__ void __launch_bounds__(TT_THREADS) tt_mode_kernel(const double2 *Z, double2 *acc, double2 *ccd, double2 *u0d,
                                                             const double *filter, int *odd, int nt, int nx, double dt_min)
{
    __shared__ double w[2];
    const int b = blockIdx.x / nt, t = blockIdx.x - b * nt;
    if (threadIdx.x == 0) {
        w[0] = tt_omega(t, nt, dt_min);
        w[1] = tt_omega_gb(t, nt, dt_min);
    }
    __syncthreads();
    const double om = w[0], gb = u0d ? w[1] : w[1] * (1.0 / TT_GB_SCALE);
    const size_t row = ((size_t)b * nt + t) * nx, mt = t ? nt - t : 0, mirror = ((size_t)b * nt + mt) * nx;
    for (int x = threadIdx.x; x < nx; x += TT_THREADS) {
        const size_t i = row + x;
        const int mx = x ? nx - x : 0;
        const double f = filter[(size_t)t * nx + x], fm = filter[mt * nx + mx], e = 0.5 * (f + fm);
        const double2 z = Z[i];
        acc[i] = make_double2(z.x * e, z.y * e);
        if (!odd) continue;
        if (b == 0 && __double_as_longlong(f) != __double_as_longlong(fm)) *odd = 1;
        const double2 m = Z[mirror + mx];
        const double sr = 0.5 * (z.x + m.x), si = 0.5 * (z.y - m.y), cr = sr * f, ci = si * f;
        if (u0d) {
            ccd[i] = make_double2(-om * ci, om * cr);
            u0d[i] = make_double2(-gb * (si * e), gb * (sr * e));
        } else {
            ccd[i] = make_double2(-om * ci - gb * cr, om * cr - gb * ci);
        }
    }
}

// sum += filter * in, unless *skip.
__global__ void __launch_bounds__(TT_THREADS) tt_sum_kernel(const double2 *in, double2 *sum, const double *filter,
                                                            const int *skip, long long n, long long plane)
{
    if (skip && *skip) return;
    const long long stride = (long long)gridDim.x * TT_THREADS;
    for (long long i = (long long)blockIdx.x * TT_THREADS + threadIdx.x; i < n; i += stride) {
        const double f = filter[i % plane];
        const double2 v = in[i];
        double2 o = sum[i];
        o.x += v.x * f;
        o.y += v.y * f;
        sum[i] = o;
    }
}

// One measured receiver: b, x (0-based), search range [timest, timefin] (1-based, clipped),
// given window (lef, rig) or picked one; results: lef, rig, loc, tau, con.
struct TTRow {
    int b, x, timest, timefin, lef, rig, loc, pad;
    double tau, con;
};

// One warp per measured receiver (driver.f90:2040-2100): window pick (first maximum of
// |Re acc| over the search range), travel time by Simpson sums (SIMPSON_REGULAR weights over
// the whole record, integrals.f90:107-130) of w u0dot (u0 - u) and w u0dot^2, and the
// normalisation con = Re(-tau / (sum_{lef..rig} ccdot^2 dt)).  acc holds u0 + i scale u; ccdot the time
// derivative and, where u0dot is null, u0dot / TT_GB_SCALE as imaginary part.
__global__ void __launch_bounds__(TT_THREADS) tt_rows_kernel(TTRow *rows, int nrows, const double2 *acc,
                                                             const TTScale *scale, const double2 *u0dot,
                                                             const double2 *ccdot, int nt, int nx, int halftime,
                                                             int given, double dt_min)
{
    const int warp = (blockIdx.x * TT_THREADS + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= nrows) return;
    TTRow r = rows[warp];
    const size_t base = (size_t)r.b * nt * nx + r.x;
    auto at = [&](const double2 *f, int t) { return f[base + (size_t)t * nx]; };
    if (!given) {
        const int a = max(r.timest, 1), e = min(r.timefin, nt);
        double best = -1.0;
        int bi = a;
        for (int t = a + lane; t <= e; t += WARP) {
            const double v = fabs(at(acc, t - 1).x);
            if (v > best) { best = v; bi = t; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        r.loc = bi;
        r.lef = max(bi - halftime, 1);
        r.rig = min(bi + halftime, nt);
    }
    double num = 0.0, den = 0.0, sr = 0.0, si = 0.0;
    const TTScale sc = scale[r.b];
    for (int t = r.lef + lane; t <= r.rig; t += WARP) {  // 1-based t
        const double wgt = (t == 1 || t == nt) ? 1.0 : ((t % 2 == 0) ? 4.0 : 2.0);
        double2 c = at(ccdot, t - 1);
        const double2 z = at(acc, t - 1);
        double ud;
        if (u0dot) {
            ud = at(u0dot, t - 1).x;
        } else {
            ud = c.y * TT_GB_SCALE;
            c.y = 0.0;
        }
        const double u0 = z.x, u = tt_data(sc, z);
        num += wgt * (ud * (u0 - u));
        den += wgt * (ud * ud);
        sr += c.x * c.x - c.y * c.y;
        si += 2.0 * c.x * c.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        num += __shfl_xor_sync(0xffffffffu, num, o);
        den += __shfl_xor_sync(0xffffffffu, den, o);
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (lane == 0) {
        const double tau = num / den;  // both Simpson sums carry the same dt / 3
        const double dr = sr * dt_min, di = si * dt_min;
        r.tau = tau;
        r.con = -tau * dr / (dr * dr + di * di);  // Re(-tau / (dr + i di))
        rows[warp] = r;
    }
}

// MISFIT_ALL (driver.f90:2294-2651), one warp per measured receiver: window pick (first maximum
// of |Re acc| over the search range, window loc -+ halftime, not clipped), then COMPUTE_TT
// (driver.f90:855-890) on the window: the cross-correlation cc(i) = dt sum u0(k) u(k + i) for
// lags i in (-n, n), its first maximum, and the vertex of the parabola through the three samples
// around it.  tau = NaN marks a receiver that is not measured: a window leaving the record or a
// peak at the end of the lag range (the reference reads past its arrays there).
__global__ void __launch_bounds__(TT_THREADS) tt_cc_kernel(TTRow *rows, int nrows, const double2 *acc,
                                                           const TTScale *scale, int nt, int nx, int halftime,
                                                           int given, double dt_min)
{
    const int warp = (blockIdx.x * TT_THREADS + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= nrows) return;
    TTRow r = rows[warp];
    const size_t base = (size_t)r.b * nt * nx + r.x;
    const TTScale sc = scale[r.b];
    auto u0 = [&](int t0) { return acc[base + (size_t)t0 * nx].x; };  // 0-based record index
    auto u = [&](int t0) { return tt_data(sc, acc[base + (size_t)t0 * nx]); };
    if (!given) {
        const int a = max(r.timest, 1), e = min(r.timefin, nt);  // 1-based, clipped
        double best = -1.0;
        int bi = a;
        for (int t = a + lane; t <= e; t += WARP) {
            const double v = fabs(u0(t - 1));
            if (v > best) { best = v; bi = t; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        r.loc = bi;
        r.lef = bi - halftime;
        r.rig = bi + halftime;
    }
    double tau = nan("");
    if (r.lef >= 1 && r.rig <= nt && r.rig >= r.lef) {
        const int n = r.rig - r.lef + 1, w0 = r.lef - 1;  // window sample k (1..n) is record w0 + k - 1
        // cc at lag i = j - (n - 1): dt sum_k u0(k - min(i, 0)) u(k + max(i, 0)) over the overlap
        auto cc = [&](int j) {
            const int i = j - (n - 1);
            double c = 0.0;
            if (i <= 0) {
                for (int k = 1; k <= n + i; k++) c += u0(w0 + k - i - 1) * u(w0 + k - 1);
            } else {
                for (int k = 1; k <= n - i; k++) c += u0(w0 + k - 1) * u(w0 + k + i - 1);
            }
            return c * dt_min;
        };
        double best = -INFINITY;
        int bl = 2 * n;
        for (int j = lane; j <= 2 * n - 2; j += WARP) {
            const double c = cc(j);
            if (c > best) { best = c; bl = j; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bl, o);
            if (ob > best || (ob == best && oi < bl)) { best = ob; bl = oi; }
        }
        if (bl > 0 && bl < 2 * n - 2) {
            const double cm = cc(bl - 1), c0 = cc(bl), cp = cc(bl + 1);
            const double t0 = (double)(bl - (n - 1)) * dt_min;
            // parabola c = p0 + p1 t + p2 t^2 through (t0 - dt, t0, t0 + dt); tau = -p1 / (2 p2)
            const double p2 = (cm - 2.0 * c0 + cp) / (2.0 * dt_min * dt_min);
            const double p1 = (cp - cm) / (2.0 * dt_min) - 2.0 * p2 * t0;
            tau = -p1 * 0.5 / p2;
        }
    }
    if (lane == 0) {
        r.tau = tau;
        rows[warp] = r;
    }
}

// Re c(x_i, t) = con_i w_i(t) Re ccdot(x_i, t) at the measured receivers (the buffer is zeroed first); whole: c.
__global__ void __launch_bounds__(TT_THREADS) tt_scatter_kernel(const TTRow *rows, int nrows, const double2 *ccdot,
                                                                double2 *c, int nt, int nx, bool whole)
{
    const int warp = (blockIdx.x * TT_THREADS + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= nrows) return;
    const TTRow r = rows[warp];
    const size_t base = (size_t)r.b * nt * nx + r.x;
    for (int t = r.lef + lane; t <= r.rig; t += WARP) {
        c[base + (size_t)(t - 1) * nx].x += r.con * ccdot[base + (size_t)(t - 1) * nx].x;
        if (whole) c[base + (size_t)(t - 1) * nx].y += r.con * ccdot[base + (size_t)(t - 1) * nx].y;
    }
}

// out[b][nt-1-t][x] = s Re(field[b][t][x]) (time reversal, driver.f90:2097-2099).
__global__ void __launch_bounds__(TT_THREADS) tt_out_kernel(const double2 *f, double *out, int nt, int nx, long long n,
                                                            double s)
{
    const long long stride = (long long)gridDim.x * TT_THREADS;
    for (long long i = (long long)blockIdx.x * TT_THREADS + threadIdx.x; i < n; i += stride) {
        const long long plane = (long long)nt * nx;
        const long long b = i / plane, r = i - b * plane;
        const int t = (int)(r / nx), x = (int)(r - (long long)t * nx);
        out[b * plane + (long long)(nt - 1 - t) * nx + x] = f[i].x * s;
    }
}

unsigned tt_grid(long long n)
{
    const long long g = (n + TT_THREADS - 1) / TT_THREADS;
    return (unsigned)(g < 152LL * 8 ? g : 152LL * 8);
}

}  // namespace

struct sparc_tt_plan {
    int nx = 0, nt = 0, nb = 0;
    std::vector<void *> allocs;
    double2 *Z = nullptr, *ACC = nullptr, *CCD = nullptr, *U0D = nullptr, *C = nullptr, *ADJ = nullptr;
    double *twr = nullptr, *twi = nullptr;
    TTScale *scale = nullptr;
    TTTop *top = nullptr;
    TTTile *all = nullptr, *tiles = nullptr;  // every tile; those of the mode's measured columns
    int width = 0, nall = 0;                  // columns of a tile, tiles of the batch
    double2 *wt = nullptr;
    TTRow *rows = nullptr;  // of a call; in front of them one whose pad says that the mode's filter is not even
    int cap = 0;
    int bm = 0;  // Bluestein length (0: direct DFT along t)
    double2 *chirp = nullptr, *bhat = nullptr;
    double *btwr = nullptr, *btwi = nullptr;
};

namespace {

template <int N>
cudaError_t fft_x_n(sparc_tt_plan *p, double2 *f, int inverse, cudaStream_t st)
{
    const long long nrows = (long long)p->nb * p->nt;
    using W = WFft<double, N, false>;
    const int slots = W::rows(TT_XWPB);
    const size_t smem = (size_t)slots * W::REGION * sizeof(double);
    auto k = inverse ? tt_fft_x_kernel<N, true> : tt_fft_x_kernel<N, false>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(unsigned)((nrows + slots - 1) / slots), TT_XWPB * WARP, smem, st>>>(f, nrows, p->twr, p->twi);
    return cudaGetLastError();
}

cudaError_t fft_x(sparc_tt_plan *p, double2 *f, int inverse, cudaStream_t st)
{
#define CASE(n_) if (p->nx == n_) return fft_x_n<n_>(p, f, inverse, st);
    CASE(64) CASE(128) CASE(192) CASE(256) CASE(384) CASE(512) CASE(768) CASE(1024)
#undef CASE
    return cudaErrorInvalidValue;
}

size_t dft_t_smem(int nt) { return ((size_t)nt * TT_COLS + nt) * sizeof(double2); }

template <int M, int COLS>
cudaError_t bluestein_t(sparc_tt_plan *p, double2 *f, int inverse, const TTTile *tiles, int n, cudaStream_t st)
{
    using W = WFft<double, M, false>;
    const size_t smem = (size_t)COLS * (W::REGION + 1) * sizeof(double);
    auto k = tt_bluestein_t_kernel<M, COLS>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<n, COLS * W::L, smem, st>>>(f, tiles, p->nt, p->nx, p->chirp, p->bhat, p->btwr, p->btwi, inverse);
    return cudaGetLastError();
}

// Columns of a t transform's tile: Bluestein of length bm (0: the direct DFT).
// Bound by the double-precision pipe, so blocks of a few warps that spread evenly over the SMs: 155 tiles of 8
// columns (8 x 141 measured columns, length 512) took two waves of 152 SMs, 166 us; 2 columns are one 32-byte sector.
int tile_width(int bm) { return bm == 0 ? TT_COLS : bm >= 512 ? 2 : bm == 256 ? 4 : 8; }

cudaError_t dft_t(sparc_tt_plan *p, double2 *f, int inverse, const TTTile *tiles, int n, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    switch (p->bm) {
        case 64: return bluestein_t<64, 8>(p, f, inverse, tiles, n, st);
        case 128: return bluestein_t<128, 8>(p, f, inverse, tiles, n, st);
        case 256: return bluestein_t<256, 4>(p, f, inverse, tiles, n, st);
        case 512: return bluestein_t<512, 2>(p, f, inverse, tiles, n, st);
        case 1024: return bluestein_t<1024, 2>(p, f, inverse, tiles, n, st);
        default: break;
    }
    const size_t smem = dft_t_smem(p->nt);
    cudaError_t e = cudaFuncSetAttribute(tt_dft_t_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    tt_dft_t_kernel<<<n, TT_THREADS, smem, st>>>(f, tiles, p->nt, p->nx, p->wt, inverse);
    return cudaGetLastError();
}

// Spectra and records of one mode: acc (and with odd, see tt_mode_kernel, ccdot and, apart, u0dot) along x
// everywhere, along t on the tiles.
cudaError_t mode_records(sparc_tt_plan *p, const double *filter, double dt_min, int *odd, bool apart, int ntiles, cudaStream_t st)
{
    double2 *u0d = odd && apart ? p->U0D : nullptr;
    tt_mode_kernel<<<p->nb * p->nt, TT_THREADS, 0, st>>>(p->Z, p->ACC, p->CCD, u0d, filter, odd, p->nt, p->nx, dt_min);
    cudaError_t e = cudaGetLastError();
    double2 *f[3] = {p->ACC, odd ? p->CCD : nullptr, u0d};
    for (double2 *q : f) {
        if (!q) continue;
        if (e == cudaSuccess) e = fft_x(p, q, 1, st);
        if (e == cudaSuccess) e = dft_t(p, q, 1, p->tiles, ntiles, st);
    }
    return e;
}

// One mode of the adjoint source on the tiles of its rows h[1..] (h[0]: see sparc_tt_plan), which come back measured.
// whole: for a filter that is not even; without it such a filter leaves the adjoint source as it is and sets h[0].pad.
cudaError_t adjoint_mode(sparc_tt_plan *p, const double *filter, std::vector<TTRow> &h, int ntiles, int halftime, int given,
                         double dt_min, bool whole, cudaStream_t st)
{
    const int nt = p->nt, nx = p->nx, nrows = (int)h.size() - 1;
    const long long n = (long long)p->nb * nt * nx;
    const bool apart = whole || nt % 2 == 0;
    int *odd = &p->rows->pad;
    TTRow *rows = p->rows + 1;
    // filtered synthetic and data, the derivatives of the filtered synthetic (driver.f90:1990-2017, 905-923)
    cudaError_t e = mode_records(p, filter, dt_min, odd, apart, ntiles, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(rows, h.data() + 1, nrows * sizeof(TTRow), cudaMemcpyHostToDevice, st);
    const unsigned g = (unsigned)(((long long)nrows * WARP + TT_THREADS - 1) / TT_THREADS);
    if (e == cudaSuccess) {
        tt_rows_kernel<<<g, TT_THREADS, 0, st>>>(rows, nrows, p->ACC, p->scale, apart ? p->U0D : nullptr, p->CCD, nt, nx,
                                                 halftime, given, dt_min);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(p->C, 0, (size_t)n * sizeof(double2), st);
    if (e == cudaSuccess) {
        tt_scatter_kernel<<<g, TT_THREADS, 0, st>>>(rows, nrows, p->CCD, p->C, nt, nx, whole);
        e = cudaGetLastError();
    }
    // adj_mode = Re IDFT2(filter * DFT2(c)): its spectrum is summed (columns that are not measured are zero)
    if (e == cudaSuccess) e = dft_t(p, p->C, 0, p->tiles, ntiles, st);
    if (e == cudaSuccess) e = fft_x(p, p->C, 0, st);
    if (e == cudaSuccess) {
        tt_sum_kernel<<<tt_grid(n), TT_THREADS, 0, st>>>(p->C, p->ADJ, filter, whole ? nullptr : odd, n, (long long)nt * nx);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), p->rows, h.size() * sizeof(TTRow), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && whole) e = cudaMemsetAsync(odd, 0, sizeof(int), st);  // for the next mode
    const cudaError_t w = cudaStreamSynchronize(st);
    return e == cudaSuccess ? w : e;
}

// The tiles of the rows' columns (rows [nrows][7] as the caller gives them), uploaded; their number.
int row_tiles(sparc_tt_plan *p, const int *rows, int nrows, std::vector<TTTile> &list, cudaStream_t st, cudaError_t &e)
{
    const int per = (p->nx + p->width - 1) / p->width;
    std::vector<char> on((size_t)p->nb * per, 0);
    for (int r = 0; r < nrows; r++) on[(size_t)rows[7 * r] * per + rows[7 * r + 1] / p->width] = 1;
    list.clear();
    for (int b = 0; b < p->nb; b++)
        for (int i = 0; i < per; i++)
            if (on[(size_t)b * per + i]) list.push_back(TTTile{b, i * p->width});
    e = cudaSuccess;
    if (!list.empty())
        e = cudaMemcpyAsync(p->tiles, list.data(), list.size() * sizeof(TTTile), cudaMemcpyHostToDevice, st);
    return (int)list.size();
}

int tt_fail(const char *what, cudaError_t e)
{
    return report_error(SPARC_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

bool tt_nx_ok(int nx)
{
    return nx == 64 || nx == 128 || nx == 192 || nx == 256 || nx == 384 || nx == 512 || nx == 768 || nx == 1024;
}

}  // namespace

extern "C" {

int sparc_tt_plan_create(int nx, int nt, int nbatch, int max_rows, sparc_tt_plan_t **out)
{
    if (!out) return report_error(SPARC_ERR_ARG, "sparc_tt_plan_create: null argument");
    *out = nullptr;
    if (!tt_nx_ok(nx)) return report_error(SPARC_ERR_SIZE, "sparc_tt_plan_create: nx not in the FFT table");
    if (nt < 2 || dft_t_smem(nt) > 220 * 1024)
        return report_error(SPARC_ERR_SIZE, "sparc_tt_plan_create: nt must be in 2..860");
    if (nbatch < 1 || nbatch > 65535 || max_rows < 1) return report_error(SPARC_ERR_ARG, "sparc_tt_plan_create: bad batch");
    sparc_tt_plan *p = new sparc_tt_plan();
    p->nx = nx;
    p->nt = nt;
    p->nb = nbatch;
    p->cap = max_rows;
    const size_t n = (size_t)nbatch * nt * nx;
    // Bluestein length: the smallest power of two M >= 2 nt - 1 in the FFT table (64..1024)
    int M = 64;
    while (M < 2 * nt - 1) M *= 2;
    p->width = tile_width(M <= 1024 ? M : 0);
    p->nall = (nx + p->width - 1) / p->width * nbatch;
    struct Req { void **ptr; size_t bytes; };
    std::vector<Req> reqs = {
        {(void **)&p->Z, n * sizeof(double2)}, {(void **)&p->ACC, n * sizeof(double2)},
        {(void **)&p->CCD, n * sizeof(double2)}, {(void **)&p->U0D, n * sizeof(double2)},
        {(void **)&p->C, n * sizeof(double2)}, {(void **)&p->ADJ, n * sizeof(double2)},
        {(void **)&p->scale, nbatch * sizeof(TTScale)}, {(void **)&p->top, nbatch * sizeof(TTTop)},
        {(void **)&p->all, p->nall * sizeof(TTTile)}, {(void **)&p->tiles, p->nall * sizeof(TTTile)},
        {(void **)&p->twr, nx * sizeof(double)}, {(void **)&p->twi, nx * sizeof(double)},
        {(void **)&p->wt, nt * sizeof(double2)}, {(void **)&p->rows, ((size_t)max_rows + 1) * sizeof(TTRow)},
    };
    for (auto &r : reqs) {
        cudaError_t e = cudaMalloc(r.ptr, r.bytes);
        if (e != cudaSuccess) {
            sparc_tt_plan_destroy(p);
            return tt_fail("sparc_tt_plan_create: cudaMalloc", e);
        }
        p->allocs.push_back(*r.ptr);
    }
    std::vector<double> tr(nx), ti(nx);
    for (int t = 0; t < nx; t++) {
        tr[t] = std::cos(2.0 * TT_PI * (double)t / (double)nx);
        ti[t] = -std::sin(2.0 * TT_PI * (double)t / (double)nx);
    }
    std::vector<double2> w(nt);
    for (int m = 0; m < nt; m++) w[m] = make_double2(std::cos(2.0 * TT_PI * (double)m / (double)nt),
                                                     -std::sin(2.0 * TT_PI * (double)m / (double)nt));
    cudaError_t e = cudaMemcpy(p->twr, tr.data(), nx * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p->twi, ti.data(), nx * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p->wt, w.data(), nt * sizeof(double2), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(p->ADJ, 0, n * sizeof(double2));
    if (e == cudaSuccess) e = cudaMemset(p->rows, 0, sizeof(TTRow));
    std::vector<TTTile> every;
    for (int b = 0; b < nbatch; b++)
        for (int x0 = 0; x0 < nx; x0 += p->width) every.push_back(TTTile{b, x0});
    if (e == cudaSuccess) e = cudaMemcpy(p->all, every.data(), every.size() * sizeof(TTTile), cudaMemcpyHostToDevice);
    // Bluestein tables
    if (e == cudaSuccess && M <= 1024) {
        p->bm = M;
        std::vector<double2> ch(nt), bext(M, make_double2(0.0, 0.0)), bh(M);
        std::vector<double> btr(M), bti(M);
        for (int m = 0; m < nt; m++) {
            // n^2 mod 2 nt keeps the phase argument small (exp(-i pi n^2 / nt) has period 2 nt in n^2)
            const long long q = ((long long)m * m) % (2LL * nt);
            const double ang = TT_PI * (double)q / (double)nt;
            ch[m] = make_double2(std::cos(ang), -std::sin(ang));
            bext[m] = make_double2(std::cos(ang), std::sin(ang));
            if (m > 0) bext[M - m] = bext[m];
        }
        for (int t = 0; t < M; t++) {
            btr[t] = std::cos(2.0 * TT_PI * (double)t / (double)M);
            bti[t] = -std::sin(2.0 * TT_PI * (double)t / (double)M);
        }
        for (int k = 0; k < M; k++) {  // FFT_M(b) by a direct sum on the host (once per plan)
            double sr = 0.0, si = 0.0;
            for (int m = 0; m < M; m++) {
                const long long q = ((long long)k * m) % M;
                const double c = btr[q], sn = bti[q];
                sr += bext[m].x * c - bext[m].y * sn;
                si += bext[m].x * sn + bext[m].y * c;
            }
            bh[k] = make_double2(sr, si);
        }
        struct Req2 { void **ptr; size_t bytes; };
        Req2 r2[4] = {{(void **)&p->chirp, nt * sizeof(double2)}, {(void **)&p->bhat, M * sizeof(double2)},
                      {(void **)&p->btwr, M * sizeof(double)}, {(void **)&p->btwi, M * sizeof(double)}};
        for (auto &r : r2) {
            if (e == cudaSuccess) e = cudaMalloc(r.ptr, r.bytes);
            if (e == cudaSuccess) p->allocs.push_back(*r.ptr);
        }
        if (e == cudaSuccess) e = cudaMemcpy(p->chirp, ch.data(), nt * sizeof(double2), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(p->bhat, bh.data(), M * sizeof(double2), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(p->btwr, btr.data(), M * sizeof(double), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(p->btwi, bti.data(), M * sizeof(double), cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess) {
        sparc_tt_plan_destroy(p);
        return tt_fail("sparc_tt_plan_create: tables", e);
    }
    *out = p;
    return SPARC_OK;
}

int sparc_tt_plan_destroy(sparc_tt_plan_t *p)
{
    if (!p) return SPARC_OK;
    for (void *q : p->allocs) cudaFree(q);
    delete p;
    return SPARC_OK;
}

int sparc_tt_set_records(sparc_tt_plan_t *p, const double *synth, const double *data, void *stream)
{
    if (!p || !synth || !data) return report_error(SPARC_ERR_ARG, "sparc_tt_set_records: null argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long n = (long long)p->nb * p->nt * p->nx;
    // real records into one complex plane, then its forward 2-D transform (driver.f90:1840-1844)
    const long long plane = (long long)p->nt * p->nx;
    cudaError_t e = cudaMemsetAsync(p->top, 0, p->nb * sizeof(TTTop), st);
    if (e != cudaSuccess) return tt_fail("sparc_tt_set_records", e);
    tt_max_kernel<<<dim3(16, p->nb), TT_THREADS, 0, st>>>(synth, data, p->top, plane);
    tt_scale_kernel<<<(p->nb + 127) / 128, 128, 0, st>>>(p->top, p->scale, p->nb);
    tt_load_kernel<<<tt_grid(n), TT_THREADS, 0, st>>>(synth, data, p->Z, p->scale, n, plane);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = fft_x(p, p->Z, 0, st);
    if (e == cudaSuccess) e = dft_t(p, p->Z, 0, p->all, p->nall, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(p->ADJ, 0, (size_t)n * sizeof(double2), st);
    return e == cudaSuccess ? SPARC_OK : tt_fail("sparc_tt_set_records", e);
}

int sparc_tt_mode(sparc_tt_plan_t *p, const double *filter, int nrows, int *rows, int halftime, int given,
                  double dt_min, double *tau, void *stream)
{
    if (!p || !filter || nrows < 0 || nrows > p->cap || (nrows > 0 && (!rows || !tau)) || halftime < 0)
        return report_error(SPARC_ERR_ARG, "sparc_tt_mode: bad argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nt = p->nt, nx = p->nx;
    for (int r = 0; r < nrows; r++) {
        const int *q = rows + 7 * r;
        if (q[0] < 0 || q[0] >= p->nb || q[1] < 0 || q[1] >= nx || (given && (q[4] < 1 || q[5] > nt || q[4] > q[5])))
            return report_error(SPARC_ERR_ARG, "sparc_tt_mode: row out of range");
        if (!given && (max(q[2], 1) > min(q[3], nt)))
            return report_error(SPARC_ERR_ARG, "sparc_tt_mode: empty search range");
    }
    std::vector<TTRow> first(nrows + 1, TTRow{});
    for (int r = 0; r < nrows; r++) {
        const int *q = rows + 7 * r;
        first[r + 1] = TTRow{q[0], q[1], q[2], q[3], q[4], q[5], 0, 0, 0.0, 0.0};
    }
    cudaError_t e = cudaSuccess;
    std::vector<TTTile> list;
    const int ntiles = row_tiles(p, rows, nrows, list, st, e);
    std::vector<TTRow> h = first;
    if (nrows == 0) {
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    } else {
        if (e == cudaSuccess) e = adjoint_mode(p, filter, h, ntiles, halftime, given, dt_min, false, st);
        if (e == cudaSuccess && h[0].pad) {
            h = first;
            e = adjoint_mode(p, filter, h, ntiles, halftime, given, dt_min, true, st);
        }
    }
    if (e != cudaSuccess) return tt_fail("sparc_tt_mode", e);
    for (int r = 0; r < nrows; r++) {
        int *q = rows + 7 * r;
        q[4] = h[r + 1].lef;
        q[5] = h[r + 1].rig;
        q[6] = h[r + 1].loc;
        tau[r] = h[r + 1].tau;
    }
    return SPARC_OK;
}

int sparc_tt_misfit_mode(sparc_tt_plan_t *p, const double *filter, int nrows, int *rows, int halftime, int given,
                         double dt_min, double *tau, void *stream)
{
    if (!p || !filter || nrows < 0 || nrows > p->cap || (nrows > 0 && (!rows || !tau)) || halftime < 0)
        return report_error(SPARC_ERR_ARG, "sparc_tt_misfit_mode: bad argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nt = p->nt, nx = p->nx;
    const long long n = (long long)p->nb * nt * nx;
    std::vector<TTRow> h(nrows);
    for (int r = 0; r < nrows; r++) {
        const int *q = rows + 7 * r;
        if (q[0] < 0 || q[0] >= p->nb || q[1] < 0 || q[1] >= nx)
            return report_error(SPARC_ERR_ARG, "sparc_tt_misfit_mode: row out of range");
        if (!given && (max(q[2], 1) > min(q[3], nt)))
            return report_error(SPARC_ERR_ARG, "sparc_tt_misfit_mode: empty search range");
        h[r] = TTRow{q[0], q[1], q[2], q[3], q[4], q[5], 0, 0, 0.0, 0.0};
    }
    cudaError_t e = cudaSuccess;
    std::vector<TTTile> list;
    const int ntiles = row_tiles(p, rows, nrows, list, st, e);
    if (e == cudaSuccess && nrows > 0) e = mode_records(p, filter, dt_min, nullptr, false, ntiles, st);
    if (e == cudaSuccess && nrows > 0) {
        e = cudaMemcpyAsync(p->rows, h.data(), nrows * sizeof(TTRow), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) {
            const unsigned g = (unsigned)(((long long)nrows * WARP + TT_THREADS - 1) / TT_THREADS);
            tt_cc_kernel<<<g, TT_THREADS, 0, st>>>(p->rows, nrows, p->ACC, p->scale, nt, nx, halftime, given, dt_min);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), p->rows, nrows * sizeof(TTRow), cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return tt_fail("sparc_tt_misfit_mode", e);
    for (int r = 0; r < nrows; r++) {
        int *q = rows + 7 * r;
        q[4] = h[r].lef;
        q[5] = h[r].rig;
        q[6] = h[r].loc;
        tau[r] = h[r].tau;
    }
    return SPARC_OK;
}

int sparc_tt_adjoint(sparc_tt_plan_t *p, double *adj, void *stream)
{
    if (!p || !adj) return report_error(SPARC_ERR_ARG, "sparc_tt_adjoint: null argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long n = (long long)p->nb * p->nt * p->nx;
    cudaError_t e = cudaMemcpyAsync(p->C, p->ADJ, (size_t)n * sizeof(double2), cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = fft_x(p, p->C, 1, st);
    if (e == cudaSuccess) e = dft_t(p, p->C, 1, p->all, p->nall, st);
    if (e == cudaSuccess) {
        tt_out_kernel<<<tt_grid(n), TT_THREADS, 0, st>>>(p->C, adj, p->nt, p->nx, n, (double)p->nt / 60.0);  // driver.f90:2201
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? SPARC_OK : tt_fail("sparc_tt_adjoint", e);
}

}  // extern "C"
