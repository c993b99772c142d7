// sparc_adjoint.cu -- dense column operators for the discrete adjoint of the option-17 step.
//
// Every z-operator of the step acts on each x-column separately and linearly: the compact
// derivative dbyd2 with its boundary closures (dbyd2.f:8-235) times the stretch factor
// (derivatives.f90:10-24), and FILTER_VARS_2D's z filter (physics2d.f90:509-583).  The discrete
// adjoint needs their transposes, closures included; held as dense nz x nz FP64 matrices (built
// once per plan by applying the device operator to the columns of the identity), a transpose is
// a matrix-vector product per column with the transposed matrix.  FP64 throughout.
//
// The transposed step itself is fused: per stage one x pass (adj_row_kernel) and one z pass
// (adj_col_kernel), the counterparts of the forward row and column passes.  The x-derivative is
// antisymmetric; a transposed compact derivative R^T T^-T S is the partitioned solve of the transposed
// tridiagonal system (same chunks, factors of T^T) followed by the transposed stencil, O(nz) per column
// where the dense product was O(nz^2); the value of the solve at a preset row is the preset's adjoint.  FP64,
// bound by the double-precision pipe: the dense products alone took 600 operations per point and derivative.
// One reverse step of 256 x 300 on a GB300: 1.2 ms (0.45 of it the stages, where they are run again), 5.2 ms as about 2000
// kernels of single operators replayed from a graph.
#include <cuda_runtime.h>

#include <string>

#include "sparc_gb300.h"
#include "sparc_wfft.cuh"

namespace sparc {
int report_error(int code, const std::string &msg);
}

namespace {

constexpr int CM_X = 32;  // columns per block (one warp per output row: W[k][m] is broadcast)
constexpr int CM_Y = 8;   // output rows per block

// out[b][k][j] (+)= sum_m W[k][m] in[b][m][j] for columns i0 <= j <= i1; other columns copy in.
__global__ void __launch_bounds__(CM_X *CM_Y) colmat_kernel(const double *__restrict__ W, int nz,
                                                           const double *__restrict__ in, double *__restrict__ out,
                                                           int nx, int i0, int i1, int accumulate)
{
    const int j = blockIdx.x * CM_X + threadIdx.x;
    const int k = blockIdx.y * CM_Y + threadIdx.y;
    if (j >= nx || k >= nz) return;
    const size_t plane = (size_t)nz * nx;
    const double *ib = in + (size_t)blockIdx.z * plane;
    double v;
    if (j >= i0 && j <= i1) {
        const double *w = W + (size_t)k * nz;
        double s0 = 0.0, s1 = 0.0;
        int m = 0;
        for (; m + 1 < nz; m += 2) {
            s0 = fma(__ldg(w + m), __ldg(ib + (size_t)m * nx + j), s0);
            s1 = fma(__ldg(w + m + 1), __ldg(ib + (size_t)(m + 1) * nx + j), s1);
        }
        if (m < nz) s0 = fma(__ldg(w + m), __ldg(ib + (size_t)m * nx + j), s0);
        v = s0 + s1;
    } else {
        v = __ldg(ib + (size_t)k * nx + j);
    }
    double *o = out + (size_t)blockIdx.z * plane + (size_t)k * nx + j;
    *o = accumulate ? *o + v : v;
}

}  // namespace

namespace sparc {
namespace {

constexpr int ADJ_WARPS = 2;

// X pass of a transposed stage at one row: the adjoints of RHS v_x, v_z (cf lX, zero where the RHS is), the
// flow gradient -2 (lRvx d_x v_x + lRvz d_x v_z), d/dx of v0x lRvx and v0x lRvz, the x-PML of d p/dx and
// d/dx of lgpx; with it, sharing its transform, -d/dx of the previous stage's ldxx: that stage's lX of xi_x.
template <int N, int MODE>
__global__ void __launch_bounds__(ADJ_WARPS *WARP) adj_row_kernel(AdjArgs g)
{
    using W = WFft<double, N>;
    constexpr int V = W::V, L = W::L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const StepArgs<double> &a = g.a;
    const int t = threadIdx.x % L, slot = threadIdx.x / L;
    const int rows = a.nb * a.nz, first = blockIdx.x * (W::rows(ADJ_WARPS)) + slot;
    const bool valid = first < rows;
    const int row = valid ? first : rows - 1, b = row / a.nz, k = row - b * a.nz;
    const RowExchange<double, N> ex{reinterpret_cast<double *>(smem_raw) + (size_t)slot * W::REGION, slot};
    const size_t F = (size_t)a.nz * N, q0 = (size_t)k * N + t;
    const double *lX = g.lX + (size_t)b * 4 * F + q0;
    double re[V], im[V];
    RowScale<double> sr, si;
    auto derivative = [&]() {
        RowMax<double> mr, mi;
#pragma unroll
        for (int m = 0; m < V; m++) {
            mr.add(re[m]);
            mi.add(im[m]);
        }
        row_maxima(mr, mi, ex);
        sr = row_scale<double>(mr);
        si = row_scale<double>(mi);
#pragma unroll
        for (int m = 0; m < V; m++) {
            re[m] = scale_in(re[m], sr);
            im[m] = scale_in(im[m], si);
        }
        wfft_deriv<double, N, V, W::RADIX4>(re, im, ex, a.twr, a.twi, a.kap, a.stretchx, t);
    };
    double lvx[MODE == 2 ? 1 : V];
    if (MODE != 2) {
        const double *c0 = g.cache + (size_t)b * F + q0, *c2 = c0 + (size_t)2 * a.nb * F;
        double *gx = g.gx + (size_t)b * F + q0;
#pragma unroll
        for (int m = 0; m < V; m++) {
            const int x = t + L * m;
            const bool rim = k == 0 || x == 0 || x == N - 1;
            const double vx = rim ? 0.0 : g.cf * lX[2 * F + L * m], vz = rim ? 0.0 : g.cf * lX[3 * F + L * m];
            const double v0 = __ldg(a.v0x + q0 + L * m);
            lvx[m] = vx;
            re[m] = v0 * vx;
            im[m] = v0 * vz;
            if (valid) gx[L * m] += -2.0 * (vx * __ldg(c0 + L * m) + vz * __ldg(c2 + L * m));
        }
        derivative();
        double *D = g.D + (size_t)b * F + q0;
        if (valid) {
#pragma unroll
            for (int m = 0; m < V; m++) {
                D[L * m] = scale_out(re[m], sr);
                D[(size_t)a.nb * F + L * m] = scale_out(im[m], si);
            }
        }
    }
    const double ri = __ldg(a.rhoinv + k);
#pragma unroll
    for (int m = 0; m < V; m++) {
        const int x = t + L * m;
        double lg = 0.0;
        if (MODE != 2) {
            lg = -ri * lvx[m];
            if (x < a.nh || x >= N - a.nh) {
                const int ai = x < a.nh ? x : x - (N - a.nh) + a.nh;
                const size_t p = (((size_t)b * 2 + 1) * a.nz + k) * a.nhx + ai, pc = (size_t)k * a.nhx + ai;
                const double w = g.cf * g.lWw[p];
                lg += __ldg(a.ax + pc) * w;
                if (valid) {
                    const double ps = lg + __ldg(a.bx + pc) * w;
                    g.lWw[p] = ps;
                    g.lW[p] += ps;
                }
            }
        }
        re[m] = lg;
        im[m] = MODE == 0 ? 0.0 : __ldg(g.ldxx + (size_t)b * F + q0 + L * m);
    }
    derivative();
    if (!valid) return;
#pragma unroll
    for (int m = 0; m < V; m++) {
        if (MODE != 2) g.D[(size_t)2 * a.nb * F + (size_t)b * F + q0 + L * m] = scale_out(re[m], sr);
        if (MODE != 0) {
            const double l = -scale_out(im[m], si);
            g.la[(size_t)b * 4 * F + q0 + L * m] += l;
            if (MODE == 1) g.lX[(size_t)b * 4 * F + q0 + L * m] = l;
        }
    }
}

constexpr int ADJ_LMAX = 16;

// Transposed compact derivative of the column values y (already times the stretch): the transposed solve, its
// result z in the tile, then the transposed stencil of the chunk's rows.  top: z at the last row.
template <int CW>
__device__ __forceinline__ void adj_dzT(const ZTab<double> &tt, const ZTab<double> &tb, int nch, double *B, double *YB,
                                        int c, int j, int k0, int n, int nz, double (&y)[ADJ_LMAX], double &top)
{
    double prev = 0.0;
#pragma unroll
    for (int m = 0; m < ADJ_LMAX; m++) {
        if (m < n) {
            const int k = k0 + m;
            double v = y[m] * __ldg(tt.ib + k);
            if (m > 0) v -= __ldg(tt.lwib + k) * prev;
            y[m] = v;
            prev = v;
        }
    }
#pragma unroll
    for (int m = ADJ_LMAX - 2; m >= 0; m--)
        if (m + 1 < n) y[m] -= __ldg(tt.gm + k0 + m + 1) * y[m + 1];
    YB[(2 * j) * CW + c] = y[0];
    YB[(2 * j + 1) * CW + c] = prev;
    __syncthreads();  // also: every row of the tile of the solve before has been read
    double xl, xr;
    zcouple(tt, YB, CW, c, j, nch, xl, xr);
#pragma unroll
    for (int m = 0; m < ADJ_LMAX; m++)
        if (m < n) B[(k0 + m) * CW + c] = zcorrect(tt, y[m], k0 + m, xl, xr);
    __syncthreads();
    const double *z = B + c;
    top = z[(nz - 1) * CW];
#pragma unroll
    for (int m = 0; m < ADJ_LMAX; m++) {
        if (m < n) {
            const int k = k0 + m;  // rows 2 .. nz-3 of the stencil reach k from k -+ 1 and k -+ 2
            double r;
            if (k >= 4 && k <= nz - 5) {
                r = tb.c1 * (z[(k - 1) * CW] - z[(k + 1) * CW]) + tb.c2 * (z[(k - 2) * CW] - z[(k + 2) * CW]);
            } else {
                r = 0.0;
                auto row = [&](int q, double w) {
                    if (q >= 2 && q <= nz - 3) r += w * z[q * CW];
                };
                row(k - 1, tb.c1);
                row(k + 1, -tb.c1);
                row(k - 2, tb.c2);
                row(k + 2, -tb.c2);
            }
            if (k <= 4) r += __ldg(tb.w5 + k) * z[0] + __ldg(tb.w5 + 5 + k) * z[CW];
            if (k >= nz - 5) {
                const int i = k - (nz - 5);
                r += __ldg(tb.w5 + 5 * (nz - 2) + i) * z[(nz - 2) * CW] + __ldg(tb.w5 + 5 * (nz - 1) + i) * z[(nz - 1) * CW];
            }
            y[m] = r;
        }
    }
}

// Z pass of a transposed stage: the four transposed z-derivatives of a column tile and everything pointwise.
template <int CW>
__global__ void __launch_bounds__(CW * 32, 2) adj_col_kernel(AdjArgs g)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const StepArgs<double> &a = g.a;
    const int nz = a.nz, nx = a.nx, nch = a.nch;
    double *B = reinterpret_cast<double *>(smem_raw), *YB = B + (size_t)nz * CW;
    const int c = threadIdx.x % CW, j = threadIdx.x / CW, x = blockIdx.x * CW + c, b = blockIdx.y;
    const int k0 = j * a.L, n = min(a.L, nz - k0);
    const size_t F = (size_t)nz * nx, NF = (size_t)a.nb * F, col = (size_t)k0 * nx + x;
    double *lX = g.lX + (size_t)b * 4 * F + col, *la = g.la + (size_t)b * 4 * F + col;
    const double *D = g.D + (size_t)b * F + col, *cache = g.cache + (size_t)b * F + col;
    const double *v0z = a.v0z + col;
    const bool edge = x == 0 || x == nx - 1;
    const double cf = g.cf;
    auto lr = [&](int f, int m) { return edge || k0 + m == 0 ? 0.0 : cf * lX[f * F + (size_t)m * nx]; };
    double y[ADJ_LMAX], top;
    // ---- v_x: lvx = lRxix + 2 d_x(v0x lRvx) - 2 D_z^T(v0z lRvx)
#pragma unroll
    for (int m = 0; m < ADJ_LMAX; m++)
        if (m < n) y[m] = __ldg(v0z + (size_t)m * nx) * lr(2, m) * __ldg(a.stretch + k0 + m);
    adj_dzT<CW>(g.t1, a.z1, nch, B, YB, c, j, k0, n, nz, y, top);
    double lrvz[ADJ_LMAX];
#pragma unroll
    for (int m = 0; m < ADJ_LMAX; m++) {
        if (m < n) {
            const size_t q = (size_t)m * nx;
            const double vx = lr(2, m), vz = lr(3, m);
            lrvz[m] = vz;
            g.gz[(size_t)b * F + col + q] += -2.0 * (vx * __ldg(cache + NF + q) + vz * __ldg(cache + 3 * NF + q));
            const double l = lr(0, m) + 2.0 * __ldg(D + q) - 2.0 * y[m];
            lX[2 * F + q] = l;
            la[2 * F + q] += l;
            y[m] = __ldg(v0z + q) * vz * __ldg(a.stretch + k0 + m);
        }
    }
    // ---- v_z
    adj_dzT<CW>(g.t1, a.z1, nch, B, YB, c, j, k0, n, nz, y, top);
#pragma unroll
    for (int m = 0; m < ADJ_LMAX; m++) {
        if (m < n) {
            const size_t q = (size_t)m * nx;
            const int k = k0 + m;
            const double l = lr(1, m) + 2.0 * __ldg(D + NF + q) - 2.0 * y[m];
            lX[3 * F + q] = l;
            la[3 * F + q] += l;
            // the pressure gradient along z and its PML
            double lg = -__ldg(a.rhoinv + k) * lrvz[m];
            const int pi = pml_row(a, k);
            if (pi >= 0) {
                const size_t p = (((size_t)b * 2 + 1) * a.nzpml + pi) * nx + x, pc = (size_t)pi * nx + x;
                const double w = cf * g.lZw[p], ps = lg + __ldg(a.bz + pc) * w;
                lg += __ldg(a.az + pc) * w;
                g.lZw[p] = ps;
                g.lZ[p] += ps;
            }
            y[m] = lg * __ldg(a.stretch + k);
        }
    }
    // ---- p: lp = D_z^T lgpz - d_x lgpx; div and the buoyancy
    adj_dzT<CW>(g.t2, a.z2, nch, B, YB, c, j, k0, n, nz, y, top);
#pragma unroll
    for (int m = 0; m < ADJ_LMAX; m++) {
        if (m < n) {
            const size_t q = (size_t)m * nx;
            const int k = k0 + m, pi = pml_row(a, k);
            const double fd = pi >= 0 ? __ldg(a.fdz + (size_t)pi * nx + x) : 1.0;
            const double lp = y[m] - __ldg(D + 2 * NF + q);
            const double lrho = -__ldg(a.rhoinv + k) * __ldg(a.g + k) * lrvz[m];
            const double c2r = a.c2d ? __ldg(a.c2rho0 + col + q) : __ldg(a.c2rho0 + k);
            const double ldiv = -__ldg(a.rho0 + k) * lrho - c2r * lp;
            g.gc[(size_t)b * F + col + q] += -(lp * __ldg(cache + 4 * NF + q));
            lrvz[m] = -(__ldg(a.gr0 + k) * fd) * lrho - (__ldg(a.gp0 + k) * fd) * lp;  // lxi_z so far
            double ldxx = ldiv, ldzz = ldiv;
            if (x < a.nh || x >= nx - a.nh) {
                const int ai = x < a.nh ? x : x - (nx - a.nh) + a.nh;
                const size_t p = (((size_t)b * 2) * nz + k) * a.nhx + ai, pc = (size_t)k * a.nhx + ai;
                const double w = cf * g.lWw[p];
                ldxx += __ldg(a.ax + pc) * w;
                const double ps = ldxx + __ldg(a.bx + pc) * w;
                g.lWw[p] = ps;
                g.lW[p] += ps;
            }
            if (pi >= 0) {
                const size_t p = (((size_t)b * 2) * a.nzpml + pi) * nx + x, pc = (size_t)pi * nx + x;
                const double w = cf * g.lZw[p], ps = ldiv + __ldg(a.bz + pc) * w;
                ldzz += __ldg(a.az + pc) * w;
                g.lZw[p] = ps;
                g.lZ[p] += ps;
            }
            g.ldxx[(size_t)b * F + col + q] = ldxx;
            y[m] = ldzz * __ldg(a.stretch + k);
        }
    }
    // ---- xi_z, and the top row's preset -d_x xi_x unstretch
    adj_dzT<CW>(g.t3, a.z3, nch, B, YB, c, j, k0, n, nz, y, top);
#pragma unroll
    for (int m = 0; m < ADJ_LMAX; m++) {
        if (m < n) {
            const size_t q = (size_t)m * nx;
            const double l = lrvz[m] + y[m];
            lX[F + q] = l;
            la[F + q] += l;
            if (k0 + m == nz - 1) g.ldxx[(size_t)b * F + col + q] -= g.unstretch_top * top;
        }
    }
}

// mu = F^T la for the z filter of FILTER_VARS_2D (rows k0 .. nz-2 of the filtered columns: the 11-point filter
// for 5 <= k <= nz-6, the two-point mean elsewhere), written to la and lX.  A block takes 8 columns of one field.
constexpr int ADJ_FCW = 8, ADJ_FT = 256;
__global__ void __launch_bounds__(ADJ_FT) adj_filter_kernel(AdjArgs g)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const StepArgs<double> &a = g.a;
    double *B = reinterpret_cast<double *>(smem_raw);
    const int nz = a.nz, nx = a.nx, c = threadIdx.x % ADJ_FCW, w = threadIdx.x / ADJ_FCW, x = blockIdx.x * ADJ_FCW + c;
    const size_t o = (size_t)blockIdx.y * nz * nx + x;
    for (int k = w; k < nz; k += ADJ_FT / ADJ_FCW) B[k * ADJ_FCW + c] = g.la[o + (size_t)k * nx];
    __syncthreads();
    const bool xf = a.filt_xall || ((x >= a.nh - 1) && (x <= nx - a.nh));
    const double h[6] = {0.75390625, 0.5 * 0.41015625, 0.5 * -0.234375, 0.5 * 0.087890625, 0.5 * -0.01953125,
                         0.5 * 0.001953125};
    for (int m = w; m < nz; m += ADJ_FT / ADJ_FCW) {
        double r = B[m * ADJ_FCW + c];
        if (xf) {
            r = 0.0;
#pragma unroll
            for (int d = -5; d <= 5; d++) {  // what row k = m + d of the filter takes from row m
                const int k = m + d, e = d < 0 ? -d : d;
                if (k < 0 || k >= nz) continue;
                const bool eleven = k >= 5 && k <= nz - 6, done = k >= a.filt_k0 && k <= nz - 2;
                const double v = !done ? (e == 0 ? 1.0 : 0.0) : eleven ? h[e] : (e == 1 ? 0.5 : 0.0);
                if (v != 0.0) r += v * B[k * ADJ_FCW + c];
            }
        }
        g.la[o + (size_t)m * nx] = r;
        g.lX[o + (size_t)m * nx] = r;
    }
}

__global__ void adj_tables_kernel(int *time, int *idx, double *w, double *inj, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) inj[i] = 1.0;
    if (i < 7) w[i] = i == 0 ? 1.0 : 0.0;
    if (i == 0) {
        *time = -1;  // the first row pass of the step advances it to 0
        *idx = 0;
    }
}

template <int N>
cudaError_t adj_row_n(const AdjArgs &g, int mode, cudaStream_t st)
{
    using W = WFft<double, N>;
    const int rows = g.a.nb * g.a.nz, slots = W::rows(ADJ_WARPS);
    const size_t smem = (size_t)slots * W::REGION * sizeof(double);
    auto k = mode == 0 ? adj_row_kernel<N, 0> : mode == 1 ? adj_row_kernel<N, 1> : adj_row_kernel<N, 2>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(rows + slots - 1) / slots, ADJ_WARPS * WARP, smem, st>>>(g);
    return cudaGetLastError();
}

template <int CW>
cudaError_t adj_col_cw(const AdjArgs &g, cudaStream_t st)
{
    const size_t smem = ((size_t)g.a.nz * CW + (size_t)2 * g.a.nch * CW) * sizeof(double);
    auto k = adj_col_kernel<CW>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<dim3(g.a.nx / CW, g.a.nb), CW * g.a.nch, smem, st>>>(g);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_adj_row(const AdjArgs &g, int mode, cudaStream_t st)
{
#define CASE(n_) if (g.a.nx == n_) return adj_row_n<n_>(g, mode, st);
    CASE(64) CASE(128) CASE(192) CASE(256) CASE(384) CASE(512) CASE(768) CASE(1024)
#undef CASE
    return cudaErrorInvalidValue;
}

// Block width as the plan's column pass (column_geometry), 8 where that is wider.
cudaError_t launch_adj_col(const AdjArgs &g, cudaStream_t st)
{
    if (g.a.nx % 8 || g.a.L > ADJ_LMAX || g.a.nch > 32) return cudaErrorInvalidValue;
    if (g.a.colw == 2) return adj_col_cw<2>(g, st);
    if (g.a.colw == 4) return adj_col_cw<4>(g, st);
    return adj_col_cw<8>(g, st);
}

cudaError_t launch_adj_filter(const AdjArgs &g, cudaStream_t st)
{
    const size_t smem = (size_t)g.a.nz * ADJ_FCW * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(adj_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    adj_filter_kernel<<<dim3(g.a.nx / ADJ_FCW, 4 * g.a.nb), ADJ_FT, smem, st>>>(g);
    return cudaGetLastError();
}

cudaError_t launch_adj_tables(int *time, int *idx, double *w, double *inj, int n, cudaStream_t st)
{
    adj_tables_kernel<<<(n + 255) / 256, 256, 0, st>>>(time, idx, w, inj, n);
    return cudaGetLastError();
}

}  // namespace sparc

extern "C" int sparc_colmat_apply(const double *W, int nz, const double *in, double *out, int nb, int nx, int i0,
                                  int i1, int accumulate, void *stream)
{
    if (!W || !in || !out || nz < 1 || nb < 1 || nx < 1 || in == out)
        return sparc::report_error(SPARC_ERR_ARG, "sparc_colmat_apply: null, empty or aliased argument");
    if (nb > 65535 || (nz + CM_Y - 1) / CM_Y > 65535)
        return sparc::report_error(SPARC_ERR_SIZE, "sparc_colmat_apply: grid too large");
    dim3 grid((nx + CM_X - 1) / CM_X, (nz + CM_Y - 1) / CM_Y, nb);
    colmat_kernel<<<grid, dim3(CM_X, CM_Y), 0, (cudaStream_t)stream>>>(W, nz, in, out, nx, i0, i1, accumulate);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SPARC_OK
                            : sparc::report_error(SPARC_ERR_CUDA, std::string("sparc_colmat_apply: ") + cudaGetErrorString(e));
}
