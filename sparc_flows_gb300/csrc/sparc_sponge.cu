// sparc_sponge.cu -- kernels of the 2-D velocity-pressure-density steps: option 5
// (MP_QUIET_SPONGE_2D, physics2d.f90:1099-1137, a sponge layer), option 6 (MP_QUIET_PML_2D,
// physics2d.f90:662-713, the vertical PML) and option 12 (MP_MHD_PML_2d, physics2d.f90:411-474,
// the same with a background magnetic field: b_x, b_z in the state, the induction equation,
// the Lorentz force, and the magnetic part of PML_BOUNDARY_ACCOUNTING_2D, 1162-1200).
//
// Fields are [nz][nb][nx] (level-major, the batch inside a level, as the 3-D step), the state
// five of them: rho, v_x, v_y, v_z, p (initialize.f90:500-504); with option 12 also b_x, b_y, b_z.  v_y and b_y
// are zero in 2-D and have no RHS: no pass touches them.  One RK stage is two passes, each forming the stage
// input A + beta SCR of the fields it needs as it reads them:
//   x pass (s5x_kernel)  d v_x/dx and d p/dx in one transform; with option 12 d flux/dx and d b_z/dx, the flux
//                        -(v_x boz - v_z box) formed on the way in
//   z pass (s5z_kernel)  the compact derivatives (ibc 1) of p and v_z (and of the flux and b_x) of a column tile in
//                        shared memory, then the whole right-hand side of the tile's rows, SCR in place
// End of step (s5_end_kernel): a += dt scr and FILTER_VARS_2D (physics2d.f90:509-560) from a column tile of one
// field in shared memory, in place.
#include "sparc_wfft.cuh"

namespace sparc {

constexpr int S5_THREADS = 256, S5X_WARPS = 2;

// ---- x pass: a unit of WFft::L threads is one row and one pair of fields (pair 1: option 12).  FP32 rows of 1024 columns:
// registers for eight blocks an SM (four solves of 300 levels 259 us a step against 268 without the limit).
template <typename T, int N>
constexpr int s5x_blocks() { return sizeof(T) == 4 && N == 1024 ? 8 : 0; }
template <typename T, int N>
__global__ void __launch_bounds__(S5X_WARPS *WARP, s5x_blocks<T, N>()) s5x_kernel(S5Step<T> a, S3Fft<T> f)
{
    using W = WFft<T, N>;
    constexpr int V = W::V, L = W::L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x % L, slot = threadIdx.x / L;
    const int rows = a.nz * a.nb, units = rows * (a.option == 12 ? 2 : 1);
    const int first = blockIdx.x * (W::rows(S5X_WARPS)) + slot;
    const bool valid = first < units;
    const int unit = valid ? first : units - 1, pair = unit / rows, row = unit - pair * rows;
    const RowExchange<T, N, L> ex{reinterpret_cast<T *>(smem_raw) + (size_t)slot * W::REGION, slot};
    const long long F = a.F, o = (long long)row * N + t;
    T re[V], im[V];
    auto load = [&](int fld, T(&v)[V]) {
#pragma unroll
        for (int m = 0; m < V; m++) v[m] = __ldg(a.A + fld * F + o + L * m);
        if (!a.first) {
#pragma unroll
            for (int m = 0; m < V; m++) v[m] = v[m] + a.b * __ldg(a.SCR + fld * F + o + L * m);
        }
    };
    load(1, re);  // v_x
    if (pair == 0) {
        load(4, im);  // p
    } else {
        T vz[V];
        load(3, vz);
        load(7, im);  // b_z
        const long long q = (long long)(row / a.nb) * N + t;
#pragma unroll
        for (int m = 0; m < V; m++) re[m] = -(re[m] * __ldg(a.bg.boz + q + L * m) - vz[m] * __ldg(a.bg.box + q + L * m));
    }
    RowMax<T> mr, mi;
#pragma unroll
    for (int m = 0; m < V; m++) {
        mr.add(re[m]);
        mi.add(im[m]);
    }
    row_maxima(mr, mi, ex);
    const RowScale<T> sr = row_scale<T>(mr), si = row_scale<T>(mi);
#pragma unroll
    for (int m = 0; m < V; m++) {
        re[m] = scale_in(re[m], sr);
        im[m] = scale_in(im[m], si);
    }
    wfft_deriv<T, N, V, W::RADIX4>(re, im, ex, f.twr, f.twi, f.kap, f.stretch, t);
    if (!valid) return;
    T *d = a.DX + 2 * pair * F + o;
#pragma unroll
    for (int m = 0; m < V; m++) {
        d[L * m] = scale_out(re[m], sr);
        d[F + L * m] = scale_out(im[m], si);
    }
}

// ---- z pass.  OPT 5: sponge (physics2d.f90:1099-1137), 6: vertical PML (662-713, 1142-1160), 12: with the
// magnetic field (411-474, 1162-1200: dv_z/dz with its PML term replaced on the PML rows 1..npmlbot-1 and
// nz-npmltop..nz-2 (0-based) by the mean of its two neighbours).  PML auxiliaries [npa][npml][nb][nx]: psi_p,
// psi_vz, psi_flux, psi_dzbx.  The top and bottom rows: zero RHS of momentum and pressure (5) or of all (6, 12).
// Thread (c, j): column c of the tile, the rows of chunk j.  The tiles hold the fields, then their derivatives.
constexpr int S5Z_LMAX = 16, S5Z_ROWS = 4;
template <typename T, int CW>
constexpr int s5z_nch() { return sizeof(T) == 8 && CW <= 8 ? 32 : 20; }

template <typename T, int CW, int OPT>
__global__ void __launch_bounds__(CW *s5z_nch<T, CW>()) s5z_kernel(S5Step<T> a, ZTab<T> z1, int nch, int LC)
{
    constexpr int NQ = OPT == 12 ? 4 : 2, LMAX = S5Z_LMAX, R = S5Z_ROWS;
    constexpr int NFLD = OPT == 12 ? 6 : 4;
    constexpr int fld[6] = {0, 1, 3, 4, 5, 7};  // rho, v_x, v_z, p, b_x, b_z
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *B = reinterpret_cast<T *>(smem_raw);
    const int nz = a.nz, c = threadIdx.x % CW, j = threadIdx.x / CW, k0 = j * LC, n = min(LC, nz - k0);
    const size_t tile = (size_t)nz * CW;
    T *YB = B + NQ * tile;
    const long long lvl = a.lvl, F = a.F, r = (long long)blockIdx.x * CW + c;
    const int x = (int)(r % a.nx);
    auto input = [&](int q, long long o) {
        const T v = a.A[q * F + o];
        return a.first ? v : v + a.b * a.SCR[q * F + o];
    };
#pragma unroll
    for (int m = 0; m < LMAX; m++) {
        if (m < n) {
            const int k = k0 + m;
            const long long o = (long long)k * lvl + r;
            const T vz = input(3, o);
            B[k * CW + c] = input(4, o);
            B[tile + k * CW + c] = vz;
            if (OPT == 12) {
                const long long q = (long long)k * a.nx + x;
                B[2 * tile + k * CW + c] = -(input(1, o) * __ldg(a.bg.boz + q) - vz * __ldg(a.bg.box + q));
                B[3 * tile + k * CW + c] = input(5, o);
            }
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int q = 0; q < NQ; q++) {
        T y[LMAX], xl, xr;
        T *yb = YB + (size_t)(q & 1) * 2 * nch * CW;
        const T last = zlocal<T, LMAX>(z1, B + q * tile, CW, c, k0, n, nz, T(0), y);
        yb[(2 * j) * CW + c] = y[0];
        yb[(2 * j + 1) * CW + c] = last;
        __syncthreads();  // the tile is read, the boundary values are there
        zcouple(z1, yb, CW, c, j, nch, xl, xr);
#pragma unroll
        for (int m = 0; m < LMAX; m++)
            if (m < n) B[q * tile + (k0 + m) * CW + c] = zcorrect(z1, y[m], k0 + m, xl, xr) * __ldg(a.stretch + k0 + m);
    }
    if (OPT != 5) {  // PML terms of the thread's rows
        const long long P = (long long)(a.npmlbot + a.npmltop) * lvl;
        for (int m = 0; m < n; m++) {
            const int k = k0 + m;
            const int pi = k < a.npmlbot ? k : k >= nz - a.npmltop ? a.npmlbot + (k - (nz - a.npmltop)) : -1;
            if (pi < 0) continue;
            const T az = __ldg(a.bg.az + pi), bz = __ldg(a.bg.bz + pi);
            for (int q = 0; q < NQ; q++) {
                const long long o = q * P + (long long)pi * lvl + r;
                T ps = a.PV[o];
                if (!a.first) ps = ps + a.b * a.SPV[o];
                T &d = B[q * tile + k * CW + c];
                a.SPV[o] = az * d + bz * ps;
                d = d + ps;
            }
        }
    }
    if (OPT == 12) __syncthreads();  // the smoothing reads the rows of the neighbouring chunks
#pragma unroll 1
    for (int m0 = 0; m0 < n; m0 += R) {
        T X[NFLD][R], D[NQ][R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            if (m0 + i < n) {
                const long long o = (long long)(k0 + m0 + i) * lvl + r;
#pragma unroll
                for (int v = 0; v < NFLD; v++) X[v][i] = input(fld[v], o);
#pragma unroll
                for (int q = 0; q < NQ; q++) D[q][i] = __ldg(a.DX + q * F + o);
            }
        }
#pragma unroll
        for (int i = 0; i < R; i++) {
            if (m0 + i < n) {
                const int k = k0 + m0 + i;
                const long long o = (long long)k * lvl + r;
                const T *b = B + k * CW + c;
                const T rho = X[0][i], vz = X[2][i], gx = D[1][i];
                const T gz = b[0];
                T dvz = b[tile];
                if (OPT == 12 && ((k >= 1 && k <= a.npmlbot - 1) || (k >= nz - a.npmltop && k <= nz - 2)))
                    dvz = T(0.5) * (b[tile - CW] + b[tile + CW]);
                const T ri = __ldg(a.bg.rhoinv + k), g = __ldg(a.bg.g + k);
                const T div = D[0][i] + dvz;
                const bool rim = k == 0 || k == nz - 1;
                T rc, rx, rz, rp;
                if (OPT == 5) {
                    const T sp = __ldg(a.bg.sponge + k);
                    rc = -__ldg(a.bg.gradrho0_z + k) * vz - __ldg(a.bg.rho0 + k) * div - sp * rho;
                    rx = -ri * gx - sp * X[1][i];
                    rz = -ri * gz - sp * vz;
                    rz = rz - rho * g * ri;
                    rp = -__ldg(a.bg.c2rho0 + k) * div - vz * __ldg(a.bg.gradp0_z + k) - sp * X[3][i];
                } else if (OPT == 6) {
                    rc = -__ldg(a.bg.rho0 + k) * div - __ldg(a.bg.gradrho0_z + k) * vz;
                    rp = -__ldg(a.bg.c2rho0 + k) * div - vz * __ldg(a.bg.gradp0_z + k);
                    rx = -ri * gx;
                    rz = -ri * (gz + rho * g);
                } else {
                    const long long q = (long long)k * a.nx + x;
                    const T bxs = X[4 % NFLD][i], bzs = X[5 % NFLD][i], cu = __ldg(a.bg.curl + q);
                    const T cur = b[3 % NQ * tile] - D[3 % NQ][i];
                    const T t1 = __ldg(a.bg.boz + q) * cur + bzs * cu;
                    const T t3 = -__ldg(a.bg.box + q) * cur - bxs * cu;
                    rc = -__ldg(a.bg.gradrho0_z + k) * vz - __ldg(a.bg.rho0 + k) * div;
                    rx = ri * (t1 - gx);
                    rz = ri * (t3 - gz);
                    rz = rz - ri * rho * g;
                    rp = -__ldg(a.bg.c2rho0 + k) * div - vz * __ldg(a.bg.gradp0_z + k);
                }
                if (abs(k - a.e_rad) <= 4) rz = rz + (__ldg(a.PAT + r) * a.amp) * __ldg(a.bg.source_dep + k);
                if (rim) {
                    if (OPT != 5) rc = T(0);
                    rx = rz = rp = T(0);
                }
                a.SCR[o] = rc;
                a.SCR[F + o] = rx;
                a.SCR[3 * F + o] = rz;
                a.SCR[4 * F + o] = rp;
                if (OPT == 12) {
                    a.SCR[5 * F + o] = rim ? T(0) : -b[2 % NQ * tile];
                    a.SCR[7 * F + o] = rim ? T(0) : D[2 % NQ][i];
                }
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(S5_THREADS) s5_axpy_kernel(long long n, T *__restrict__ Y, const T *__restrict__ X,
                                                             T a)
{
    const long long stride = (long long)gridDim.x * S5_THREADS;
    for (long long i = (long long)blockIdx.x * S5_THREADS + threadIdx.x; i < n; i += stride) Y[i] = Y[i] + a * X[i];
}

// End of step: a block takes CW columns of one field (those with a RHS), a += dt scr into a tile, then
// FILTER_VARS_2D in place: the 11-point filter on rows 5 .. nz-6 and two-point means on rows nz-5 .. nz-2 (0-based)
// for x in [i0, i1] (HORIZONTAL_PMLS).  One thread walking a column took 206 us at 8 x 512 x 300 FP32 (80 blocks).
template <typename T, int CW>
__global__ void __launch_bounds__(S5_THREADS) s5_end_kernel(S5Step<T> a)
{
    constexpr int ROWS = S5_THREADS / CW;
    constexpr int fld[6] = {0, 1, 3, 4, 5, 7};
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *B = reinterpret_cast<T *>(smem_raw);
    const int c = threadIdx.x % CW, w = threadIdx.x / CW, nz = a.nz, v = fld[blockIdx.y];
    const long long lvl = a.lvl, r = (long long)blockIdx.x * CW + c;
    const int x = (int)(r % a.nx);
    T *col = a.A + v * a.F + r;
    const T *sc = a.SCR + v * a.F + r;
#pragma unroll 4
    for (int k = w; k < nz; k += ROWS) B[k * CW + c] = col[(long long)k * lvl] + a.dt * __ldg(sc + (long long)k * lvl);
    __syncthreads();
    const bool xf = x >= a.i0 && x <= a.i1;
    const T c0 = T(0.75390625), h1 = T(0.5 * 0.41015625), h2 = T(0.5 * -0.234375), h3 = T(0.5 * 0.087890625),
            h4 = T(0.5 * -0.01953125), h5 = T(0.5 * 0.001953125);
#pragma unroll 2
    for (int k = w; k < nz; k += ROWS) {
        const T *b = B + k * CW + c;
        T out = b[0];
        if (xf && k >= 5 && k <= nz - 2) {
            if (k <= nz - 6)
                out = c0 * b[0] + h1 * (b[-CW] + b[CW]) + h2 * (b[-2 * CW] + b[2 * CW]) + h3 * (b[-3 * CW] + b[3 * CW]) +
                      h4 * (b[-4 * CW] + b[4 * CW]) + h5 * (b[-5 * CW] + b[5 * CW]);
            else
                out = T(0.5) * (b[CW] + b[-CW]);
        }
        col[(long long)k * lvl] = out;
    }
}

static unsigned s5_grid(long long n)
{
    const long long g = (n + S5_THREADS - 1) / S5_THREADS;
    return (unsigned)(g < 152LL * 16 ? g : 152LL * 16);
}

template <typename T, int N>
static cudaError_t s5x_n(const S5Step<T> &a, const S3Fft<T> &f, cudaStream_t st)
{
    using W = WFft<T, N>;
    const int units = a.nz * a.nb * (a.option == 12 ? 2 : 1), slots = W::rows(S5X_WARPS);
    const size_t smem = (size_t)slots * W::REGION * sizeof(T);
    auto k = s5x_kernel<T, N>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(units + slots - 1) / slots, S5X_WARPS * WARP, smem, st>>>(a, f);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_s5x(const S5Step<T> &a, const S3Fft<T> &f, cudaStream_t st)
{
#define CASE(n_) if (a.nx == n_) return s5x_n<T, n_>(a, f, st);
    CASE(64) CASE(128) CASE(192) CASE(256) CASE(384) CASE(512) CASE(768) CASE(1024)
#undef CASE
    return cudaErrorInvalidValue;
}

template <typename T, int CW, int OPT>
static cudaError_t s5z_cw(const S5Step<T> &a, const ZTab<T> &z1, int nch, int L, cudaStream_t st)
{
    if (a.lvl % CW || L > S5Z_LMAX || nch > s5z_nch<T, CW>()) return cudaErrorInvalidValue;
    const size_t smem = ((size_t)(OPT == 12 ? 4 : 2) * a.nz * CW + (size_t)4 * nch * CW) * sizeof(T);
    auto k = s5z_kernel<T, CW, OPT>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(unsigned)(a.lvl / CW), CW * nch, smem, st>>>(a, z1, nch, L);
    return cudaGetLastError();
}

template <typename T, int CW>
static cudaError_t s5z_option(const S5Step<T> &a, const ZTab<T> &z1, int nch, int L, cudaStream_t st)
{
    return a.option == 12 ? s5z_cw<T, CW, 12>(a, z1, nch, L, st)
                          : a.option == 6 ? s5z_cw<T, CW, 6>(a, z1, nch, L, st) : s5z_cw<T, CW, 5>(a, z1, nch, L, st);
}

template <typename T>
cudaError_t launch_s5z(const S5Step<T> &a, const ZTab<T> &z1, int nch, int L, int cw, cudaStream_t st)
{
    if constexpr (sizeof(T) == 8) {
        if (cw == 2) return s5z_option<T, 2>(a, z1, nch, L, st);
        if (cw == 4) return s5z_option<T, 4>(a, z1, nch, L, st);
    } else {
        if (cw == 32) return s5z_option<T, 32>(a, z1, nch, L, st);
    }
    return cw == 8 ? s5z_option<T, 8>(a, z1, nch, L, st) : cudaErrorInvalidValue;
}

template <typename T, int CW>
static cudaError_t s5_end_cw(const S5Step<T> &a, cudaStream_t st)
{
    const size_t smem = (size_t)a.nz * CW * sizeof(T);
    auto k = s5_end_kernel<T, CW>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<dim3((unsigned)(a.lvl / CW), a.option == 12 ? 6 : 4), S5_THREADS, smem, st>>>(a);
    return cudaGetLastError();
}

// Tile width: one 128-byte row segment where that gives two blocks per SM, else one 32-byte sector.
template <typename T>
cudaError_t launch_s5_end(const S5Step<T> &a, long long npv, cudaStream_t st)
{
    constexpr int WIDE = 128 / sizeof(T), NARROW = 32 / sizeof(T);
    const long long wide = a.lvl / WIDE * (a.option == 12 ? 6 : 4);
    const cudaError_t e = a.lvl % WIDE == 0 && wide >= 2 * 152 ? s5_end_cw<T, WIDE>(a, st) : s5_end_cw<T, NARROW>(a, st);
    if (e != cudaSuccess || npv == 0) return e;
    s5_axpy_kernel<T><<<s5_grid(npv), S5_THREADS, 0, st>>>(npv, a.PV, a.SPV, a.dt);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_s5_axpy(long long n, T *Y, const T *X, T a, cudaStream_t st)
{
    s5_axpy_kernel<T><<<s5_grid(n), S5_THREADS, 0, st>>>(n, Y, X, a);
    return cudaGetLastError();
}

#define S5_INST(T)                                                                                                   \
    template cudaError_t launch_s5x<T>(const S5Step<T> &, const S3Fft<T> &, cudaStream_t);                           \
    template cudaError_t launch_s5z<T>(const S5Step<T> &, const ZTab<T> &, int, int, int, cudaStream_t);             \
    template cudaError_t launch_s5_end<T>(const S5Step<T> &, long long, cudaStream_t);                               \
    template cudaError_t launch_s5_axpy<T>(long long, T *, const T *, T, cudaStream_t);
S5_INST(float)
S5_INST(double)
#undef S5_INST

}  // namespace sparc
