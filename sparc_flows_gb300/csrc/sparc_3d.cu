// sparc_3d.cu -- kernels of the 3-D displacement step (option 16, MP_FLOWS_PML_3D_DISPL,
// displacement.f90:377-477) for a batch of solves.
//
// Layout: every field is [nz][nb][ny][nx] -- level-major with the solves of the batch inside a
// level -- so that a z-derivative is one launch over nb*ny*nx columns of stride nb*ny*nx, an
// x-derivative one launch over nz*nb*ny rows, and a y-derivative one launch over nz*nb planes.
// The state is six such fields (xi_x, xi_y, xi_z, v_x, v_y, v_z), the vertical PML
// auxiliaries two fields of npml levels (psi_vz, psi_p).  Background profiles depend on z
// only; the flow fields v0 are [nz][ny][nx], shared by the batch.
//
// One RK stage s, with Xv the stage's velocities (step.f90:48-63: A_v + beta RHS of the stage before) and S
// the sum of the advection terms, is five passes, each doing the pointwise work of its direction:
//   x pass  (s3x_kernel)   d p/dx of stage s-1 completes its RHS of v_x and Xv_x; d xi_x/dx; v0x d_x Xv
//   y pass  (s3y_kernel)   d xi_y/dy; v0y d_y Xv
//   z pass  (s3z_div)      d xi_z/dz (ibc 1), z-PML psi_vz, div, p, rho'     (displacement.f90:396-416)
//   z pass  (s3z_rhs)      v0z d_z Xv (ibc 1), d p/dz (ibc 0), z-PML psi_p, buoyancy, source: RHS of v_z and
//                          the next Xv_z                                      (displacement.f90:419-474)
//   y pass  (s3y_kernel)   d p/dy: RHS of v_y and the next Xv_y
// and a last x pass completes v_x.  The RHS of xi is Xv (zero on the top and bottom rows, as every RHS), so
// no RHS is stored: Xv alternates between two slots, xi of stage s is A_xi + beta Xv_{s-1}.  The passes of
// the last stage write the new v into the state.
// End of step: xi += dt Xv and FILTER_VARS_3D_HORIZ_PML when due (s3_end_kernel, a column tile of one
// field in shared memory, in place), the PML auxiliaries, the record.
//
// A stage moves 47 words per point where the separate derivative, advection, divergence and RHS passes
// moved 75; the step is bound by HBM in FP32 and by the double-precision pipe in FP64.
#include "sparc_wfft.cuh"

namespace sparc {

constexpr int S3_THREADS = 256;

// ---------------------------------------------------------------------------------------------
// y-derivative: neighbouring threads are neighbouring x-columns, so every load and store of a plane is
// contiguous and goes straight between global memory and the registers of the transform.  A block takes
// 2 XL columns of one (level, solve) plane, columns x0 + c and x0 + XL + c sharing a transform as real and
// imaginary part; thread (c, t) holds y = t + L m of both (sparc_wfft.cuh), and the exchanges between the
// stages go through shared memory [NY][XL], free of bank conflicts.
template <typename T, int NY>
struct DdyCfg {
    static constexpr int V = NY == 512 ? 16 : WFft<T, NY>::V, L = NY / V;
    // columns of a 128-byte row segment; half of that where the threads of a block would be 1024
    static constexpr int XL = sizeof(T) == 4 && L < 32 ? 32 : 16;
    static constexpr int THREADS = L * XL;
    // resident blocks that the registers are limited for: FP32 is bound by memory and wants two
    static constexpr int BLOCKS = sizeof(T) == 4 && V == 8 ? 2 : 1;
    static constexpr size_t SMEM = ColExchange<T, NY, XL>::BYTES;
};

template <typename T, int NY>
__global__ void __launch_bounds__((DdyCfg<T, NY>::THREADS), (DdyCfg<T, NY>::BLOCKS)) ddy_kernel(const T *__restrict__ var, T *__restrict__ dvar,
                                                                      int nx, T stretchy, const T *twr, const T *twi,
                                                                      const T *kap)
{
    using C = DdyCfg<T, NY>;
    constexpr int XL = C::XL, V = C::V, L = C::L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RowMax<T> red[2][L][XL];
    const int c = threadIdx.x % XL, t = threadIdx.x / XL;
    // a last block that would pass the plane's end starts earlier and repeats columns (same values)
    const int x0 = min((int)blockIdx.x * 2 * XL, nx - 2 * XL);
    const T *src = var + (size_t)blockIdx.y * NY * nx + x0 + c;
    T *dst = dvar + (size_t)blockIdx.y * NY * nx + x0 + c;
    T re[V], im[V];
    RowMax<T> mr, mi;
#pragma unroll
    for (int m = 0; m < V; m++) {
        re[m] = src[(size_t)(t + L * m) * nx];
        im[m] = src[(size_t)(t + L * m) * nx + XL];
    }
#pragma unroll
    for (int m = 0; m < V; m++) {
        mr.add(re[m]);
        mi.add(im[m]);
    }
    red[0][t][c] = mr;
    red[1][t][c] = mi;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < L; j++) {
        mr.merge(red[0][j][c]);
        mi.merge(red[1][j][c]);
    }
    const RowScale<T> sr = row_scale<T>(mr), si = row_scale<T>(mi);
#pragma unroll
    for (int m = 0; m < V; m++) {
        re[m] = scale_in(re[m], sr);
        im[m] = scale_in(im[m], si);
    }
    const ColExchange<T, NY, XL> ex{reinterpret_cast<T *>(smem_raw), c};
    wfft_deriv<T, NY, V, WFft<T, NY>::RADIX4>(re, im, ex, twr, twi, kap, stretchy, t);
#pragma unroll
    for (int m = 0; m < V; m++) {
        dst[(size_t)(t + L * m) * nx] = scale_out(re[m], sr);
        dst[(size_t)(t + L * m) * nx + XL] = scale_out(im[m], si);
    }
}

template <typename T, int NY>
static cudaError_t ddy_n(const T *var, T *dvar, int nplanes, int nx, T stretchy, const T *twr, const T *twi,
                         const T *kap, cudaStream_t st)
{
    using C = DdyCfg<T, NY>;
    auto k = ddy_kernel<T, NY>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return e;
    dim3 grid((nx + 2 * C::XL - 1) / (2 * C::XL), nplanes);
    k<<<grid, C::THREADS, C::SMEM, st>>>(var, dvar, nx, stretchy, twr, twi, kap);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_ddy(const T *var, T *dvar, int nplanes, int nx, int ny, T stretchy, const T *twr, const T *twi,
                       const T *kap, cudaStream_t st)
{
    if (nplanes <= 0) return cudaSuccess;
    if (nx < 64 || nx % 16) return cudaErrorInvalidValue;
    if (nplanes > 65535) return cudaErrorInvalidValue;
#define CASE(n_) if (ny == n_) return ddy_n<T, n_>(var, dvar, nplanes, nx, stretchy, twr, twi, kap, st);
    CASE(64) CASE(128) CASE(192) CASE(256) CASE(384)
    if constexpr (sizeof(T) == 4) { CASE(512) }
#undef CASE
    return cudaErrorInvalidValue;
}

bool ddy_size_supported(int ny)
{
    return ny == 64 || ny == 128 || ny == 192 || ny == 256 || ny == 384 || ny == 512;
}

// ---------------------------------------------------------------------------------------------
// PML level of row k (-1 outside the vertical PML).
template <typename T>
__device__ __forceinline__ int s3_pml(const S3Step<T> &a, int k)
{
    if (k < a.npmlbot) return k;
    if (k >= a.nz - a.npmltop) return a.npmlbot + (k - (a.nz - a.npmltop));
    return -1;
}

// ---------------------------------------------------------------------------------------------
// The stage passes.  Rows k = 0 and nz - 1 carry no RHS: Xv and xi of those rows are A's.
// ---------------------------------------------------------------------------------------------
// X pass: thread group of WFft lanes, two consecutive rows (same level and solve).  MODE 0: first stage (no
// pressure yet, Xv = A_v); 1: later stages; 2: after the last stage, d p/dx and the new v_x.  The four
// fields (p, xi_x and Xv_x, Xv_y) of a row share two transforms, Xv_z of both rows a third.
template <typename T, int N, int V>
struct S3Pair {  // one transform: two real rows, their scales
    T re[V], im[V];
    RowScale<T> sr, si;
    __device__ __forceinline__ T dre(int m) const { return scale_out(re[m], sr); }
    __device__ __forceinline__ T dim(int m) const { return scale_out(im[m], si); }
};

template <typename T, int N, int V, int L>
__device__ __forceinline__ void s3x_deriv(S3Pair<T, N, V> &p, const RowExchange<T, N> &ex, const S3Fft<T> &f, int t)
{
    RowMax<T> mr, mi;
#pragma unroll
    for (int m = 0; m < V; m++) {
        mr.add(p.re[m]);
        mi.add(p.im[m]);
    }
    row_maxima(mr, mi, ex);
    p.sr = row_scale<T>(mr);
    p.si = row_scale<T>(mi);
#pragma unroll
    for (int m = 0; m < V; m++) {
        p.re[m] = scale_in(p.re[m], p.sr);
        p.im[m] = scale_in(p.im[m], p.si);
    }
    wfft_deriv<T, N, V, WFft<T, N>::RADIX4>(p.re, p.im, ex, f.twr, f.twi, f.kap, f.stretch, t);
}

constexpr int S3X_WARPS = 4;

template <typename T, int N, int MODE>
__global__ void __launch_bounds__(S3X_WARPS *WARP) s3x_kernel(S3Step<T> a, S3Fft<T> f)
{
    using W = WFft<T, N>;
    constexpr int V = W::V, L = W::L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x % L, slot = threadIdx.x / L;
    const int pairs = a.nz * a.nb * a.ny / 2, first = blockIdx.x * (W::rows(S3X_WARPS)) + slot;
    const bool valid = first < pairs;
    const int r0 = 2 * (valid ? first : pairs - 1);
    const RowExchange<T, N> ex{reinterpret_cast<T *>(smem_raw) + (size_t)slot * W::REGION, slot};
    const int k = r0 / (a.nb * a.ny);
    const bool rim = k == 0 || k == a.nz - 1;
    const long long o0 = (long long)r0 * N + t, q0 = (long long)k * a.nxy + (long long)(r0 % a.ny) * N + t, F = a.F;
    const T ri = __ldg(a.bg.rhoinv + k);
    S3Pair<T, N, V> p;
    if (MODE != 1) {
        const T *src = MODE == 0 ? a.A : a.P;
#pragma unroll
        for (int m = 0; m < V; m++) {
            p.re[m] = __ldg(src + o0 + L * m);
            p.im[m] = __ldg(src + o0 + N + L * m);
        }
        s3x_deriv<T, N, V, L>(p, ex, f, t);
    }
    if (MODE == 2) {
#pragma unroll
        for (int m = 0; m < V; m++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const long long o = o0 + r * N + L * m;
                const T acc = rim ? T(0) : (a.flows ? a.S[o] : T(0)) - ri * (r == 0 ? p.dre(m) : p.dim(m));
                if (!valid) continue;
                if (!rim) a.A[3 * F + o] = a.A[3 * F + o] + a.bn * acc;
                if (a.acc) a.acc[o] = acc;
            }
        return;
    }
    if (MODE == 0 && valid) {
#pragma unroll
        for (int m = 0; m < V; m++) {
            a.D[o0 + L * m] = p.dre(m);
            a.D[o0 + N + L * m] = p.dim(m);
        }
    }
    if (MODE == 0 && !a.flows) return;
#pragma unroll 1
    for (int r = 0; r < 2; r++) {
        const long long o = o0 + r * N;
        T xv[V];
        if (MODE == 0) {
#pragma unroll
            for (int m = 0; m < V; m++) xv[m] = __ldg(a.Xv + o + L * m);
        } else {
#pragma unroll
            for (int m = 0; m < V; m++) {
                p.re[m] = __ldg(a.P + o + L * m);
                p.im[m] = __ldg(a.A + o + L * m);
                if (!rim) p.im[m] = p.im[m] + a.b * __ldg(a.Xp + o + L * m);
            }
            s3x_deriv<T, N, V, L>(p, ex, f, t);
#pragma unroll
            for (int m = 0; m < V; m++) {
                const T av = __ldg(a.A + 3 * F + o + L * m);
                const T acc = (a.flows ? a.S[o + L * m] : T(0)) - ri * p.dre(m);
                xv[m] = rim ? av : av + a.b * acc;
            }
#pragma unroll
            for (int m = 0; m < V; m++) {
                if (!valid) continue;
                a.D[o + L * m] = p.dim(m);
                a.Xv[o + L * m] = xv[m];
            }
        }
        if (!a.flows) continue;
#pragma unroll
        for (int m = 0; m < V; m++) {
            p.re[m] = xv[m];
            p.im[m] = __ldg(a.Xv + F + o + L * m);
        }
        s3x_deriv<T, N, V, L>(p, ex, f, t);
#pragma unroll
        for (int m = 0; m < V; m++) {
            const T v0 = __ldg(a.v0 + q0 + r * N + L * m);
            if (!valid) continue;
            a.S[o + L * m] = v0 * p.dre(m);
            a.S[F + o + L * m] = v0 * p.dim(m);
        }
    }
    if (!a.flows) return;
#pragma unroll
    for (int m = 0; m < V; m++) {
        p.re[m] = __ldg(a.Xv + 2 * F + o0 + L * m);
        p.im[m] = __ldg(a.Xv + 2 * F + o0 + N + L * m);
    }
    s3x_deriv<T, N, V, L>(p, ex, f, t);
#pragma unroll
    for (int m = 0; m < V; m++) {
        if (!valid) continue;
        a.S[2 * F + o0 + L * m] = __ldg(a.v0 + q0 + L * m) * p.dre(m);
        a.S[2 * F + o0 + N + L * m] = __ldg(a.v0 + q0 + N + L * m) * p.dim(m);
    }
}

// Y pass over a tile of 2 XL columns of one plane (as ddy_kernel).  PRESSURE: d p/dy completes the RHS of v_y
// and writes a.Xn (the next Xv_y, or the new v_y after the last stage); otherwise d xi_y/dy and the
// y-advection terms.
template <typename T, int NY, bool PRESSURE>
__global__ void __launch_bounds__((DdyCfg<T, NY>::THREADS), (DdyCfg<T, NY>::BLOCKS)) s3y_kernel(S3Step<T> a, S3Fft<T> f)
{
    using C = DdyCfg<T, NY>;
    constexpr int XL = C::XL, V = C::V, L = C::L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RowMax<T> red[2][L][XL];
    const int c = threadIdx.x % XL, t = threadIdx.x / XL, nx = a.nx, k = blockIdx.y / a.nb;
    const bool rim = k == 0 || k == a.nz - 1;
    const long long o0 = (long long)blockIdx.y * a.nxy + blockIdx.x * 2 * XL + c + (long long)t * nx, F = a.F;
    const long long q0 = (long long)k * a.nxy + blockIdx.x * 2 * XL + c + (long long)t * nx;
    const long long step = (long long)L * nx;
    const ColExchange<T, NY, XL> ex{reinterpret_cast<T *>(smem_raw), c};
    const T ri = __ldg(a.bg.rhoinv + k);
    const int nf = PRESSURE ? 1 : a.flows ? 4 : 1;
#pragma unroll 1
    for (int fl = 0; fl < nf; fl++) {
        S3Pair<T, NY, V> p;
        const T *src = PRESSURE ? a.P : fl == 0 ? a.A + F : a.Xv + (long long)(fl - 1) * F;
        RowMax<T> mr, mi;
#pragma unroll
        for (int m = 0; m < V; m++) {
            p.re[m] = __ldg(src + o0 + m * step);
            p.im[m] = __ldg(src + o0 + m * step + XL);
        }
        if (!PRESSURE && fl == 0 && a.Xp && !rim) {  // xi_y of this stage
#pragma unroll
            for (int m = 0; m < V; m++) {
                p.re[m] = p.re[m] + a.b * __ldg(a.Xp + F + o0 + m * step);
                p.im[m] = p.im[m] + a.b * __ldg(a.Xp + F + o0 + m * step + XL);
            }
        }
#pragma unroll
        for (int m = 0; m < V; m++) {
            mr.add(p.re[m]);
            mi.add(p.im[m]);
        }
        red[0][t][c] = mr;
        red[1][t][c] = mi;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < L; j++) {
            mr.merge(red[0][j][c]);
            mi.merge(red[1][j][c]);
        }
        p.sr = row_scale<T>(mr);
        p.si = row_scale<T>(mi);
#pragma unroll
        for (int m = 0; m < V; m++) {
            p.re[m] = scale_in(p.re[m], p.sr);
            p.im[m] = scale_in(p.im[m], p.si);
        }
        // the barriers of the transform's exchanges also keep the next field's maxima behind these
        wfft_deriv<T, NY, V, WFft<T, NY>::RADIX4>(p.re, p.im, ex, f.twr, f.twi, f.kap, f.stretch, t);
#pragma unroll
        for (int m = 0; m < V; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const long long o = o0 + m * step + h * XL;
                const T d = h == 0 ? p.dre(m) : p.dim(m);
                if (PRESSURE) {
                    const T acc = rim ? T(0) : (a.flows ? a.S[F + o] : T(0)) - ri * d;
                    const T av = a.A[4 * F + o];
                    a.Xn[F + o] = rim ? av : av + a.bn * acc;
                    if (a.acc) a.acc[F + o] = acc;
                } else if (fl == 0) {
                    a.D[o] = a.D[o] + d;
                } else {
                    a.S[(long long)(fl - 1) * F + o] += __ldg(a.v0 + a.v0n + q0 + m * step + h * XL) * d;
                }
            }
    }
}

// Z passes: a block owns CW adjacent columns over the full depth, thread (c, j) the rows of chunk j, the
// partitioned compact solve of ddz_kernel from a tile in shared memory.  Only the solve's result is in
// registers: what else a row needs stays in the tile, so that two FP32 blocks of 20 warps share an SM, and
// the rows are then done Z_ROWS at a time, every load of a batch before its first store.
template <typename T>
struct S3Z {
    static constexpr int CW = sizeof(T) == 4 ? 32 : 8, LMAX = 16, MAXNCH = 20, BLOCKS = sizeof(T) == 4 ? 2 : 3;
};
constexpr int Z_ROWS = 4;

// The own rows of an array that a later phase reads, into L2 while this one waits for its barriers: one
// instruction per 128-byte row segment.
template <typename T>
__device__ __forceinline__ void s3z_prefetch(const T *p, long long lvl, int k0, int n, int c)
{
    if (c % (128 / (int)sizeof(T)) == 0)
        for (int m = 0; m < n; m++) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (long long)(k0 + m) * lvl));
}

template <typename T, int LMAX>
__device__ __forceinline__ void s3z_solve(const ZTab<T> &tb, int nch, const T *B, T *YB, int CW, int c, int j, int k0,
                                          int n, int nz, const T *stretch, T (&y)[LMAX])
{
    const T last = zlocal<T, LMAX>(tb, B, CW, c, k0, n, nz, T(0), y);
    YB[(2 * j) * CW + c] = y[0];
    YB[(2 * j + 1) * CW + c] = last;
    __syncthreads();
    T xl, xr;
    zcouple(tb, YB, CW, c, j, nch, xl, xr);
#pragma unroll
    for (int m = 0; m < LMAX; m++)
        if (m < n) y[m] = zcorrect(tb, y[m], k0 + m, xl, xr) * __ldg(stretch + k0 + m);
}

// displacement.f90:396-416: psi_vz, d xi_z/dz + psi_vz, div, p, rho'.
template <typename T>
__global__ void __launch_bounds__(S3Z<T>::CW *S3Z<T>::MAXNCH, S3Z<T>::BLOCKS) s3z_div_kernel(S3Step<T> a, ZTab<T> z1,
                                                                                            int nch, int LC)
{
    constexpr int CW = S3Z<T>::CW, LMAX = S3Z<T>::LMAX;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *B = reinterpret_cast<T *>(smem_raw), *YB = B + (size_t)a.nz * CW;
    const int c = threadIdx.x % CW, j = threadIdx.x / CW, k0 = j * LC, n = min(LC, a.nz - k0), nz = a.nz;
    const long long lvl = a.lvl, r = (long long)blockIdx.x * CW + c;
    const T *axz = a.A + 2 * a.F + r, *xp = a.Xp ? a.Xp + 2 * a.F + r : nullptr;
    s3z_prefetch(a.D + r, lvl, k0, n, c);
#pragma unroll
    for (int m0 = 0; m0 < LMAX; m0 += Z_ROWS) {
        T v[Z_ROWS], w[Z_ROWS];
#pragma unroll
        for (int i = 0; i < Z_ROWS; i++) {
            const int k = k0 + m0 + i;
            if (m0 + i < n) {
                v[i] = __ldg(axz + (long long)k * lvl);
                w[i] = xp && k != 0 && k != nz - 1 ? __ldg(xp + (long long)k * lvl) : T(0);
            }
        }
#pragma unroll
        for (int i = 0; i < Z_ROWS; i++)
            if (m0 + i < n) B[(k0 + m0 + i) * CW + c] = v[i] + a.b * w[i];
    }
    __syncthreads();
    T y[LMAX];
    s3z_solve<T, LMAX>(z1, nch, B, YB, CW, c, j, k0, n, nz, a.stretch, y);
#pragma unroll
    for (int m0 = 0; m0 < LMAX; m0 += Z_ROWS) {
        T d[Z_ROWS];
#pragma unroll
        for (int i = 0; i < Z_ROWS; i++)
            if (m0 + i < n) d[i] = __ldg(a.D + (long long)(k0 + m0 + i) * lvl + r);
#pragma unroll
        for (int i = 0; i < Z_ROWS; i++) {
            const int k = k0 + m0 + i;
            if (m0 + i < n) {
                T dz = y[m0 + i];
                const int pi = s3_pml(a, k);
                if (pi >= 0) {
                    const long long q = (long long)pi * lvl + r;
                    T ps = a.PV[q];
                    if (a.Xp) ps = ps + a.b * a.SPV[q];
                    a.SPV[q] = __ldg(a.bg.az + pi) * dz + __ldg(a.bg.bz + pi) * ps;
                    dz = dz + ps;
                }
                const T div = d[i] + dz, xz = B[k * CW + c];
                a.P[(long long)k * lvl + r] = -__ldg(a.bg.c2rho0 + k) * div - xz * __ldg(a.bg.gradp0_z + k);
                a.RHO[(long long)k * lvl + r] = -__ldg(a.bg.rho0 + k) * div - xz * __ldg(a.bg.gradrho0_z + k);
            }
        }
    }
}

// One field's own rows into the tile.
template <typename T, int LMAX>
__device__ __forceinline__ void s3z_tile(const T *src, long long lvl, T *B, int CW, int k0, int n)
{
#pragma unroll
    for (int m = 0; m < LMAX; m++)
        if (m < n) B[(k0 + m) * CW] = __ldg(src + (long long)(k0 + m) * lvl);
}

// Advection along z of component comp: y = -2 (S + v0z d_z Xv).  v0z is shared by the batch.
template <typename T, int LMAX>
__device__ __forceinline__ void s3z_advection(const S3Step<T> &a, const ZTab<T> &z1, int nch, int comp, T *B, T *YB,
                                              int CW, int c, int j, int k0, int n, long long r, T (&y)[LMAX])
{
    s3z_tile<T, LMAX>(a.Xv + (long long)comp * a.F + r, a.lvl, B + c, CW, k0, n);
    __syncthreads();
    s3z_solve<T, LMAX>(z1, nch, B, YB, CW, c, j, k0, n, a.nz, a.stretch, y);
    const T *S = a.S + (long long)comp * a.F + r, *v0z = a.v0 + 2 * a.v0n + r % a.nxy;
#pragma unroll
    for (int m0 = 0; m0 < LMAX; m0 += Z_ROWS) {
        T s[Z_ROWS], v[Z_ROWS];
#pragma unroll
        for (int i = 0; i < Z_ROWS; i++)
            if (m0 + i < n) {
                s[i] = S[(long long)(k0 + m0 + i) * a.lvl];
                v[i] = __ldg(v0z + (long long)(k0 + m0 + i) * a.nxy);
            }
#pragma unroll
        for (int i = 0; i < Z_ROWS; i++)
            if (m0 + i < n) y[m0 + i] = T(-2.0) * (s[i] + v[i] * y[m0 + i]);
    }
}

// displacement.f90:419-474 along z.  blockIdx.y 0: v_z (pressure gradient, psi_p, buoyancy, source and
// advection), 1, 2: advection of v_x, v_y.
template <typename T>
__global__ void __launch_bounds__(S3Z<T>::CW *S3Z<T>::MAXNCH, S3Z<T>::BLOCKS) s3z_rhs_kernel(S3Step<T> a, ZTab<T> z0,
                                                                                            ZTab<T> z1, int nch, int LC)
{
    constexpr int CW = S3Z<T>::CW, LMAX = S3Z<T>::LMAX;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *B = reinterpret_cast<T *>(smem_raw), *YB = B + (size_t)a.nz * CW, *ADV = YB + (size_t)2 * nch * CW;
    const int c = threadIdx.x % CW, j = threadIdx.x / CW, k0 = j * LC, n = min(LC, a.nz - k0), nz = a.nz;
    const long long lvl = a.lvl, F = a.F, r = (long long)blockIdx.x * CW + c;
    const int comp = blockIdx.y == 0 ? 2 : blockIdx.y - 1;
    T y[LMAX];
    if (a.flows) {
        s3z_advection<T, LMAX>(a, z1, nch, comp, B, YB, CW, c, j, k0, n, r, y);
        if (comp < 2) {
            T *S = a.S + (long long)comp * F + r;
#pragma unroll
            for (int m = 0; m < LMAX; m++)
                if (m < n) S[(long long)(k0 + m) * lvl] = y[m];
            return;
        }
    }
#pragma unroll
    for (int m = 0; m < LMAX; m++)
        if (m < n) ADV[(k0 + m) * CW + c] = a.flows ? y[m] : T(0);
    if (a.flows) __syncthreads();  // every chunk has read the tile and its boundary values
    s3z_tile<T, LMAX>(a.P + r, lvl, B + c, CW, k0, n);
    __syncthreads();
    s3z_solve<T, LMAX>(z0, nch, B, YB, CW, c, j, k0, n, nz, a.stretch, y);
    const T *az = a.A + 5 * F + r, *rho = a.RHO + r;
#pragma unroll
    for (int m0 = 0; m0 < LMAX; m0 += Z_ROWS) {
        T av[Z_ROWS], rh[Z_ROWS];
#pragma unroll
        for (int i = 0; i < Z_ROWS; i++)
            if (m0 + i < n) {
                av[i] = az[(long long)(k0 + m0 + i) * lvl];
                rh[i] = __ldg(rho + (long long)(k0 + m0 + i) * lvl);
            }
#pragma unroll
        for (int i = 0; i < Z_ROWS; i++) {
            if (m0 + i < n) {
                const int k = k0 + m0 + i;
                T gz = y[m0 + i];
                const int pi = s3_pml(a, k);
                if (pi >= 0) {
                    const long long q = a.npv + (long long)pi * lvl + r;
                    T ps = a.PV[q];
                    if (a.Xp) ps = ps + a.b * a.SPV[q];
                    a.SPV[q] = __ldg(a.bg.az + pi) * gz + __ldg(a.bg.bz + pi) * ps;
                    gz = gz + ps;
                }
                const bool rim = k == 0 || k == nz - 1;
                T rz = T(0);
                if (!rim) {
                    const T ri = __ldg(a.bg.rhoinv + k);
                    rz = ADV[k * CW + c] - ri * gz;
                    rz = rz - ri * rh[i] * __ldg(a.bg.g + k);
                    if (a.ADJ) {  // kernel-mode adjoint: forcing / rho0 * delta_width at o_rad (displacement.f90:615-627)
                        if (k == a.k_obs) rz = rz + a.ADJ[r];
                    } else if (abs(k - a.e_rad) <= 4) {
                        rz = rz + (a.PAT[r] * a.amp) * __ldg(a.bg.source_dep + k);
                    }
                }
                a.Xn[2 * F + r + (long long)k * lvl] = rim ? av[i] : av[i] + a.bn * rz;
                if (a.acc) a.acc[2 * F + r + (long long)k * lvl] = rz;
            }
        }
    }
}

// End of a step whose fields are filtered: a block takes CW columns of one field, xi updated with dt Xv (v has
// its new value), then FILTER_VARS_3D_HORIZ_PML (physics.f90:836-882) on levels [npmlbot, nz - npmltop) from
// the tile, in place.
template <typename T>
__global__ void __launch_bounds__(S3_THREADS) s3_end_kernel(S3Step<T> a)
{
    constexpr int CW = 128 / sizeof(T), ROWS = S3_THREADS / CW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *B = reinterpret_cast<T *>(smem_raw);
    const int c = threadIdx.x % CW, w = threadIdx.x / CW, v = blockIdx.y, nz = a.nz;
    const long long lvl = a.lvl, r = (long long)blockIdx.x * CW + c;
    T *col = a.A + (long long)v * a.F + r;
    const T *xv = a.Xv + (long long)v * a.F + r;  // v < 3
#pragma unroll 4
    for (int k = w; k < nz; k += ROWS) {
        T u = col[(long long)k * lvl];
        if (v < 3 && k != 0 && k != nz - 1) u = u + a.dt * __ldg(xv + (long long)k * lvl);
        B[k * CW + c] = u;
    }
    __syncthreads();
    const T c0 = T(0.75390625), h1 = T(0.5 * 0.41015625), h2 = T(0.5 * -0.234375), h3 = T(0.5 * 0.087890625),
            h4 = T(0.5 * -0.01953125), h5 = T(0.5 * 0.001953125);
    const int f0 = a.npmlbot, f1 = nz - a.npmltop;
    const bool filter = f0 >= 5 && f1 + 5 <= nz && f0 < f1;
#pragma unroll 2
    for (int k = w; k < nz; k += ROWS) {
        const T *b = B + k * CW + c;
        const bool in = filter && k >= f0 && k < f1;
        if (!in && v >= 3) continue;
        T out = b[0];
        if (in)
            out = c0 * b[0] + h1 * (b[-CW] + b[CW]) + h2 * (b[-2 * CW] + b[2 * CW]) + h3 * (b[-3 * CW] + b[3 * CW]) +
                  h4 * (b[-4 * CW] + b[4 * CW]) + h5 * (b[-5 * CW] + b[5 * CW]);
        col[(long long)k * lvl] = out;
    }
}

// Adjoint forcing of one step at the observation level, [nb][ny][nx]: LAGRANGE_INTERP of the
// adjoint-source slices (physics.f90:678-737), forcing = sum_j w[j] rows[b][i0 + j] (rows outside
// 0 .. nrows-1 count as zero), times scale = delta_width / rho0(o_rad).
template <typename T>
__global__ void __launch_bounds__(S3_THREADS) s3_adjsrc_kernel(long long lvl, long long nxy, const double *__restrict__ rows,
                                                               int nrows, int i0, S3Lagr w, double scale,
                                                               T *__restrict__ ADJ)
{
    const long long stride = (long long)gridDim.x * S3_THREADS;
    for (long long i = (long long)blockIdx.x * S3_THREADS + threadIdx.x; i < lvl; i += stride) {
        const long long b = i / nxy, q = i - b * nxy;
        double f = 0.0;
#pragma unroll
        for (int j = 0; j < 7; j++) {
            const int r = i0 + j;
            if (r >= 0 && r < nrows && w.w[j] != 0.0) f += w.w[j] * rows[((size_t)b * nrows + r) * nxy + q];
        }
        ADJ[i] = (T)(f * scale);
    }
}

// Kernel-stage record of the forward state (what PRODUCE_KERNELS reads from the partial states,
// kernels.f90:221-280): div xi = D1 + D2 + D3 (the x, y and filtered z derivatives), v_x, v_y, v_z,
// and |acc|^2 of the last stage's RHS of v (hessian integrand), [5][F].
template <typename T>
__global__ void __launch_bounds__(S3_THREADS) s3_record_kernel(long long F, const T *__restrict__ D1,
                                                               const T *__restrict__ D2, const T *__restrict__ D3,
                                                               const T *__restrict__ A, const T *__restrict__ ACC,
                                                               T *__restrict__ snap)
{
    const long long stride = (long long)gridDim.x * S3_THREADS;
    for (long long i = (long long)blockIdx.x * S3_THREADS + threadIdx.x; i < F; i += stride) {
        snap[i] = D1[i] + D2[i] + D3[i];
        snap[F + i] = A[3 * F + i];
        snap[2 * F + i] = A[4 * F + i];
        snap[3 * F + i] = A[5 * F + i];
        const double ax = ACC[i], ay = ACC[F + i], az = ACC[2 * F + i];
        snap[4 * F + i] = (T)(ax * ax + ay * ay + az * az);
    }
}

// Kernel integrands, FP64 accumulation into out [5][F] (kc, kv_x, kv_y, kv_z, hessian):
// kc += div xi_f div v_a (div v_a = D1 + D2 + D3 of the adjoint v), hessian += |acc_f|^2.
template <typename T>
__global__ void __launch_bounds__(S3_THREADS) s3_kacc_div_kernel(long long F, const T *__restrict__ D1,
                                                                 const T *__restrict__ D2, const T *__restrict__ D3,
                                                                 const T *__restrict__ snap, double *__restrict__ out)
{
    const long long stride = (long long)gridDim.x * S3_THREADS;
    for (long long i = (long long)blockIdx.x * S3_THREADS + threadIdx.x; i < F; i += stride) {
        const T diva = D1[i] + D2[i] + D3[i];
        out[i] += (double)snap[i] * (double)diva;
        out[4 * F + i] += (double)snap[4 * F + i];
    }
}

// kv_i += d_i(v_f,j) v_a,j for one component j (D1, D2, D3: x, y, filtered z derivatives of v_f,j).
template <typename T>
__global__ void __launch_bounds__(S3_THREADS) s3_kacc_v_kernel(long long F, const T *__restrict__ D1,
                                                               const T *__restrict__ D2, const T *__restrict__ D3,
                                                               const T *__restrict__ va, double *__restrict__ out)
{
    const long long stride = (long long)gridDim.x * S3_THREADS;
    for (long long i = (long long)blockIdx.x * S3_THREADS + threadIdx.x; i < F; i += stride) {
        const double a = va[i];
        out[F + i] += (double)D1[i] * a;
        out[2 * F + i] += (double)D2[i] * a;
        out[3 * F + i] += (double)D3[i] * a;
    }
}

template <typename T>
__global__ void __launch_bounds__(S3_THREADS) s3_axpy_kernel(long long n, T *__restrict__ Y, const T *__restrict__ X,
                                                             T a)
{
    const long long stride = (long long)gridDim.x * S3_THREADS;
    for (long long i = (long long)blockIdx.x * S3_THREADS + threadIdx.x; i < n; i += stride) Y[i] = Y[i] + a * X[i];
}

// ---------------------------------------------------------------------------------------------
static unsigned s3_grid(long long n)
{
    const long long g = (n + S3_THREADS - 1) / S3_THREADS;
    return (unsigned)(g < 152LL * 16 ? g : 152LL * 16);
}

template <typename T, int N>
static cudaError_t s3x_n(const S3Step<T> &a, const S3Fft<T> &f, int mode, cudaStream_t st)
{
    using W = WFft<T, N>;
    const int pairs = a.nz * a.nb * a.ny / 2, slots = W::rows(S3X_WARPS);
    const size_t smem = (size_t)slots * W::REGION * sizeof(T);
    auto k = mode == 0 ? s3x_kernel<T, N, 0> : mode == 1 ? s3x_kernel<T, N, 1> : s3x_kernel<T, N, 2>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(pairs + slots - 1) / slots, S3X_WARPS * WARP, smem, st>>>(a, f);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_s3x(const S3Step<T> &a, const S3Fft<T> &f, int mode, cudaStream_t st)
{
#define CASE(n_) if (a.nx == n_) return s3x_n<T, n_>(a, f, mode, st);
    CASE(64) CASE(128) CASE(192) CASE(256) CASE(384) CASE(512) CASE(768) CASE(1024)
#undef CASE
    return cudaErrorInvalidValue;
}

template <typename T, int NY>
static cudaError_t s3y_n(const S3Step<T> &a, const S3Fft<T> &f, bool pressure, cudaStream_t st)
{
    using C = DdyCfg<T, NY>;
    auto k = pressure ? s3y_kernel<T, NY, true> : s3y_kernel<T, NY, false>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return e;
    k<<<dim3(a.nx / (2 * C::XL), a.nz * a.nb), C::THREADS, C::SMEM, st>>>(a, f);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_s3y(const S3Step<T> &a, const S3Fft<T> &f, bool pressure, cudaStream_t st)
{
    if (a.nx % 64 || a.nz * a.nb > 65535) return cudaErrorInvalidValue;  // whole tiles: a pass updates in place
#define CASE(n_) if (a.ny == n_) return s3y_n<T, n_>(a, f, pressure, st);
    CASE(64) CASE(128) CASE(192) CASE(256) CASE(384)
    if constexpr (sizeof(T) == 4) { CASE(512) }
#undef CASE
    return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_s3z(const S3Step<T> &a, const ZTab<T> &z0, const ZTab<T> &z1, int nch, int L, bool rhs, cudaStream_t st)
{
    constexpr int CW = S3Z<T>::CW;
    if (a.lvl % CW || L > S3Z<T>::LMAX || nch > S3Z<T>::MAXNCH || a.lvl / CW > 2147483647LL) return cudaErrorInvalidValue;
    const size_t smem = ((size_t)(rhs ? 2 : 1) * a.nz * CW + (size_t)2 * nch * CW) * sizeof(T);
    const dim3 grid((unsigned)(a.lvl / CW), rhs && a.flows ? 3 : 1);
    if (rhs) {
        auto k = s3z_rhs_kernel<T>;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        k<<<grid, CW * nch, smem, st>>>(a, z0, z1, nch, L);
    } else {
        auto k = s3z_div_kernel<T>;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        k<<<grid, CW * nch, smem, st>>>(a, z1, nch, L);
    }
    return cudaGetLastError();
}

// xi += dt Xv, the filter when due, and the PML auxiliaries.
template <typename T>
cudaError_t launch_s3_end(const S3Step<T> &a, bool filter, cudaStream_t st)
{
    if (filter) {
        constexpr int CW = 128 / sizeof(T);
        const size_t smem = (size_t)a.nz * CW * sizeof(T);
        auto k = s3_end_kernel<T>;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        k<<<dim3((unsigned)(a.lvl / CW), 6), S3_THREADS, smem, st>>>(a);
    } else {
        const long long n = (a.nz - 2) * a.lvl;  // the top and bottom rows carry no RHS
        for (int v = 0; v < 3; v++)
            s3_axpy_kernel<T><<<s3_grid(n), S3_THREADS, 0, st>>>(n, a.A + v * a.F + a.lvl, a.Xv + v * a.F + a.lvl, a.dt);
    }
    s3_axpy_kernel<T><<<s3_grid(2 * a.npv), S3_THREADS, 0, st>>>(2 * a.npv, a.PV, a.SPV, a.dt);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_s3_adjsrc(long long lvl, long long nxy, const double *rows, int nrows, int i0, const S3Lagr &w,
                             double scale, T *ADJ, cudaStream_t st)
{
    s3_adjsrc_kernel<T><<<s3_grid(lvl), S3_THREADS, 0, st>>>(lvl, nxy, rows, nrows, i0, w, scale, ADJ);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_s3_record(long long F, const T *D1, const T *D2, const T *D3, const T *A, const T *ACC, T *snap,
                             cudaStream_t st)
{
    s3_record_kernel<T><<<s3_grid(F), S3_THREADS, 0, st>>>(F, D1, D2, D3, A, ACC, snap);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_s3_kacc_div(long long F, const T *D1, const T *D2, const T *D3, const T *snap, double *out,
                               cudaStream_t st)
{
    s3_kacc_div_kernel<T><<<s3_grid(F), S3_THREADS, 0, st>>>(F, D1, D2, D3, snap, out);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_s3_kacc_v(long long F, const T *D1, const T *D2, const T *D3, const T *va, double *out,
                             cudaStream_t st)
{
    s3_kacc_v_kernel<T><<<s3_grid(F), S3_THREADS, 0, st>>>(F, D1, D2, D3, va, out);
    return cudaGetLastError();
}

#define S3_INST(T)                                                                                                    \
    template cudaError_t launch_ddy<T>(const T *, T *, int, int, int, T, const T *, const T *, const T *,            \
                                       cudaStream_t);                                                                \
    template cudaError_t launch_s3x<T>(const S3Step<T> &, const S3Fft<T> &, int, cudaStream_t);                      \
    template cudaError_t launch_s3y<T>(const S3Step<T> &, const S3Fft<T> &, bool, cudaStream_t);                     \
    template cudaError_t launch_s3z<T>(const S3Step<T> &, const ZTab<T> &, const ZTab<T> &, int, int, bool,          \
                                       cudaStream_t);                                                                \
    template cudaError_t launch_s3_end<T>(const S3Step<T> &, bool, cudaStream_t);                                    \
    template cudaError_t launch_s3_adjsrc<T>(long long, long long, const double *, int, int, const S3Lagr &, double, \
                                             T *, cudaStream_t);                                                     \
    template cudaError_t launch_s3_record<T>(long long, const T *, const T *, const T *, const T *, const T *, T *,  \
                                             cudaStream_t);                                                          \
    template cudaError_t launch_s3_kacc_div<T>(long long, const T *, const T *, const T *, const T *, double *,      \
                                               cudaStream_t);                                                        \
    template cudaError_t launch_s3_kacc_v<T>(long long, const T *, const T *, const T *, const T *, double *,        \
                                             cudaStream_t);
S3_INST(float)
S3_INST(double)
#undef S3_INST

}  // namespace sparc
