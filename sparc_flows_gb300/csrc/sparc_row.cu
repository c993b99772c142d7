// sparc_row.cu -- row (x-direction) passes of the RK stage: spectral x-derivatives
// (derivatives.f90:28-58) with the horizontal PML (physics2d.f90:970-986, 1003-1020).
//
// One warp owns one x-row of one solve.  Two real rows are differentiated by one complex
// FFT (real part + i * imaginary part), the derivative operator mapping real rows to real
// rows.  Stage s of the RK step needs, along x:
//   d/dx of p from stage s-1   -> completes RHS v_x of stage s-1 (-rhoinv * dp/dx);
//   d/dx of xi_x at stage s    -> divergence input of stage s (plus the top-row value that
//                                 the column pass needs for its ibc=3 boundary);
//   d/dx of v_x, v_z at stage s -> advection terms -2 v0x d/dx (physics2d.f90:1065-1079).
#include "sparc_fft512.cuh"
#include "sparc_wfft.cuh"

namespace sparc {

constexpr int ROW_WPB = 4;  // rows (warps) per block

// Per-row state of a row pass and its three per-column steps, shared by the Stockham kernel and
// the register-FFT kernel.  MODE 0: stage 1 (no pressure yet), MODE 1: stages 2..5, MODE 2:
// closing pass after stage 5.
template <typename T>
struct RowCtx {
    int b, k, nx, nh, nhx;
    size_t F, ro;
    const T *Ab;
    T bs, bsm1, rhoinv_k;
    T *PXb;
    const T *axk, *bxk;
    __device__ RowCtx(const StepArgs<T> &a, int row, int N)
    {
        b = row / a.nz;
        k = row - b * a.nz;
        nx = N;
        nh = a.nh;
        nhx = a.nhx;
        F = (size_t)a.nz * nx;
        ro = (size_t)k * nx;
        Ab = a.A + (size_t)b * 4 * F;
        bs = a.bs;
        bsm1 = a.bsm1;
        rhoinv_k = __ldg(a.rhoinv + k);
        PXb = a.PX + (size_t)b * 2 * a.nz * nhx;
        axk = a.ax + (size_t)b * a.bgx + (size_t)k * nhx;
        bxk = a.bx + (size_t)b * a.bgx + (size_t)k * nhx;
    }
};

// Inputs of the first FFT at column x: (p_{s-1}, xi_x at stage s) or (p_5, 0).
template <typename T, int MODE>
__device__ __forceinline__ void row_load(const StepArgs<T> &a, const RowCtx<T> &r, int x, T &p, T &xis)
{
    const int b = r.b, k = r.k;
    const size_t F = r.F, ro = r.ro;
    p = T(0);
    xis = T(0);
    if (MODE != 0) p = __ldg(a.P + (size_t)b * F + ro + x);
    if (MODE == 0) {
        xis = __ldg(r.Ab + F_XIX * F + ro + x);
    } else if (MODE == 1) {
        T avx = __ldg(r.Ab + F_VX * F + ro + x);
        T s = (a.stage == 2) ? avx : avx + r.bsm1 * __ldg(svp(a, a.slot_sm2, b, 0) + ro + x);
        if (k == 0 || x == 0 || x == r.nx - 1) s = T(0);  // RHS boundary zeros (physics2d.f90:1083-1093)
        xis = __ldg(r.Ab + F_XIX * F + ro + x) + r.bs * s;
    }
}

// From gpx = dp/dx and dxx = dxi_x/dx at column x: x-PML, RHS v_x of stage s-1, dxi_x/dx for the
// column pass, and the inputs (v_x, v_z at stage s) of the second FFT (MODE != 2).  Loads and arithmetic
// only: what is to be stored is returned (svx: RHS v_x of stage s-1, dxo: dxi_x/dx) or, for the x-PML
// columns, left in the row's scratch P ([3][nhx]: psi_vx RHS or, closing pass, the new psi_vx;
// psi_gradp_x RHS; closing pass, the new psi_gradp_x).  The stores follow in row_mid_store.
template <typename T, int MODE>
__device__ __forceinline__ void row_mid_load(const StepArgs<T> &a, const RowCtx<T> &r, int x, T gpx, T dxx, T *P,
                                             T &svx, T &dxo, T &vxs, T &vzs)
{
    const int b = r.b, k = r.k, nx = r.nx, nh = r.nh, nhx = r.nhx;
    const size_t F = r.F, ro = r.ro;
    const bool pml = (x < nh) || (x >= nx - nh);
    const int ai = (x < nh) ? x : x - (nx - nh) + nh;
    if (pml) {
        const T axv = __ldg(r.axk + ai), bxv = __ldg(r.bxk + ai);
        T ngp = T(0);
        if (MODE != 0) {  // psi_gradp_x of stage s-1
            const size_t q = ((size_t)1 * a.nz + k) * nhx + ai;
            T ps = r.PXb[q];
            if (a.stage >= 3) ps += r.bsm1 * a.SPX[((size_t)a.slot_sm2 * a.nb + b) * 2 * a.nz * nhx + q];
            gpx += ps;
            ngp = axv * gpx + bxv * ps;
            P[nhx + ai] = ngp;
        }
        if (MODE != 2) {  // psi_vx of stage s
            const size_t q = ((size_t)0 * a.nz + k) * nhx + ai;
            T ps = r.PXb[q];
            if (MODE == 1) ps += r.bs * a.SPX[((size_t)a.slot_sm1 * a.nb + b) * 2 * a.nz * nhx + q];
            dxx += ps;
            P[ai] = axv * dxx + bxv * ps;
        } else {  // closing pass: pmlvarsx += deltat * scrpmlx (step.f90:112-115)
            const size_t q0 = ((size_t)0 * a.nz + k) * nhx + ai, q1 = ((size_t)1 * a.nz + k) * nhx + ai;
            P[ai] = r.PXb[q0] + a.dt * a.SPX[((size_t)a.slot_sm1 * a.nb + b) * 2 * a.nz * nhx + q0];
            P[2 * nhx + ai] = r.PXb[q1] + a.dt * ngp;
        }
    }
    svx = T(0);
    if (MODE != 0) {
        svx = __ldg(a.RVXP + (size_t)b * F + ro + x) - r.rhoinv_k * gpx;
        if (k == 0 || x == 0 || x == nx - 1) svx = T(0);
    }
    dxo = dxx;
    vxs = T(0);
    vzs = T(0);
    if (MODE != 2) {
        vxs = __ldg(r.Ab + F_VX * F + ro + x);
        vzs = __ldg(r.Ab + F_VZ * F + ro + x);
        if (MODE == 1) {
            vxs += r.bs * svx;
            vzs += r.bs * __ldg(svp(a, a.slot_sm1, b, 1) + ro + x);
        }
    }
}

// The x-PML stores of row_mid_load from the scratch P (the row's lanes over the PML columns).
template <typename T, int MODE, int LANES>
__device__ __forceinline__ void row_mid_store_pml(const StepArgs<T> &a, const RowCtx<T> &r, const T *P, int lane)
{
    const int b = r.b, k = r.k, nhx = r.nhx;
    for (int ai = lane; ai < nhx; ai += LANES) {
        const size_t q0 = ((size_t)0 * a.nz + k) * nhx + ai, q1 = ((size_t)1 * a.nz + k) * nhx + ai;
        if (MODE != 0) a.SPX[((size_t)a.slot_sm1 * a.nb + b) * 2 * a.nz * nhx + q1] = P[nhx + ai];
        if (MODE != 2) {
            a.SPX[((size_t)a.slot_s * a.nb + b) * 2 * a.nz * nhx + q0] = P[ai];
        } else {
            r.PXb[q0] = P[ai];
            r.PXb[q1] = P[2 * nhx + ai];
        }
    }
}

// The row pass with the register transforms of sparc_wfft.cuh: WFft<T, N>::L threads a row, thread t of a
// row holding columns t + L m.
template <typename T, int N, int MODE, bool TIGHT>
__global__ void __launch_bounds__(ROW_WPB *WARP, TIGHT ? 3 : 0) row_stage_kernel(StepArgs<T> a, int region)
{
    using W = WFft<T, N>;
    constexpr int V = W::V, L = W::L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x % L, slot = threadIdx.x / L;  // row of the block
    if (MODE == 0 && blockIdx.x == 0 && threadIdx.x == 0) *a.d_time += 1;  // new step begins
    const int rows = a.nb * a.nz, first = blockIdx.x * (blockDim.x / L) + slot;
    const bool valid = first < rows;
    const int row = valid ? first : rows - 1;  // the warp's other rows need every lane
    T *S = reinterpret_cast<T *>(smem_raw) + (size_t)slot * region;
    const RowExchange<T, N> ex{S, slot};
    const RowCtx<T> r(a, row, N);

    T re[V], im[V];
    RowMax<T> mr, mi;
#pragma unroll
    for (int m = 0; m < V; m++) {
        row_load<T, MODE>(a, r, t + L * m, re[m], im[m]);
        mr.add(re[m]);
        mi.add(im[m]);
    }
    row_maxima(mr, mi, ex);
    RowScale<T> sr = row_scale<T>(mr), si = row_scale<T>(mi);
#pragma unroll
    for (int m = 0; m < V; m++) {
        re[m] = scale_in(re[m], sr);
        im[m] = scale_in(im[m], si);
    }
    wfft_deriv<T, N, V, W::RADIX4>(re, im, ex, a.twr, a.twi, a.kap, a.stretchx, t);

    RowMax<T> mr2, mi2;
    // FP32: every load of the row before its first store, where the registers hold what is to be stored
    constexpr bool DEFER = sizeof(T) == 4 && !TIGHT;
    constexpr int VD = DEFER ? V : 1;
    T svx[VD], dxo[VD];
    ex.sync();  // the transform's last reads of S are done before S holds the x-PML values
#pragma unroll
    for (int m = 0; m < V; m++) {
        const int x = t + L * m, md = DEFER ? m : 0;
        T vxs, vzs;
        const T dxx = scale_out(im[m], si);
        if (MODE != 2 && r.k == a.nz - 1 && valid) a.TOPDX[(size_t)r.b * N + x] = dxx;  // without the x-PML term
        row_mid_load<T, MODE>(a, r, x, scale_out(re[m], sr), dxx, S, svx[md], dxo[md], vxs, vzs);
        if (!DEFER && valid) {
            if (MODE != 0) svp(a, a.slot_sm1, r.b, 0)[r.ro + x] = svx[md];
            if (MODE != 2) a.DX[(size_t)r.b * r.F + r.ro + x] = dxo[md];
        }
        re[m] = vxs;
        im[m] = vzs;
        mr2.add(vxs);
        mi2.add(vzs);
    }
    ex.sync();
    if (valid) row_mid_store_pml<T, MODE, L>(a, r, S, t);
    if (DEFER && valid) {
#pragma unroll
        for (int m = 0; m < V; m++) {
            const int x = t + L * m, md = DEFER ? m : 0;
            if (MODE != 0) svp(a, a.slot_sm1, r.b, 0)[r.ro + x] = svx[md];
            if (MODE != 2) a.DX[(size_t)r.b * r.F + r.ro + x] = dxo[md];
        }
    }
    if (MODE == 2 || !a.flows) return;
    ex.sync();  // the x-PML values are read before the next transform reuses S
    row_maxima(mr2, mi2, ex);
    sr = row_scale<T>(mr2);
    si = row_scale<T>(mi2);
#pragma unroll
    for (int m = 0; m < V; m++) {
        re[m] = scale_in(re[m], sr);
        im[m] = scale_in(im[m], si);
    }
    wfft_deriv<T, N, V, W::RADIX4>(re, im, ex, a.twr, a.twi, a.kap, a.stretchx, t);
    if (!valid) return;
    T wv[V];  // -2 v0x of the row, loaded before the advection terms are stored
#pragma unroll
    for (int m = 0; m < V; m++) wv[m] = T(-2) * a.fsign * __ldg(a.v0x + (size_t)r.b * a.bg2 + r.ro + t + L * m);
#pragma unroll
    for (int m = 0; m < V; m++) {
        const size_t q = (size_t)r.b * r.F + r.ro + t + L * m;
        const T dvx = scale_out(re[m], sr), dvz = scale_out(im[m], si);
        a.FXX[q] = wv[m] * dvx;
        a.FXZ[q] = wv[m] * dvz;
        if (sizeof(T) == 8 && a.cache) {
            a.cache[q] = dvx;
            a.cache[2 * a.nb * r.F + q] = dvz;
        }
    }
}

// The row pass with the transforms in shared memory, one row to a warp: 109 registers where the register form with 24
// values a thread takes 254, four blocks an SM instead of two (where it is taken: row_stage_n).  Same bits.
template <int N, int MODE>
__global__ void __launch_bounds__(ROW_WPB *WARP) row_stage_shared_kernel(StepArgs<float> a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x / WARP, lane = threadIdx.x % WARP;
    if (MODE == 0 && blockIdx.x == 0 && threadIdx.x == 0) *a.d_time += 1;  // new step begins
    const int row = blockIdx.x * ROW_WPB + warp;
    if (row >= a.nb * a.nz) return;
    float *xr = reinterpret_cast<float *>(smem_raw) + (size_t)warp * 4 * N, *yr = xr + 2 * N;  // real, imaginary parts
    const RowCtx<float> r(a, row, N);
    float mr = 0.f, mi = 0.f;
    for (int x = lane; x < N; x += WARP) {
        float p, xis;
        row_load<float, MODE>(a, r, x, p, xis);
        xr[x] = p;
        xr[N + x] = xis;
        mr = fmaxf(mr, fabsf(p));
        mi = fmaxf(mi, fabsf(xis));
    }
    float sr, si, isr, isi, *re, *im;
    warp_row_scale(mr, sr, isr);
    warp_row_scale(mi, si, isi);
    __syncwarp();
    fft_deriv<float, N>(xr, xr + N, yr, yr + N, a.twr, a.twi, a.kap, a.stretchx, lane, re, im, sr, si);
    __syncwarp();
    float *P = re == xr ? yr : xr;  // the x-PML values, then the next transform's other arrays
    float mr2 = 0.f, mi2 = 0.f;
    for (int x = lane; x < N; x += WARP) {
        float svx, dxo, vxs, vzs;
        const float dxx = im[x] * isi;
        if (MODE != 2 && r.k == a.nz - 1) a.TOPDX[(size_t)r.b * N + x] = dxx;  // without the x-PML term
        row_mid_load<float, MODE>(a, r, x, re[x] * isr, dxx, P, svx, dxo, vxs, vzs);
        if (MODE != 0) svp(a, a.slot_sm1, r.b, 0)[r.ro + x] = svx;
        if (MODE != 2) a.DX[(size_t)r.b * r.F + r.ro + x] = dxo;
        re[x] = vxs;
        im[x] = vzs;
        mr2 = fmaxf(mr2, fabsf(vxs));
        mi2 = fmaxf(mi2, fabsf(vzs));
    }
    __syncwarp();
    row_mid_store_pml<float, MODE, WARP>(a, r, P, lane);
    if (MODE == 2 || !a.flows) return;
    warp_row_scale(mr2, sr, isr);
    warp_row_scale(mi2, si, isi);
    __syncwarp();  // the x-PML values are read before the transform takes their place
    float *o2r, *o2i;
    fft_deriv<float, N>(re, im, P, P + N, a.twr, a.twi, a.kap, a.stretchx, lane, o2r, o2i, sr, si);
    __syncwarp();
    for (int x = lane; x < N; x += WARP) {
        const size_t q = (size_t)r.b * r.F + r.ro + x;
        const float w = -2.f * a.fsign * __ldg(a.v0x + (size_t)r.b * a.bg2 + r.ro + x);
        a.FXX[q] = w * (o2r[x] * isr);
        a.FXZ[q] = w * (o2i[x] * isi);
    }
}

// FP32 rows of 512 columns: the same row pass with the register-resident FFT (sparc_fft512.cuh);
// register n2 of a lane holds column lane + 32 n2.  Each part loads everything it needs before it
// stores anything, so no load waits behind a store of the row it may alias.
constexpr uint32_t STAGE_WAIT_ITERS = 1u << 21;  // polls of 128 ns: about 0.3 s

// Stage overlap: wait (bounded) until every column tile of the solves of this block's rows is
// done.  Thread 0 polls with acquire loads; the barrier passes what it saw to the block.  Returns
// false to every thread on a time-out, with the device error flag set (and at once once that
// flag is set).
__device__ __forceinline__ bool stage_wait(const StepArgs<float> &a, int row0, int nrows)
{
    bool ok = true;
    if (threadIdx.x == 0) {
        // once any device error is flagged (a wait that gave up, a column block that left early)
        // the waits of the rest fail at once
        if (*(volatile int *)a.d_err != 0) ok = false;
        const int last = min(row0 + nrows, a.nb * a.nz) - 1;
        const int *cnt = a.tile_cnt + (size_t)(a.stage - 2) * a.nb;
        for (int b = row0 / a.nz; ok && b <= last / a.nz; b++) {
            uint32_t it = 0;
            for (;;) {
                int v;
                asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(cnt + b) : "memory");
                if (v >= a.tiles_per_solve) break;
                if (++it > STAGE_WAIT_ITERS) {
                    ok = false;
                    break;
                }
                __nanosleep(128);
            }
        }
        if (!ok) atomicExch(a.d_err, SPARC_DEV_ERR_STAGE_WAIT);
    }
    return !__syncthreads_or(!ok);
}

template <int MODE, int MINB>
__global__ void __launch_bounds__(ROW_WPB *WARP, MINB) row_stage_reg512_kernel(StepArgs<float> a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (MODE != 0 && a.tile_cnt && !stage_wait(a, blockIdx.x * ROW_WPB, ROW_WPB)) return;
    if (MODE == 0 && blockIdx.x == 0 && threadIdx.x == 0) *a.d_time += 1;  // new step begins
    const int row = blockIdx.x * ROW_WPB + warp;
    if (row >= a.nb * a.nz) return;
    float *S = reinterpret_cast<float *>(smem_raw) + warp * FFT512_SCRATCH;
    const RowCtx<float> r(a, row, 512);

    float re[16], im[16];
    float mr = 0.f, mi = 0.f;
#pragma unroll
    for (int n2 = 0; n2 < 16; n2++) {
        row_load<float, MODE>(a, r, lane + 32 * n2, re[n2], im[n2]);
        mr = fmaxf(mr, fabsf(re[n2]));
        mi = fmaxf(mi, fabsf(im[n2]));
    }
    float sr, si, isr, isi;
    warp_row_scale(mr, sr, isr);
    warp_row_scale(mi, si, isi);
    fft512_deriv(re, im, S, a.twr, a.twi, a.kap, a.stretchx, lane, sr, si);

    float mr2 = 0.f, mi2 = 0.f;
    float svx[16], dxo[16];
    __syncwarp();  // the transform's last reads of S are done before S holds the x-PML values
#pragma unroll
    for (int n2 = 0; n2 < 16; n2++) {
        float vxs, vzs;
        row_mid_load<float, MODE>(a, r, lane + 32 * n2, re[n2] * isr, im[n2] * isi, S, svx[n2], dxo[n2], vxs, vzs);
        re[n2] = vxs;
        im[n2] = vzs;
        mr2 = fmaxf(mr2, fabsf(vxs));
        mi2 = fmaxf(mi2, fabsf(vzs));
    }
    __syncwarp();
    row_mid_store_pml<float, MODE, WARP>(a, r, S, lane);
    {
        const size_t F = r.F, ro = r.ro;
#pragma unroll
        for (int n2 = 0; n2 < 16; n2++) {
            const int x = lane + 32 * n2;
            if (MODE != 0) svp(a, a.slot_sm1, r.b, 0)[ro + x] = svx[n2];
            if (MODE != 2) {
                a.DX[(size_t)r.b * F + ro + x] = dxo[n2];
                // with the x-PML term, where physics2d.f90:954-955 and the generic pass take it without: from rest the
                // difference is below FP32's rounding, but any other rounding here moves the FP32 kernels by 1.5e-5
                if (r.k == a.nz - 1) a.TOPDX[(size_t)r.b * 512 + x] = dxo[n2];
            }
        }
    }
    if (MODE == 2 || !a.flows) return;
    __syncwarp();  // the x-PML values are read before the next transform reuses S
    float sr2, si2, isr2, isi2;
    warp_row_scale(mr2, sr2, isr2);
    warp_row_scale(mi2, si2, isi2);
    fft512_deriv(re, im, S, a.twr, a.twi, a.kap, a.stretchx, lane, sr2, si2);
    float wv[16];  // -2 v0x of the row, loaded before the advection terms are stored
#pragma unroll
    for (int n2 = 0; n2 < 16; n2++) wv[n2] = -2.f * a.fsign * __ldg(a.v0x + (size_t)r.b * a.bg2 + r.ro + lane + 32 * n2);
#pragma unroll
    for (int n2 = 0; n2 < 16; n2++) {
        const size_t q = (size_t)r.b * r.F + r.ro + lane + 32 * n2;
        a.FXX[q] = wv[n2] * (re[n2] * isr2);
        a.FXZ[q] = wv[n2] * (im[n2] * isi2);
    }
}

// Generic spectral x-derivative of nrows rows, two to a transform.
template <typename T, int N, bool FOUR>
__global__ void __launch_bounds__(ROW_WPB *WARP) ddx_kernel(const T *__restrict__ var, T *__restrict__ dvar,
                                                              int nrows, T stretchx, const T *twr, const T *twi,
                                                              const T *kap)
{
    using W = WFft<T, N, FOUR>;
    constexpr int V = W::V, L = W::L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x % L, slot = threadIdx.x / L;
    const int r0 = 2 * (blockIdx.x * (blockDim.x / L) + slot);
    const bool one = r0 < nrows, two = r0 + 1 < nrows;
    const RowExchange<T, N, L> ex{reinterpret_cast<T *>(smem_raw) + (size_t)slot * W::REGION, slot};
    const T *src = var + (size_t)r0 * N + t;
    T re[V], im[V];
    RowMax<T> mr, mi;
#pragma unroll
    for (int m = 0; m < V; m++) {
        re[m] = one ? src[L * m] : T(0);
        im[m] = two ? src[N + L * m] : T(0);
    }
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
    wfft_deriv<T, N, V, W::RADIX4>(re, im, ex, twr, twi, kap, stretchx, t);
    T *dst = dvar + (size_t)r0 * N + t;
#pragma unroll
    for (int m = 0; m < V; m++) {
        if (one) dst[L * m] = scale_out(re[m], sr);
        if (two) dst[N + L * m] = scale_out(im[m], si);
    }
}

// The same of few FP64 rows: a transform in shared memory, a pair of rows to a warp.  With radix 8 the register form
// holds 24 values a thread at 192 and 384 columns, eight and sixteen lanes to a pair: too few warps for the FP64 pipe.
template <int N>
__global__ void __launch_bounds__(ROW_WPB *WARP) ddx_shared_kernel(const double *__restrict__ var, double *__restrict__ dvar,
                                                                    int nrows, double stretchx, const double *twr,
                                                                    const double *twi, const double *kap)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x / WARP, lane = threadIdx.x % WARP, r0 = 2 * (blockIdx.x * ROW_WPB + warp);
    if (r0 >= nrows) return;
    const bool two = r0 + 1 < nrows;
    double *xr = reinterpret_cast<double *>(smem_raw) + (size_t)warp * 4 * N, *xi = xr + N, *yr = xi + N, *yi = yr + N;
    const double *src = var + (size_t)r0 * N;
    double mr = 0.0, mi = 0.0;
    for (int x = lane; x < N; x += WARP) {
        xr[x] = src[x];
        xi[x] = two ? src[N + x] : 0.0;
        mr = fmax(mr, fabs(xr[x]));
        mi = fmax(mi, fabs(xi[x]));
    }
    double sr, si, isr, isi;
    warp_row_scale(mr, sr, isr);
    warp_row_scale(mi, si, isi);
    __syncwarp();
    double *re, *im, *dst = dvar + (size_t)r0 * N;
    fft_deriv<double, N>(xr, xi, yr, yi, twr, twi, kap, stretchx, lane, re, im, sr, si);
    __syncwarp();
    for (int x = lane; x < N; x += WARP) {
        dst[x] = re[x] * isr;
        if (two) dst[N + x] = im[x] * isi;
    }
}

#define SPARC_FFT_SIZES(X) X(64) X(128) X(192) X(256) X(384) X(512) X(768) X(1024)

bool fft_size_supported(int n)
{
#define CASE(n_) if (n == n_) return true;
    SPARC_FFT_SIZES(CASE)
#undef CASE
    return false;
}

template <int MODE, int MINB>
static void row_reg512_n(const StepArgs<float> &a, cudaStream_t st)
{
    const size_t smem = (size_t)ROW_WPB * FFT512_SCRATCH * sizeof(float);
    const int grid = (a.nb * a.nz + ROW_WPB - 1) / ROW_WPB;
    auto k = row_stage_reg512_kernel<MODE, MINB>;
    if (MODE != 0 && a.tile_cnt) {  // a programmatic dependent of the column pass before it
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(ROW_WPB * WARP);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, k, a);
        return;
    }
    k<<<grid, ROW_WPB * WARP, smem, st>>>(a);
}

// Few rows (at most one block on every SM): registers for all loads of a row at once (two blocks per SM, 255
// registers) instead of four blocks: 11.9 us a launch for one solve of 512 x 300 against 12.9.
template <int MODE>
static void row_reg512_launch(const StepArgs<float> &a, cudaStream_t st)
{
    if (a.nb * a.nz <= 152 * ROW_WPB) return row_reg512_n<MODE, 2>(a, st);
    return row_reg512_n<MODE, 4>(a, st);
}

template <typename T, int N, bool TIGHT>
static cudaError_t row_generic(const StepArgs<T> &a, cudaStream_t st)
{
    // four warps a block; two, so that the blocks reach every SM, where the rows are few
    const int rows = a.nb * a.nz, wpb = rows <= 152 * WFft<T, N>::rows(ROW_WPB) ? 2 : ROW_WPB;
    const int slots = WFft<T, N>::rows(wpb), grid = (rows + slots - 1) / slots;
    const int region = max(WFft<T, N>::REGION, 3 * a.nhx);  // exchange arrays, or the row's x-PML values
    const size_t smem = (size_t)slots * region * sizeof(T);
    auto k = a.stage == 1   ? row_stage_kernel<T, N, 0, false>
             : a.stage <= 5 ? row_stage_kernel<T, N, 1, TIGHT>
                            : row_stage_kernel<T, N, 2, false>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<grid, wpb * WARP, smem, st>>>(a, region);
    return cudaGetLastError();
}

template <int N>
static cudaError_t row_shared(const StepArgs<float> &a, cudaStream_t st)
{
    const size_t smem = (size_t)ROW_WPB * 4 * N * sizeof(float);
    auto k = a.stage == 1   ? row_stage_shared_kernel<N, 0>
             : a.stage <= 5 ? row_stage_shared_kernel<N, 1>
                            : row_stage_shared_kernel<N, 2>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(a.nb * a.nz + ROW_WPB - 1) / ROW_WPB, ROW_WPB * WARP, smem, st>>>(a);
    return cudaGetLastError();
}

template <typename T, int N>
static cudaError_t row_stage_n(const StepArgs<T> &a, cudaStream_t st)
{
    if constexpr (sizeof(T) == 4 && N == 512) {
        if (a.stage == 1) row_reg512_launch<0>(a, st);
        else if (a.stage <= 5) row_reg512_launch<1>(a, st);
        else row_reg512_launch<2>(a, st);
        return cudaGetLastError();
    }
    // FP32 with 24 values a thread (192, 384 and 768 columns): stages 2 to 5 hold every load of a row at once, two blocks
    // an SM.  Rows that would make a second wave of those and one wave of three blocks take three, with 168 registers and
    // their stores where the values arise (a solve keeps its bits): 12 solves of 384 x 300 353 us a step against 371, 24 of
    // 192 x 300 335 against 387 (GB300).  At 768 columns that spills, and what would be the second wave
    // goes to the transforms in shared memory, four blocks an SM: six solves of 768 x 300 403 us a step against 455
    if constexpr (sizeof(T) == 4 && N == 768) {
        const int rows = a.nb * a.nz;
        if (rows > 152 * 2 * ROW_WPB && rows <= 152 * 4 * ROW_WPB && 3 * a.nhx <= 2 * N) return row_shared<N>(a, st);
    }
    if constexpr (sizeof(T) == 4 && (N == 192 || N == 384)) {
        const int rows = a.nb * a.nz, block = WFft<T, N>::rows(ROW_WPB);
        if (rows > 152 * 2 * block && rows <= 152 * 3 * block) return row_generic<T, N, true>(a, st);
    }
    return row_generic<T, N, false>(a, st);
}

template <typename T>
cudaError_t launch_row_stage(const StepArgs<T> &a, cudaStream_t st)
{
#define CASE(n_) if (a.nx == n_) return row_stage_n<T, n_>(a, st);
    SPARC_FFT_SIZES(CASE)
#undef CASE
    return cudaErrorInvalidValue;
}

template <typename T, int N, bool FOUR>
static cudaError_t ddx_n(const T *var, T *dvar, int nrows, T stretchx, const T *twr, const T *twi, const T *kap,
                         cudaStream_t st)
{
    const int pairs = (nrows + 1) / 2, wpb = pairs > 152 * WFft<T, N, FOUR>::rows(ROW_WPB) ? ROW_WPB : WFft<T, N, FOUR>::L > WARP ? 2 : 1;
    const int slots = WFft<T, N, FOUR>::rows(wpb), grid = (pairs + slots - 1) / slots;
    const size_t smem = (size_t)slots * WFft<T, N, FOUR>::REGION * sizeof(T);
    auto k = ddx_kernel<T, N, FOUR>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k<<<grid, wpb * WARP, smem, st>>>(var, dvar, nrows, stretchx, twr, twi, kap);
    return cudaGetLastError();
}

template <int N>
static cudaError_t ddx_shared_n(const double *var, double *dvar, int nrows, double stretchx, const double *twr,
                                const double *twi, const double *kap, cudaStream_t st)
{
    const size_t smem = (size_t)ROW_WPB * 4 * N * sizeof(double);
    auto k = ddx_shared_kernel<N>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(nrows + 2 * ROW_WPB - 1) / (2 * ROW_WPB), ROW_WPB * WARP, smem, st>>>(var, dvar, nrows, stretchx, twr, twi, kap);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_ddx(const T *var, T *dvar, int nrows, int nx, T stretchx, const T *twr, const T *twi,
                       const T *kap, cudaStream_t st, bool radix8)
{
    if (nrows <= 0) return cudaSuccess;
    // FP64 at radix 8: three (192 columns) and one (384) waves of a pair of rows to each of four warps per SM.  192: 23 us
    // up to 1200 rows and 50 at 3600 against 51 in registers, 66 against 56 at 4800; 384: 55 against 60, 93 against 60 at
    // 1800 (GB300).  Both give the same bits.
    if constexpr (sizeof(T) == 8) {
        const int wave = 152 * ROW_WPB * 2;
        if (radix8 && nx == 192 && nrows <= 3 * wave) return ddx_shared_n<192>(var, dvar, nrows, stretchx, twr, twi, kap, st);
        if (radix8 && nx == 384 && nrows <= wave) return ddx_shared_n<384>(var, dvar, nrows, stretchx, twr, twi, kap, st);
    }
#define CASE(n_)                                                                                                     \
    if (nx == n_)                                                                                                    \
        return radix_four<T, n_>() && !radix8                                                                         \
                   ? ddx_n<T, n_, radix_four<T, n_>()>(var, dvar, nrows, stretchx, twr, twi, kap, st)                 \
                   : ddx_n<T, n_, false>(var, dvar, nrows, stretchx, twr, twi, kap, st);
    SPARC_FFT_SIZES(CASE)
#undef CASE
    return cudaErrorInvalidValue;
}

// Kernel integral, x-derivatives of one record pair: d/dx of forward xi_x, v_x, v_z and of the
// adjoint v_x (compute_div / compute_del, kernels.f90:843-887).
template <typename T, int N>
__global__ void __launch_bounds__(ROW_WPB *WARP) kacc_row_kernel(KAccArgs<T> a)
{
    using W = WFft<T, N>;
    constexpr int V = W::V, L = W::L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x % L, slot = threadIdx.x / L;
    const int rows = a.nb * a.nz, first = blockIdx.x * (blockDim.x / L) + slot;
    const bool valid = first < rows;
    const int row = valid ? first : rows - 1;
    const RowExchange<T, N> ex{reinterpret_cast<T *>(smem_raw) + (size_t)slot * W::REGION, slot};
    const int b = row / a.nz, k = row - b * a.nz;
    const size_t F = (size_t)a.nz * N, q = (size_t)k * N + t;
    const T *f = a.fsn + a.fbase + (size_t)b * a.fstride + q;
    const T *av = a.adj + (size_t)b * a.astride + q;
    T *w = a.work + (size_t)b * 4 * F + q;
    // forward xi_x with adjoint v_x, then forward v_x with v_z: the forward and adjoint fields
    // carry unrelated normalisations, so each row is scaled before it shares an FFT
#pragma unroll
    for (int pair = 0; pair < 2; pair++) {
        const T *p0 = pair == 0 ? f : f + 2 * F, *p1 = pair == 0 ? av : f + 3 * F;
        T re[V], im[V];
        RowMax<T> mr, mi;
#pragma unroll
        for (int m = 0; m < V; m++) {
            re[m] = __ldg(p0 + L * m);
            im[m] = __ldg(p1 + L * m);
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
        wfft_deriv<T, N, V, W::RADIX4>(re, im, ex, a.twr, a.twi, a.kap, a.stretchx, t);
#pragma unroll
        for (int m = 0; m < V; m++) {
            if (!valid) continue;
            w[(size_t)(2 * pair) * F + L * m] = scale_out(re[m], sr);
            w[(size_t)(2 * pair + 1) * F + L * m] = scale_out(im[m], si);
        }
    }
}

template <typename T, int N>
static cudaError_t kacc_row_n(const KAccArgs<T> &a, cudaStream_t st)
{
    const int rows = a.nb * a.nz, slots = WFft<T, N>::rows(ROW_WPB);
    const size_t smem = (size_t)slots * WFft<T, N>::REGION * sizeof(T);
    auto k = kacc_row_kernel<T, N>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<(rows + slots - 1) / slots, ROW_WPB * WARP, smem, st>>>(a);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_kacc_row(const KAccArgs<T> &a, cudaStream_t st)
{
#define CASE(n_) if (a.nx == n_) return kacc_row_n<T, n_>(a, st);
    SPARC_FFT_SIZES(CASE)
#undef CASE
    return cudaErrorInvalidValue;
}
template cudaError_t launch_kacc_row<float>(const KAccArgs<float> &, cudaStream_t);
template cudaError_t launch_kacc_row<double>(const KAccArgs<double> &, cudaStream_t);

template cudaError_t launch_row_stage<float>(const StepArgs<float> &, cudaStream_t);
template cudaError_t launch_row_stage<double>(const StepArgs<double> &, cudaStream_t);
template cudaError_t launch_ddx<float>(const float *, float *, int, int, float, const float *, const float *,
                                       const float *, cudaStream_t, bool);
template cudaError_t launch_ddx<double>(const double *, double *, int, int, double, const double *,
                                        const double *, const double *, cudaStream_t, bool);

}  // namespace sparc
