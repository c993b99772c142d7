// sparc_wfft.cuh -- register-resident spectral transforms of N-point complex rows.
//
// Thread t of the L = N / V threads of a row holds elements t + L m, m = 0..V-1, in registers.  Each
// Stockham stage of radix R is V / R butterflies on the thread's own registers (element j + r N / R of
// butterfly j = t + L q is register q + r V / R), so only the exchanges between stages go through
// shared memory, the first stage reads what was loaded from global memory, and the last leaves
// element t + L m in register m again: the multiplication by i k and the inverse transform follow in
// place.  Radices and operation order are those of stockham_stage (sparc_common.cuh), so the results
// are the same bits; the radix-4 form (FOUR, below) has its own.
//
// V is a multiple of every radix of N, which gives every thread whole butterflies at every
// stage: rows of 64 and 128 columns share a warp (four and two to a warp), where one row to a warp left 24
// and 16 lanes of it idle.  That matters most in FP64, whose pipe takes 64 cycles per warp-wide
// instruction and quadrant whether one lane works or all.  Radices 8, 8, ... with V = 8 for 64, 128, 256, 16
// for 512 and 1024, 24 for 192, 384, 768.  FP64 passes of 192, 384 and 768 columns (FOUR) take radix 4 and V = 12,
// for twice the warps at the same operations (V = 24 leaves a 300-row pass 75 warps for 608 quadrants).
// A row of 1024 columns, and of 768 in FP64, is held by two warps: one warp would need V = 32 or 24, which fills its
// registers (FP64 spilled up to 1 KB a thread; FP32 left 8 warps on an SM).  Step of 1024 x 300, two warps against
// one: FP32 one solve 214 us against 280, six 545 against 797; FP64 one 946 against 1371, four 3390 against 3414.  Of
// 768 x 300: FP64 one 818 against 1118 (GB300).  FP32 rows of 768 columns keep radix 8, and with it their bits.
#pragma once
#include "sparc_common.cuh"

namespace sparc {

template <typename T, int N, bool FOUR>
struct WRadices {
    static_assert(!FOUR || N == 192 || N == 384 || N == 768, "radix-4 form");
    static constexpr int V = FOUR ? 12 : N % 3 == 0 ? 24 : N <= 256 ? 8 : 16;
    static constexpr int count() { return FOUR ? (N == 192 ? 4 : 5) : Radices<N>::count(); }
    static constexpr int at(int i)
    {
        if (!FOUR) return Radices<N>::at(i);
        return i < 3 || (N == 768 && i == 3) ? 4 : N == 384 && i == 3 ? 2 : 3;
    }
};

// FP64 passes of a step use the radix-4 form where there is one.
template <typename T, int N>
constexpr bool radix_four() { return sizeof(T) == 8 && (N == 192 || N == 384 || N == 768); }

template <typename T, int N, bool FOUR = radix_four<T, N>()>
struct WFft {
    static constexpr bool RADIX4 = FOUR;
    static constexpr int V = WRadices<T, N, FOUR>::V;
    static constexpr int L = N / V;          // threads of a row: lanes of one warp or (64) two warps
    static constexpr int rows(int warps) { return warps * WARP / L; }  // rows of so many warps
    static constexpr int SPAN = N + N / 8;   // words of one exchange array (one word of padding per 8)
    static constexpr int REGION = 2 * SPAN + 8;  // real and imaginary parts of a row
};

// Exchange buffers.  Row: a row of L threads, of one warp or two (which meet at a barrier of the row's own, its
// number in the block + 1); one padding word per 8 keeps the strided writes of every stage on distinct banks.
template <typename T, int N, int L = WFft<T, N>::L>
struct RowExchange {
    static constexpr bool TWO = false;  // a warp's barrier costs less than a second buffer
    static constexpr int SPAN = N + N / 8;
    T *s;
    int row = 0;  // of the block
    __device__ __forceinline__ void sync() const
    {
        __syncwarp();
        if constexpr (L > WARP) asm volatile("bar.sync %0, %1;" ::"r"(row + 1), "n"(L) : "memory");
    }
    template <int BUF>
    __device__ __forceinline__ void put(int i, T re, T im) const
    {
        const int q = i + (i >> 3);
        s[q] = re;
        s[SPAN + q] = im;
    }
    template <int BUF>
    __device__ __forceinline__ void get(int i, T &re, T &im) const
    {
        const int q = i + (i >> 3);
        re = s[q];
        im = s[SPAN + q];
    }
};

// Column: a block transforms XL adjacent columns (neighbouring threads are neighbouring columns, so
// global and shared accesses are contiguous), rows of XL values.  Where a row is half of the 32 banks
// (16 columns of FP32), a row of padding per 8 keeps the two rows that a warp writes on different halves.
// Two buffers in turn: a thread that writes one has passed the barrier behind every read of it, so an
// exchange takes one block barrier instead of two.
template <typename T, int N, int XL>
struct ColExchange {
    static constexpr bool TWO = true;
    static constexpr bool PAD = XL * sizeof(T) < 128;
    static constexpr int SPAN = (PAD ? N + N / 8 : N) * XL;
    T *s;
    int x;
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    __device__ __forceinline__ int at(int i) const { return (PAD ? i + (i >> 3) : i) * XL + x; }
    static constexpr size_t BYTES = (size_t)4 * SPAN * sizeof(T);  // both buffers
    template <int BUF>
    __device__ __forceinline__ void put(int i, T re, T im) const
    {
        s[2 * BUF * SPAN + at(i)] = re;
        s[(2 * BUF + 1) * SPAN + at(i)] = im;
    }
    template <int BUF>
    __device__ __forceinline__ void get(int i, T &re, T &im) const
    {
        re = s[2 * BUF * SPAN + at(i)];
        im = s[(2 * BUF + 1) * SPAN + at(i)];
    }
};

// BUF: buffer of the stage's exchange.
template <typename T, int N, int V, bool FOUR, int I, int NS, bool INV, int BUF, class EX>
__device__ __forceinline__ void wfft_stages(T (&re)[V], T (&im)[V], const EX &ex, const T *__restrict__ twr,
                                            const T *__restrict__ twi, int t)
{
    using RX = WRadices<T, N, FOUR>;
    if constexpr (I < RX::count()) {
        constexpr int R = RX::at(I), Q = V / R, L = N / V, TS = N / (NS * R);
        static_assert(V % R == 0, "every thread holds whole butterflies");
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int k = (t + q * L) % NS;
            T vr[R], vi[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const T ar = re[q + r * Q], ai = im[q + r * Q];
                if (NS == 1 || r == 0) {
                    vr[r] = ar;
                    vi[r] = ai;
                } else {
                    const int w = r * k * TS;  // < N
                    const T wr = __ldg(twr + w), wi = INV ? -__ldg(twi + w) : __ldg(twi + w);
                    vr[r] = ar * wr - ai * wi;
                    vi[r] = ar * wi + ai * wr;
                }
            }
            butterfly<T, R>(vr, vi, INV);
#pragma unroll
            for (int r = 0; r < R; r++) {
                re[q + r * Q] = vr[r];
                im[q + r * Q] = vi[r];
            }
        }
        if constexpr (I + 1 < RX::count()) {
            if constexpr (!EX::TWO) ex.sync();  // the buffer's last readers are done
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const int j = t + q * L, base = (j / NS) * NS * R + j % NS;
#pragma unroll
                for (int r = 0; r < R; r++) ex.template put<BUF>(base + r * NS, re[q + r * Q], im[q + r * Q]);
            }
            ex.sync();
#pragma unroll
            for (int m = 0; m < V; m++) ex.template get<BUF>(t + L * m, re[m], im[m]);
        }
        wfft_stages<T, N, V, FOUR, I + 1, NS * R, INV, 1 - BUF>(re, im, ex, twr, twi, t);
    }
}

__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// Spectral derivative of a complex row held as re, im[m] = x[t + L m] (real and imaginary parts: two
// real rows), in place; kap (which carries 1 / N and a zero Nyquist bin) and scale as fft_deriv (sparc_common.cuh).
template <typename T, int N, int V, bool FOUR, class EX>
__device__ __forceinline__ void wfft_deriv(T (&re)[V], T (&im)[V], const EX &ex, const T *__restrict__ twr,
                                           const T *__restrict__ twi, const T *__restrict__ kap, T scale, int t)
{
    wfft_stages<T, N, V, FOUR, 0, 1, false, 0>(re, im, ex, twr, twi, t);
#pragma unroll
    for (int m = 0; m < V; m++) {
        const T kk = mul_rn(__ldg(kap + t + (N / V) * m), scale);
        const T a = re[m], b = im[m];
        re[m] = mul_rn(-kk, b);  // rounded here, not contracted into the next stage's additions
        im[m] = mul_rn(kk, a);
    }
    // the forward transform's exchanges took the buffers 0, 1, ... in turn
    wfft_stages<T, N, V, FOUR, 0, 1, true, (WRadices<T, N, FOUR>::count() - 1) % 2>(re, im, ex, twr, twi, t);
}

// ---- power-of-two row scales (pow2_scale_of): only the exponent of a row's largest |v| and whether
// the row is zero are needed, so the maximum is taken on bit patterns, and for FP64 the scaling itself is
// an integer addition to the exponent: no double-precision instruction in either.
template <typename T>
struct RowMax;
template <>
struct RowMax<float> {
    unsigned m = 0u;
    __device__ __forceinline__ void add(float v) { m = max(m, __float_as_uint(v) & 0x7fffffffu); }
    __device__ __forceinline__ void merge(const RowMax &o) { m = max(m, o.m); }
    template <int W>
    __device__ __forceinline__ void reduce()
    {
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    __device__ __forceinline__ float value() const { return __uint_as_float(m); }
};
template <>
struct RowMax<double> {  // m: the high words' maximum; any: a low word that is not zero (hi 0: subnormal)
    unsigned m = 0u, any = 0u;
    __device__ __forceinline__ void add(double v)
    {
        m = max(m, (unsigned)__double2hiint(v) & 0x7fffffffu);
        any |= (unsigned)__double2loint(v);
    }
    __device__ __forceinline__ void merge(const RowMax &o)
    {
        m = max(m, o.m);
        any |= o.any;
    }
    template <int W>
    __device__ __forceinline__ void reduce()
    {
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) {
            m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            any |= __shfl_xor_sync(0xffffffffu, any, o);
        }
    }
    __device__ __forceinline__ double value() const { return __hiloint2double((int)m, m == 0u ? (int)any : 0); }
};

// The maxima of two rows that share a transform, over its threads; rows of two warps meet in the exchange's last words.
template <typename T, int N, int L>
__device__ __forceinline__ void row_maxima(RowMax<T> &re, RowMax<T> &im, const RowExchange<T, N, L> &ex)
{
    re.template reduce<(L < WARP ? L : WARP)>();
    im.template reduce<(L < WARP ? L : WARP)>();
    if constexpr (L > WARP) {
        static_assert(L == 2 * WARP && 4 * sizeof(RowMax<T>) <= 8 * sizeof(T), "the words behind the exchange arrays");
        RowMax<T> *w = reinterpret_cast<RowMax<T> *>(ex.s + 2 * RowExchange<T, N, L>::SPAN);
        const int h = (threadIdx.x / WARP) % 2;
        if (threadIdx.x % WARP == 0) {
            w[2 * h] = re;
            w[2 * h + 1] = im;
        }
        ex.sync();
        re.merge(w[2 * (1 - h)]);
        im.merge(w[2 * (1 - h) + 1]);
    }
}

template <typename T>
struct RowScale {
    T s, inv;
    int d;  // s = 2^d
};
template <typename T>
__device__ __forceinline__ RowScale<T> row_scale(const RowMax<T> &m)
{
    const T v = m.value();
    RowScale<T> r;
    r.s = pow2_scale_of(v);
    r.inv = (v == T(0)) ? T(0) : pow2_inverse(r.s);
    r.d = pow2_exponent(r.s);
    return r;
}
// v s and v inv, exactly as the multiplications give them.
__device__ __forceinline__ float scale_in(float v, const RowScale<float> &r) { return v * r.s; }
__device__ __forceinline__ float scale_out(float v, const RowScale<float> &r) { return v * r.inv; }
__device__ __forceinline__ double add_exponent(double v, int d, double s)
{
    const int hi = __double2hiint(v), e = (hi >> 20) & 0x7ff, n = e + d;
    if (e != 0 && e != 0x7ff && n > 0 && n < 0x7ff) return __hiloint2double(hi + (d << 20), __double2loint(v));
    return v * s;  // zero, subnormal or not finite, before or after
}
__device__ __forceinline__ double scale_in(double v, const RowScale<double> &r) { return add_exponent(v, r.d, r.s); }
__device__ __forceinline__ double scale_out(double v, const RowScale<double> &r)
{
    if (r.inv == 0.0) return v * 0.0;
    return add_exponent(v, -r.d, r.inv);
}

}  // namespace sparc
