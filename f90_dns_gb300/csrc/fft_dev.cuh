// Device building blocks of the plane transforms with compile-time lengths:
// register DFTs, the block-wide Stockham pass, 64-bit block fixed point and
// its conversions (fft_ct.cu, fft_nl.cu).
#pragma once

#include <type_traits>

#include "cvt.cuh"
#include "dns3d_internal.cuh"

namespace dns3d {

// Instantiated lengths: ny in {16..512}, nx/2 in {16..256}, 2^a or 3 2^a.
#define DNS3D_CT_Y_LENGTHS(X) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(384) X(512)
#define DNS3D_CT_X_LENGTHS(X) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256)

namespace {

constexpr int kThreads = 256;

template <typename C> __device__ __forceinline__ C mk(decltype(C::x) a, decltype(C::x) b) { C r; r.x = a; r.y = b; return r; }
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return mk<C>(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return mk<C>(a.x - b.x, a.y - b.y); }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
    return mk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// (SIGN i) a
template <int SIGN, typename C> __device__ __forceinline__ C mul_si(C a) {
    return SIGN > 0 ? mk<C>(-a.y, a.x) : mk<C>(a.y, -a.x);
}

// ------------------------------------------------------------------ 64-bit fixed point
// The FP64 path's transforms run in block fixed point on the integer pipes:
// this GPU issues FP64 arithmetic at 1/64 of its FP32 rate, and the FP64
// plane transforms were bound by it.  One transform (a y column or an x row)
// is scaled by the power of two that gives its largest input component
// B <= 53 significant bits (as an FP64 mantissa has), with B small enough
// that no partial DFT can leave int64 (a length-N DFT grows a modulus at most
// N-fold); butterflies then add exactly, and every twiddle product is rounded once to
// the transform's grid.  Twiddles are Q62 integers (value * 2^62).  The result differs from an FP64
// transform's by the same order as that transform's own rounding error
// (normwise ~2^-B per rounding step).
using fx2 = longlong2;

// Products on the 32-bit multiply-add units.  A 64-bit integer is split into
// signed limbs, x = x1 2^32 + x0 with x0 in [-2^31, 2^31), so that every limb
// product is one signed 32 x 32 + 64-bit multiply-add; tables hold their
// entries split already (pack_limbs, fft.cu; |w0| < 2^31).  A sum of products
// is wanted over 2^64, where its high limbs add as they are and the middle
// ones give their high word: an operand is shifted left on being split so that
// a Q62 table entry gives its product over 2^64 (by 2, for |x| < 2^61), a Q63
// constant likewise (by 1, for |x| < 2^62).  The low products enter by their
// high words alone: the sum is rounded once (half up) but for 2^-31 of a unit.
// A complex product is 18 multiply-adds and a dozen other integer operations;
// from the compiler's 128-bit products it was 16 and about four dozen, and the
// inverse y pass of three fields at 128x128x65 took 41 us against 29 us.
struct FxLimbs {
    int lo, hi;
};
template <int S = 0> __device__ __forceinline__ FxLimbs fx_split(long long x) {
    const long long y = (long long)((unsigned long long)x << S);
    const int lo = (int)y;
    return {lo, (int)(y >> 32) + (int)((unsigned)lo >> 31)};
}
__device__ __forceinline__ FxLimbs fx_packed(long long w) { return {(int)w, (int)(w >> 32)}; }
__device__ __forceinline__ FxLimbs fx_neg(FxLimbs a) { return {-a.lo, -a.hi}; }

// round(x w / 2^64)
__device__ __forceinline__ long long fx_prod(FxLimbs x, FxLimbs w) {
    long long m = (long long)__mulhi(x.lo, w.lo) + (1LL << 31);
    m += (long long)x.hi * w.lo;
    m += (long long)x.lo * w.hi;
    return (m >> 32) + (long long)x.hi * w.hi;
}
// round((x w + y v) / 2^64)
__device__ __forceinline__ long long fx_prod2(FxLimbs x, FxLimbs w, FxLimbs y, FxLimbs v) {
    // |lo| <= 2^31 and |w0|, |v0| < 2^31: the two high words fit their sum
    long long m = (long long)(__mulhi(x.lo, w.lo) + __mulhi(y.lo, v.lo)) + (1LL << 31);
    m += (long long)x.hi * w.lo;
    m += (long long)x.lo * w.hi;
    m += (long long)y.hi * v.lo;
    m += (long long)y.lo * v.hi;
    long long h = m >> 32;
    h += (long long)x.hi * w.hi;
    h += (long long)y.hi * v.hi;
    return h;
}

// round(x c / 2^63) for a constant c as limbs, |x| < 2^62
__device__ __forceinline__ long long fx_mulq(long long x, FxLimbs c) { return fx_prod(fx_split<1>(x), c); }

// a times the table entry w (SIGN < 0) or its conjugate (SIGN > 0)
template <int SIGN, typename C> __device__ __forceinline__ C tw_mul(C a, C w) {
    if (SIGN > 0) w.y = -w.y;
    return cmul(a, w);
}
template <int SIGN> __device__ __forceinline__ fx2 tw_mul(fx2 a, fx2 w) {
    const FxLimbs ax = fx_split<2>(a.x), ay = fx_split<2>(a.y), wx = fx_packed(w.x), wy = fx_packed(w.y), ny = fx_neg(wy);
    return mk<fx2>(fx_prod2(ax, wx, ay, SIGN > 0 ? wy : ny), fx_prod2(ay, wx, ax, SIGN > 0 ? ny : wy));
}

// round(2^63 / sqrt 2), round(2^63 sqrt(3) / 2) as limbs
constexpr long long kFxInvSqrt2 = 6521908912666391106LL;
constexpr long long kFxSqrt3h = 7987674492471257551LL;
__host__ __device__ constexpr FxLimbs fx_const(long long w) {
    return {(int)(unsigned)(w & 0xFFFFFFFFLL), (int)(w >> 32) + (int)((unsigned)(w & 0xFFFFFFFFLL) >> 31)};
}

template <typename C> __host__ __device__ constexpr bool is_fx() { return std::is_same<C, fx2>::value; }

// Register DFTs, natural-order output, w = e^{SIGN 2 pi i / R}.
template <int SIGN, typename C> __device__ __forceinline__ void dft2(C* v) {
    const C a = v[0];
    v[0] = cadd(a, v[1]);
    v[1] = csub(a, v[1]);
}

template <int SIGN, typename C> __device__ __forceinline__ void dft4(C* v) {
    const C s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
    const C s13 = cadd(v[1], v[3]), d13 = mul_si<SIGN>(csub(v[1], v[3]));
    v[0] = cadd(s02, s13);
    v[2] = csub(s02, s13);
    v[1] = cadd(d02, d13);
    v[3] = csub(d02, d13);
}

// y[q] = E[q] + w8^q O[q], y[q+4] = E[q] - w8^q O[q] (E, O: 4-point DFTs of
// the even and odd inputs); w8 = (1 + SIGN i)/sqrt2, w8^2 = SIGN i,
// w8^3 = (-1 + SIGN i)/sqrt2.
template <int SIGN, typename C> __device__ __forceinline__ void dft8(C* v) {
    using R = decltype(C::x);
    C e[4] = {v[0], v[2], v[4], v[6]};
    C o[4] = {v[1], v[3], v[5], v[7]};
    dft4<SIGN>(e);
    dft4<SIGN>(o);
    C t1, t3;
    if constexpr (is_fx<C>()) {
        const long long s = SIGN;
        t1 = mk<C>(fx_mulq(o[1].x - s * o[1].y, fx_const(kFxInvSqrt2)), fx_mulq(o[1].y + s * o[1].x, fx_const(kFxInvSqrt2)));
        t3 = mk<C>(fx_mulq(-o[3].x - s * o[3].y, fx_const(kFxInvSqrt2)), fx_mulq(-o[3].y + s * o[3].x, fx_const(kFxInvSqrt2)));
    } else {
        const R h = (R)0.70710678118654752440;
        const R s = (R)SIGN;
        t1 = mk<C>(h * (o[1].x - s * o[1].y), h * (o[1].y + s * o[1].x));
        t3 = mk<C>(h * (-o[3].x - s * o[3].y), h * (-o[3].y + s * o[3].x));
    }
    const C t2 = mul_si<SIGN>(o[2]);
    v[0] = cadd(e[0], o[0]);
    v[4] = csub(e[0], o[0]);
    v[1] = cadd(e[1], t1);
    v[5] = csub(e[1], t1);
    v[2] = cadd(e[2], t2);
    v[6] = csub(e[2], t2);
    v[3] = cadd(e[3], t3);
    v[7] = csub(e[3], t3);
}

template <int SIGN, typename C> __device__ __forceinline__ void dft3(C* v) {
    using R = decltype(C::x);
    const C t1 = cadd(v[1], v[2]);
    const C d = csub(v[1], v[2]);
    C m, id;
    if constexpr (is_fx<C>()) {
        // t/2 rounded half up; sqrt(3)/2 as a Q63 constant
        m = mk<C>(v[0].x - ((t1.x + 1) >> 1), v[0].y - ((t1.y + 1) >> 1));
        const long long hx = fx_mulq(d.x, fx_const(kFxSqrt3h)), hy = fx_mulq(d.y, fx_const(kFxSqrt3h));
        id = SIGN > 0 ? mk<C>(-hy, hx) : mk<C>(hy, -hx);
    } else {
        const R h = (R)0.86602540378443864676;  // sqrt(3)/2
        m = mk<C>(v[0].x - (R)0.5 * t1.x, v[0].y - (R)0.5 * t1.y);
        id = SIGN > 0 ? mk<C>(-h * d.y, h * d.x) : mk<C>(h * d.y, -h * d.x);
    }
    v[0] = cadd(v[0], t1);
    v[1] = cadd(m, id);
    v[2] = csub(m, id);
}

template <int R, int SIGN, typename C> __device__ __forceinline__ void dft(C* v) {
    if constexpr (R == 8) dft8<SIGN>(v);
    else if constexpr (R == 4) dft4<SIGN>(v);
    else if constexpr (R == 2) dft2<SIGN>(v);
    else dft3<SIGN>(v);
}

// field pointer i of a by-value FieldsT without a dynamic index into the
// parameter block (which would copy the array to local memory)
template <typename P> __device__ __forceinline__ P* field_ptr(const FieldsT<P>& f, int i) {
    P* r = f.p[0];
#pragma unroll
    for (int k = 1; k < kMaxFields; ++k)
        if (i == k) r = f.p[k];
    return r;
}

__host__ __device__ constexpr int next_radix(int m) { return m % 8 == 0 ? 8 : (m % 4 == 0 ? 4 : (m % 2 == 0 ? 2 : 3)); }

// Transforms per CTA: a power of two near 2048 / N, in [1, 64].
__host__ __device__ constexpr int per_cta(int n) {
    int c = 1;
    while (c * 2 * n <= 2048 && c < 64) c *= 2;
    return c;
}

// Shared-memory slot of element t of one transform.  FP32 passes insert one
// padding slot after every 16 elements, so that a Stockham pass's writes at
// stride R (8 for the radix-8 passes) fall in distinct banks instead of in
// two: those passes are bound by shared-memory throughput.  The FP64 passes
// and the fixed-point ones of host transfers and diagnostics (16-byte elements,
// bound by their arithmetic) keep the plain layout, which needs fewer
// registers; the nonlinear term's integer passes pad every 8 (swp<3>, fft_nl.cu).
template <typename C> __host__ __device__ constexpr int sw(int t) {
    return std::is_same<C, float2>::value ? t + (t >> 4) : t;
}
// Slots per transform: elements 0..N (slot sw(N) holds an x pass's kx = nx/2 input).
template <typename C> __host__ __device__ constexpr int ld_of(int n) { return sw<C>(n) + 1; }

// One Stockham pass (radix R, Ns finished sub-length) over CNT transforms of
// length N stored at buf[c*LD + sw(t)], in place: all inputs of the thread's
// butterflies are read into registers before a barrier, then written.
// tw[t] = e^{-2 pi i t / N}.
// PAD: one padding slot after every 2^PAD elements (0: none).
template <int PAD> __host__ __device__ constexpr int swp(int t) { return PAD ? t + (t >> PAD) : t; }
template <typename C> __host__ __device__ constexpr int pad_of() { return std::is_same<C, float2>::value ? 4 : 0; }

template <int N, int R, int NS, int SIGN, int CNT, int LD, int PAD, typename C>
__device__ __forceinline__ void ct_pass(C* buf, const C* __restrict__ tw) {
    constexpr int NB = N / R;
    constexpr int TSTEP = N / (NS * R);
    constexpr int TOTAL = CNT * NB;
    constexpr int PER = (TOTAL + kThreads - 1) / kThreads;
    C v[PER][R];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int t = threadIdx.x + p * kThreads;
        if (TOTAL % kThreads == 0 || t < TOTAL) {
            const int c = t / NB, j = t - c * NB;
            const C* src = buf + c * LD;
#pragma unroll
            for (int r = 0; r < R; ++r) v[p][r] = src[swp<PAD>(j + r * NB)];
            if constexpr (NS > 1) {
                const int k = j % NS;
#pragma unroll
                for (int r = 1; r < R; ++r) {
                    v[p][r] = tw_mul<SIGN>(v[p][r], __ldg(&tw[r * k * TSTEP]));
                }
            }
            dft<R, SIGN>(v[p]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int t = threadIdx.x + p * kThreads;
        if (TOTAL % kThreads == 0 || t < TOTAL) {
            const int c = t / NB, j = t - c * NB;
            const int k = j % NS;
            C* dst = buf + c * LD;
            const int o = (j / NS) * NS * R + k;
#pragma unroll
            for (int q = 0; q < R; ++q) dst[swp<PAD>(o + q * NS)] = v[p][q];
        }
    }
    __syncthreads();
}

template <int N, int NS, int SIGN, int CNT, int LD, int PAD, typename C>
__device__ __forceinline__ void ct_fft_pad(C* buf, const C* __restrict__ tw) {
    if constexpr (NS < N) {
        constexpr int R = next_radix(N / NS);
        ct_pass<N, R, NS, SIGN, CNT, LD, PAD>(buf, tw);
        ct_fft_pad<N, NS * R, SIGN, CNT, LD, PAD>(buf, tw);
    }
}
template <int N, int NS, int SIGN, int CNT, int LD, typename C>
__device__ __forceinline__ void ct_fft(C* buf, const C* __restrict__ tw) {
    ct_fft_pad<N, NS, SIGN, CNT, LD, pad_of<C>()>(buf, tw);
}

// Conversions between FP64 and a transform's fixed-point grid, integer
// operations only.  A transform whose largest input has biased exponent em
// (|x| < 2^(em - 1022)) stores x as X = round(x 2^(B - em + 1022)), so that
// |X| <= 2^B, and an output X stands for X 2^(em - 1022 - B).

// Significant bits of a transform's largest input: 53, less whatever a length
// n transform (log2 n + 1 bits, the +1 for a complex modulus) and `extra` bits
// of packing growth need below 2^62.
__host__ __device__ constexpr int fx_bits(int n, int extra) {
    int l = 0;
    while ((1 << l) < n) ++l;
    return 62 - l - 1 - extra < 53 ? 62 - l - 1 - extra : 53;
}

__device__ __forceinline__ unsigned fx_expo(double x) { return ((unsigned)__double2hiint(x) >> 20) & 0x7FFu; }
__device__ __forceinline__ unsigned fx_expo(double2 v) { return max(fx_expo(v.x), fx_expo(v.y)); }

// round(x 2^(B - em + 1022)) given rsb = 53 - B + em (em >= 1, B <= 53): the
// mantissa m of x = m 2^(ex - 1075) shifted right by rsb - ex >= 0, half up.
__device__ __forceinline__ long long fx_from(double x, int rsb) {
    const long long b = __double_as_longlong(x);
    const int ex = (int)((b >> 52) & 0x7FF);
    const long long m = (b & 0xFFFFFFFFFFFFFLL) | (ex ? (1LL << 52) : 0LL);
    unsigned long long t;  // 2 m >> (rsb - ex), zero from a shift of 64 on
    asm("shr.u64 %0, %1, %2;" : "=l"(t) : "l"((unsigned long long)m << 1), "r"(rsb - max(ex, 1)));
    const long long u = (long long)((t + 1) >> 1);
    return b < 0 ? -u : u;
}

__device__ __forceinline__ double fx_to(long long X, int e2) { return i2d_scaled(X, e2); }

__device__ __forceinline__ double fx_nan() { return __longlong_as_double(0x7FF8000000000000LL); }

// emax[key] = max(emax[key], e) over the calling warp's lanes, one shared
// atomic per distinct key.  Every lane of the warp must call it.
__device__ __forceinline__ void fx_key_max(unsigned* emax, int key, unsigned e) {
    const unsigned grp = __match_any_sync(0xFFFFFFFFu, key);
    e = __reduce_max_sync(grp, e);
    if ((threadIdx.x & 31) == __ffs(grp) - 1) atomicMax(&emax[key], e);
}

// y pass: complex transforms of length N = ny along the (plane, kx) columns
// with kx < ncol (ncol = nx/2+1, or fewer when the 2/3 filter discards the
// rest); CX columns per CTA taken from the flattened index plane * ncol + kx.
// grid (ceil(nplanes * ncol / CX), 1, nf).
// Block bx of field f; buf holds at least per_cta(N) ld_of(N) values.  S: type
// of the source spectra (an FP32 pass may read FP64 ones, rounded on loading).
__device__ __forceinline__ float2 load_as(float2 a, float2) { return a; }
__device__ __forceinline__ double2 load_as(double2 a, double2) { return a; }
__device__ __forceinline__ float2 load_as(double2 a, float2) { return d2f(a); }

template <int N, int SIGN, typename C, typename S = C>
__device__ __forceinline__ void fft_y_body(const FieldsT<S>& src, const FieldsT<C>& dst, const GridDev& g,
                                           int nplanes, int ncol, const C* __restrict__ tw, int bx, int f,
                                           C* buf) {
    constexpr int CX = per_cta(N);
    constexpr int LD = ld_of<C>(N);
    const long long ncols = (long long)nplanes * ncol;
    const long long vc = (long long)bx * CX + (threadIdx.x % CX);
    const bool live = vc < ncols;
    size_t base = 0;
    if (live) {
        const int p = (int)(vc / ncol);
        const int kx = (int)(vc - (long long)p * ncol);
        base = (size_t)p * g.nm + kx;
    }
    const S* __restrict__ s = field_ptr(src, f);
    C* d = field_ptr(dst, f);
    constexpr int ROWS_PER_ITER = kThreads / CX;  // CX divides kThreads
    constexpr int ITERS = N / ROWS_PER_ITER;
    static_assert(N % ROWS_PER_ITER == 0, "rows split evenly over the threads");
    const int c = threadIdx.x % CX, y0 = threadIdx.x / CX;
    // all of a thread's loads are issued before any is used
    C v[ITERS];
#pragma unroll
    for (int it = 0; it < ITERS; ++it)
        v[it] = live ? load_as(s[base + (size_t)(y0 + it * ROWS_PER_ITER) * g.nxhp], C{}) : mk<C>(0, 0);
#pragma unroll
    for (int it = 0; it < ITERS; ++it) buf[c * LD + sw<C>(y0 + it * ROWS_PER_ITER)] = v[it];
    __syncthreads();
    ct_fft<N, 1, SIGN, CX, LD>(buf, tw);
    if (live) {
#pragma unroll
        for (int it = 0; it < ITERS; ++it)
            d[base + (size_t)(y0 + it * ROWS_PER_ITER) * g.nxhp] = buf[c * LD + sw<C>(y0 + it * ROWS_PER_ITER)];
    }
}

// x 2^-s rounded to nearest (half up) for s > 0, x 2^-s exactly for s <= 0
// (the caller keeps it below 2^63); shifts from 64 on give 0 (PTX clamps them).
__device__ __forceinline__ long long fx_rshift(long long x, int s) {
    long long t;
    if (s > 0) {
        asm("shr.s64 %0, %1, %2;" : "=l"(t) : "l"(x), "r"(s - 1));
        return (t + 1) >> 1;
    }
    asm("shl.b64 %0, %1, %2;" : "=l"(t) : "l"(x), "r"(-s));
    return t;
}

}  // namespace

}  // namespace dns3d
