// Plane transforms with the transform length fixed at compile time: the same
// transforms as fft.cu (FFTW's r2c / non-Hermitian c2r conventions), for the
// lengths that the supported grids use, with
//  - the radix schedule, the per-pass index arithmetic and the loop trip
//    counts resolved by the compiler (no runtime division in the passes);
//  - radix-8 butterflies in registers (a length-128 transform is 3 passes
//    instead of 4, length 512 is 3 instead of 5);
//  - one shared-memory buffer per CTA: each pass reads all of a thread's
//    butterfly inputs into registers, synchronises, and writes the outputs
//    in place, so a CTA holds ~2048 complex values in 16-33 KB (no opt-in);
//  - the y pass over a flattened (plane, kx) column index, so grids whose
//    nx/2+1 columns do not fill a CTA waste no lanes.
// Lengths outside the instantiated set use the generic kernels of fft.cu.
#include "fft_dev.cuh"
#include "ragged.cuh"
#include "tc.cuh"

namespace dns3d {

namespace {

template <int N, int SIGN, typename C>
__global__ void __launch_bounds__(kThreads) k_fft_y_ct(FieldsT<C> src, FieldsT<C> dst, GridDev g, int nplanes,
                                                       int ncol, const C* __restrict__ tw) {
    __shared__ C buf[per_cta(N) * ld_of<C>(N)];
    fft_y_body<N, SIGN, C>(src, dst, g, nplanes, ncol, tw, blockIdx.x, blockIdx.z, buf);
}

// c2r along x on the FP64 pipe, N = nx/2: RX rows per CTA (row = plane * ny + y).  Packs the
// nx/2+1 inputs of a row (Re only at kx = 0, nx/2) into Z[k] =
// (X[k] + conj(X[N-k])) + i e^{+2 pi i k/nx} (X[k] - conj(X[N-k])), runs the
// inverse length-N transform and writes z[m] = (x[2m], x[2m+1]) / (nx ny).
template <int N>
__device__ __forceinline__ void c2r_x_body(const Fields& src, const RFields& dst, const GridDev& g, int nrows,
                                           const double2* __restrict__ tw_n, const double2* __restrict__ tw_nx,
                                           int bx, int f, double2* buf) {
    using C = double2;
    constexpr int RX = per_cta(N);
    constexpr int LD = ld_of<C>(N);
    const int row0 = bx * RX;
    const C* __restrict__ s = field_ptr(src, f);
    C* d = reinterpret_cast<C*>(field_ptr(dst, f));
    const int nxhp = N + 1;
    constexpr int ITERS = RX * N / kThreads;
    static_assert((RX * N) % kThreads == 0, "rows split evenly over the threads");
    // all of a thread's loads are issued before any is used
    C xa[ITERS], xb[ITERS];
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        xa[it] = xb[it] = mk<C>(0, 0);
        if (row0 + r < nrows) {
            const C* row = s + (size_t)(row0 + r) * nxhp;
            xa[it] = row[k];
            xb[it] = row[N - k];
        }
    }
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        C a = xa[it], b = xb[it];
        if (k == 0) {
            a.y = 0;
            b.y = 0;
        }
        const C sm = mk<C>(a.x + b.x, a.y - b.y);
        const C df = mk<C>(a.x - b.x, a.y + b.y);
        C w = __ldg(&tw_nx[k]);
        w.y = -w.y;
        const C p = cmul(w, df);
        buf[r * LD + sw<C>(k)] = mk<C>(sm.x - p.y, sm.y + p.x);
    }
    __syncthreads();
    ct_fft<N, 1, +1, RX, LD>(buf, tw_n);
    const double sc = g.inv_nxny;
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        if (row0 + r < nrows) {
            const C z = buf[r * LD + sw<C>(k)];
            d[(size_t)(row0 + r) * N + k] = mk<C>(z.x * sc, z.y * sc);
        }
    }
}

template <int N>
__global__ void __launch_bounds__(kThreads) k_c2r_x_ct(Fields src, RFields dst, GridDev g, int nrows,
                                                       const double2* __restrict__ tw_n,
                                                       const double2* __restrict__ tw_nx) {
    __shared__ double2 buf[per_cta(N) * ld_of<double2>(N)];
    c2r_x_body<N>(src, dst, g, nrows, tw_n, tw_nx, blockIdx.x, blockIdx.y, buf);
}

// r2c along x, N = nx/2: z[m] = x[2m] + i x[2m+1], forward length-N
// transform, X[k] = E + e^{-2 pi i k/nx} O with E = (Z[k] + conj(Z[N-k]))/2,
// O = (Z[k] - conj(Z[N-k]))/(2i), k = 0..N.
template <int N>
__device__ __forceinline__ void r2c_x_body(const RFields& src, const Fields& dst, const GridDev& g, int nrows,
                                           const double2* __restrict__ tw_n, const double2* __restrict__ tw_nx,
                                           int bx, int f, double2* buf) {
    using C = double2;
    constexpr int RX = per_cta(N);
    constexpr int LD = ld_of<C>(N);
    const int row0 = bx * RX;
    const C* __restrict__ s = reinterpret_cast<const C*>(field_ptr(src, f));
    C* d = field_ptr(dst, f);
    constexpr int ITERS = RX * N / kThreads;
    static_assert((RX * N) % kThreads == 0, "rows split evenly over the threads");
    C v[ITERS];
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        v[it] = (row0 + r < nrows) ? s[(size_t)(row0 + r) * N + k] : mk<C>(0, 0);
    }
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        buf[r * LD + sw<C>(k)] = v[it];
    }
    __syncthreads();
    ct_fft<N, 1, -1, RX, LD>(buf, tw_n);
    for (int t = threadIdx.x; t < RX * (N + 1); t += kThreads) {
        const int r = t / (N + 1), k = t - r * (N + 1);
        if (row0 + r < nrows) {
            const C za = buf[r * LD + sw<C>(k == N ? 0 : k)];
            const C zb = buf[r * LD + sw<C>(k == 0 ? 0 : N - k)];
            const double hf = 0.5;
            const C e = mk<C>(hf * (za.x + zb.x), hf * (za.y - zb.y));
            const C o = mk<C>(hf * (za.y + zb.y), -hf * (za.x - zb.x));
            const C p = cmul(__ldg(&tw_nx[k]), o);
            d[(size_t)(row0 + r) * (N + 1) + k] = mk<C>(e.x + p.x, e.y + p.y);
        }
    }
}

template <int N>
__global__ void __launch_bounds__(kThreads) k_r2c_x_ct(RFields src, Fields dst, GridDev g, int nrows,
                                                       const double2* __restrict__ tw_n,
                                                       const double2* __restrict__ tw_nx) {
    __shared__ double2 buf[per_cta(N) * ld_of<double2>(N)];
    r2c_x_body<N>(src, dst, g, nrows, tw_n, tw_nx, blockIdx.x, blockIdx.y, buf);
}

// ------------------------------------------------------------------ fixed-point passes
// y pass in fixed point (FP64 fields); emax holds per_cta(N) exponents.
template <int N, int SIGN>
__device__ __forceinline__ void fft_y_body_fx(const Fields& src, const Fields& dst, const GridDev& g, int nplanes,
                                              int ncol, const fx2* __restrict__ tw, int bx, int f, fx2* buf,
                                              unsigned* emax) {
    constexpr int CX = per_cta(N);
    constexpr int LD = ld_of<fx2>(N);
    constexpr int B = fx_bits(N, 0);
    const long long ncols = (long long)nplanes * ncol;
    const long long vc = (long long)bx * CX + (threadIdx.x % CX);
    const bool live = vc < ncols;
    size_t base = 0;
    if (live) {
        const int p = (int)(vc / ncol);
        const int kx = (int)(vc - (long long)p * ncol);
        base = (size_t)p * g.nm + kx;
    }
    const double2* __restrict__ s = field_ptr(src, f);
    double2* d = field_ptr(dst, f);
    constexpr int ROWS_PER_ITER = kThreads / CX;
    constexpr int ITERS = N / ROWS_PER_ITER;
    static_assert(N % ROWS_PER_ITER == 0, "rows split evenly over the threads");
    const int c = threadIdx.x % CX, y0 = threadIdx.x / CX;
    if (threadIdx.x < CX) emax[threadIdx.x] = 1u;
    double2 v[ITERS];
    unsigned e = 1u;
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        v[it] = live ? s[base + (size_t)(y0 + it * ROWS_PER_ITER) * g.nxhp] : make_double2(0.0, 0.0);
        e = max(e, fx_expo(v[it]));
    }
    __syncthreads();
    fx_key_max(emax, c, e);
    __syncthreads();
    const int em = (int)emax[c];
    const int rsb = 53 - B + em;
#pragma unroll
    for (int it = 0; it < ITERS; ++it)
        buf[c * LD + sw<fx2>(y0 + it * ROWS_PER_ITER)] = mk<fx2>(fx_from(v[it].x, rsb), fx_from(v[it].y, rsb));
    __syncthreads();
    ct_fft<N, 1, SIGN, CX, LD>(buf, tw);
    if (live) {
        const int e2 = em - 1022 - B;
#pragma unroll
        for (int it = 0; it < ITERS; ++it) {
            const fx2 z = buf[c * LD + sw<fx2>(y0 + it * ROWS_PER_ITER)];
            d[base + (size_t)(y0 + it * ROWS_PER_ITER) * g.nxhp] =
                em == 0x7FF ? make_double2(fx_nan(), fx_nan()) : make_double2(fx_to(z.x, e2), fx_to(z.y, e2));
        }
    }
}

template <int N, int SIGN>
__global__ void __launch_bounds__(kThreads) k_fft_y_fx(Fields src, Fields dst, GridDev g, int nplanes, int ncol,
                                                       const fx2* __restrict__ tw) {
    __shared__ fx2 buf[per_cta(N) * ld_of<fx2>(N)];
    __shared__ unsigned emax[per_cta(N)];
    fft_y_body_fx<N, SIGN>(src, dst, g, nplanes, ncol, tw, blockIdx.x, blockIdx.z, buf, emax);
}

// c2r along x in fixed point: the packing of c2r_x_body (inputs of one row
// scaled together, the packing's growth of 4 within the headroom), the
// inverse transform, and the 1/(nx ny) scaling as a multiple of the FP64
// constant's mantissa rounded once.
template <int N>
__device__ __forceinline__ void c2r_x_body_fx(const Fields& src, const RFields& dst, const RFields& dst2,
                                              const GridDev& g, int nrows, const fx2* __restrict__ tw_n,
                                              const fx2* __restrict__ tw_nx, int bx, int f, fx2* buf,
                                              unsigned* emax, uint64_t* mbar) {
    constexpr int RX = per_cta(N);
    constexpr int LD = ld_of<fx2>(N);
    constexpr int B = fx_bits(N, 2);
    const int row0 = bx * RX;
    const double2* __restrict__ s = field_ptr(src, f);
    double2* d = reinterpret_cast<double2*>(field_ptr(dst, f));
    double2* d2 = reinterpret_cast<double2*>(field_ptr(dst2, f));  // optional second copy (null: none)
    const int nxhp = N + 1;
    constexpr int ITERS = RX * N / kThreads;
    static_assert((RX * N) % kThreads == 0, "rows split evenly over the threads");
    if (threadIdx.x < RX) emax[threadIdx.x] = 1u;
    // The CTA's rows are contiguous in memory and the fixed-point slots are
    // as wide as a complex FP64 value, so one bulk copy (TMA engine, completion
    // on an mbarrier) stages the rows' nx/2+1 inputs into the slots as they
    // are; a copy that does not land within the wait limit marks the rows
    // non-finite.
    const int nvalid = min(RX, nrows - row0);
    if (threadIdx.x == 0) tc_mbar_init(mbar);
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t bytes = (uint32_t)nvalid * (uint32_t)nxhp * (uint32_t)sizeof(fx2);
        tc_mbar_expect(mbar, bytes);
        tc_bulk_g2s(buf, s + (size_t)row0 * nxhp, bytes, mbar);
    }
    const bool landed = __syncthreads_and(tc_mbar_wait(mbar, 0, 1 << 22));
    unsigned e[ITERS];
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        fx2 ra = buf[r * LD + sw<fx2>(k)], rb = mk<fx2>(0, 0);
        if (k == 0) {  // Im of kx = 0 and kx = nx/2 is ignored
            rb = buf[r * LD + sw<fx2>(N)];
            ra.y = 0;
            rb.y = 0;
        }
        e[it] = landed ? max(fx_expo(__longlong_as_double(ra.x)), max(fx_expo(__longlong_as_double(ra.y)),
                                                                      max(fx_expo(__longlong_as_double(rb.x)),
                                                                          fx_expo(__longlong_as_double(rb.y)))))
                       : 0x7FFu;
    }
#pragma unroll
    for (int it = 0; it < ITERS; ++it) fx_key_max(emax, (threadIdx.x + it * kThreads) / N, e[it]);
    __syncthreads();
    fx2 z[ITERS];
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        const int rsb = 53 - B + (int)emax[r];
        fx2 ra = buf[r * LD + sw<fx2>(k)], rb = buf[r * LD + sw<fx2>(N - k)];
        if (k == 0) {  // Im of kx = 0 and kx = nx/2 is ignored
            ra.y = 0;
            rb.y = 0;
        }
        const fx2 a = mk<fx2>(fx_from(__longlong_as_double(ra.x), rsb), fx_from(__longlong_as_double(ra.y), rsb));
        const fx2 b = mk<fx2>(fx_from(__longlong_as_double(rb.x), rsb), fx_from(__longlong_as_double(rb.y), rsb));
        const fx2 sm = mk<fx2>(a.x + b.x, a.y - b.y);
        const fx2 df = mk<fx2>(a.x - b.x, a.y + b.y);
        const fx2 p = tw_mul<+1>(df, __ldg(&tw_nx[k]));
        z[it] = mk<fx2>(sm.x - p.y, sm.y + p.x);
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        buf[(t / N) * LD + sw<fx2>(t % N)] = z[it];
    }
    __syncthreads();
    ct_fft<N, 1, +1, RX, LD>(buf, tw_n);
    // 1/(nx ny) = M 2^(E - 1075), M its 53-bit mantissa: Y = round(Z M / 2^52),
    // no coarser than Z (over 2^63, as the limb products give it, a constant
    // field came back two bits short)
    const long long sb = __double_as_longlong(g.inv_nxny);
    const long long M = (sb & 0xFFFFFFFFFFFFFLL) | (1LL << 52);
    const int E = (int)((sb >> 52) & 0x7FF);
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        if (row0 + r < nrows) {
            const int em = (int)emax[r];
            const int e2 = em + E - 2045 - B;
            const fx2 z = buf[r * LD + sw<fx2>(k)];
            const long long yx = (long long)(((__int128)z.x * M + ((__int128)1 << 51)) >> 52);
            const long long yy = (long long)(((__int128)z.y * M + ((__int128)1 << 51)) >> 52);
            const double2 o =
                em == 0x7FF ? make_double2(fx_nan(), fx_nan()) : make_double2(fx_to(yx, e2), fx_to(yy, e2));
            d[(size_t)(row0 + r) * N + k] = o;
            if (d2) d2[(size_t)(row0 + r) * N + k] = o;
        }
    }
}

template <int N>
__global__ void __launch_bounds__(kThreads, 3) k_c2r_x_fx(Fields src, RFields dst, RFields dst2, GridDev g,
                                                          int nrows, const fx2* __restrict__ tw_n,
                                                          const fx2* __restrict__ tw_nx) {
    __shared__ fx2 buf[per_cta(N) * ld_of<fx2>(N)];
    __shared__ unsigned emax[per_cta(N)];
    __shared__ uint64_t mbar;
    c2r_x_body_fx<N>(src, dst, dst2, g, nrows, tw_n, tw_nx, blockIdx.x, blockIdx.y, buf, emax, &mbar);
}

// r2c along x in fixed point: z[m] = x[2m] + i x[2m+1] of one row scaled
// together, forward transform, and 2 X[k] = (Z[k] + conj Z[N-k]) +
// e^{-2 pi i k/nx} (-i)(Z[k] - conj Z[N-k]) formed exactly, the factor 1/2
// taken into the exponent.
template <int N>
__device__ __forceinline__ void r2c_x_body_fx(const RFields& src, const Fields& dst, const GridDev& g, int nrows,
                                              const fx2* __restrict__ tw_n, const fx2* __restrict__ tw_nx, int bx,
                                              int f, fx2* buf, unsigned* emax, uint64_t* mbar, bool bulk) {
    constexpr int RX = per_cta(N);
    constexpr int LD = N;  // rows back to back, as in memory (no kx = nx/2 slot needed)
    constexpr int B = fx_bits(N, 2);
    const int row0 = bx * RX;
    const double2* __restrict__ s = reinterpret_cast<const double2*>(field_ptr(src, f));
    double2* d = field_ptr(dst, f);
    constexpr int ITERS = RX * N / kThreads;
    static_assert((RX * N) % kThreads == 0, "rows split evenly over the threads");
    if (threadIdx.x < RX) emax[threadIdx.x] = 1u;
    // the rows' FP64 values go into the fixed-point slots as they are (z[m] =
    // x[2m] + i x[2m+1] is the row's own memory layout, and the CTA's rows are
    // contiguous): from device memory by one bulk copy (TMA engine,
    // completion on an mbarrier; a copy that does not land within the wait
    // limit marks the rows non-finite), from host memory the device maps
    // (pinned buffers read in place) by plain loads
    const int nvalid = min(RX, nrows - row0);
    bool landed = true;
    if (bulk) {
        if (threadIdx.x == 0) tc_mbar_init(mbar);
        __syncthreads();
        if (threadIdx.x == 0) {
            const uint32_t bytes = (uint32_t)nvalid * (uint32_t)(N * sizeof(fx2));
            tc_mbar_expect(mbar, bytes);
            tc_bulk_g2s(buf, s + (size_t)row0 * N, bytes, mbar);
        }
        landed = __syncthreads_and(tc_mbar_wait(mbar, 0, 1 << 22));
    } else {
        double2 h[ITERS];
#pragma unroll
        for (int it = 0; it < ITERS; ++it) {
            const int t = threadIdx.x + it * kThreads;
            const int r = t / N, k = t - r * N;
            h[it] = r < nvalid ? s[(size_t)(row0 + r) * N + k] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int it = 0; it < ITERS; ++it) {
            const int t = threadIdx.x + it * kThreads;
            buf[(t / N) * LD + sw<fx2>(t % N)] = mk<fx2>(__double_as_longlong(h[it].x), __double_as_longlong(h[it].y));
        }
        __syncthreads();
    }
    fx2 v[ITERS];
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        v[it] = buf[r * LD + sw<fx2>(k)];
        fx_key_max(emax, r,
                   landed ? max(fx_expo(__longlong_as_double(v[it].x)), fx_expo(__longlong_as_double(v[it].y)))
                          : 0x7FFu);
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int t = threadIdx.x + it * kThreads;
        const int r = t / N, k = t - r * N;
        const int rsb = 53 - B + (int)emax[r];
        buf[r * LD + sw<fx2>(k)] = mk<fx2>(fx_from(__longlong_as_double(v[it].x), rsb),
                                           fx_from(__longlong_as_double(v[it].y), rsb));
    }
    __syncthreads();
    ct_fft<N, 1, -1, RX, LD>(buf, tw_n);
    for (int t = threadIdx.x; t < RX * (N + 1); t += kThreads) {
        const int r = t / (N + 1), k = t - r * (N + 1);
        if (row0 + r < nrows) {
            const fx2 za = buf[r * LD + sw<fx2>(k == N ? 0 : k)];
            const fx2 zb = buf[r * LD + sw<fx2>(k == 0 ? 0 : N - k)];
            const fx2 e = mk<fx2>(za.x + zb.x, za.y - zb.y);
            const fx2 o = mk<fx2>(za.y + zb.y, zb.x - za.x);
            const fx2 p = tw_mul<-1>(o, __ldg(&tw_nx[k]));
            const int em = (int)emax[r];
            const int e2 = em - 1023 - B;
            d[(size_t)(row0 + r) * (N + 1) + k] = em == 0x7FF
                                                      ? make_double2(fx_nan(), fx_nan())
                                                      : make_double2(fx_to(e.x + p.x, e2), fx_to(e.y + p.y, e2));
        }
    }
}

template <int N>
__global__ void __launch_bounds__(kThreads) k_r2c_x_fx(RFields src, Fields dst, GridDev g, int nrows,
                                                       const fx2* __restrict__ tw_n, const fx2* __restrict__ tw_nx,
                                                       int bulk) {
    __shared__ fx2 buf[per_cta(N) * ld_of<fx2>(N)];
    __shared__ unsigned emax[per_cta(N)];
    __shared__ uint64_t mbar;
    r2c_x_body_fx<N>(src, dst, g, nrows, tw_n, tw_nx, blockIdx.x, blockIdx.y, buf, emax, &mbar, bulk != 0);
}

// ------------------------------------------------------------------ ragged stages
// The four transform passes of the nonlinear term over many runs in one launch
// (k_stage, ragged.cuh): the transform length is a run property, so each CTA
// switches to the compile-time kernel body of its run's length and uses one
// shared buffer sized for the longest.
__host__ __device__ constexpr int ct_buf_max() {
    int m = 0;
#define BUF_MAX(n) m = (per_cta(n) * ld_of<float2>(n) > m) ? per_cta(n) * ld_of<float2>(n) : m;
    DNS3D_CT_Y_LENGTHS(BUF_MAX)
    DNS3D_CT_X_LENGTHS(BUF_MAX)
#undef BUF_MAX
    return m;
}

// Field f of a descriptor pointer list as field 0 of a FieldsT: the bodies
// then select field 0, and only the one pointer is held in registers.
template <typename P>
__device__ __forceinline__ FieldsT<P> one_field(void* const* p, int f) {
    FieldsT<P> r;
#pragma unroll
    for (int i = 0; i < kMaxFields; ++i) r.p[i] = nullptr;
    r.p[0] = static_cast<P*>(p[f]);
    return r;
}

// y pass: inverse over three of the six inputs (F0 = 0: the state u, v, w,
// F0 = 3: the vorticity; S the spectra's type) into the scratch fields, or
// forward in place over the three sources (2/3-filtered columns only).
template <int SIGN, int F0, typename T, typename S>
struct RsFftY {
    static constexpr int kMinCtas = sizeof(T) == 8 ? 3 : 4;
    static __device__ __forceinline__ void run(const RunDesc& d, int b) {
        using C = typename Cx<T>::type;
        __shared__ C buf[ct_buf_max()];
        const int gx = d.gx[SIGN > 0 ? kRsFftYInv : kRsFftYFwd];
        const int f = b / gx, bx = b - f * gx;
        const FieldsT<S> src = one_field<S>(SIGN > 0 ? d.spec : d.src, F0 + f);
        const FieldsT<C> dst = one_field<C>(SIGN > 0 ? d.tmp : d.src, F0 + f);
        const int ncol = SIGN > 0 ? d.g.nxhp : d.ncol;
        const C* tw = static_cast<const C*>(d.tw_ny);
        switch (d.g.ny) {
#define Y_CASE(n) \
    case n: fft_y_body<n, SIGN, C, S>(src, dst, d.g, d.g.nz, ncol, tw, bx, 0, buf); break;
            DNS3D_CT_Y_LENGTHS(Y_CASE)
#undef Y_CASE
        }
    }
};

struct RsC2R {
    static constexpr int kMinCtas = 2;
    static __device__ __forceinline__ void run(const RunDesc& d, int b) {
        using C = double2;
        __shared__ C buf[ct_buf_max()];
        const int gx = d.gx[kRsFftC2R];
        const int f = b / gx, bx = b - f * gx;
        const C* twn = static_cast<const C*>(d.tw_nx2);
        const C* twx = static_cast<const C*>(d.tw_nx);
        switch (d.g.nxh) {
#define X_CASE(n) \
    case n: \
        c2r_x_body<n>(one_field<C>(d.tmp, f), one_field<double>(d.phys, f), d.g, d.g.nz * d.g.ny, twn, twx, bx, \
                         0, buf); \
        break;
            DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        }
    }
};

struct RsR2C {
    static constexpr int kMinCtas = 3;
    static __device__ __forceinline__ void run(const RunDesc& d, int b) {
        using C = double2;
        __shared__ C buf[ct_buf_max()];
        const int gx = d.gx[kRsFftR2C];
        const int f = b / gx, bx = b - f * gx;
        const C* twn = static_cast<const C*>(d.tw_nx2);
        const C* twx = static_cast<const C*>(d.tw_nx);
        switch (d.g.nxh) {
#define X_CASE(n) \
    case n: \
        r2c_x_body<n>(one_field<double>(d.phys, f), one_field<C>(d.src, f), d.g, d.g.nz * d.g.ny, twn, twx, bx, \
                         0, buf); \
        break;
            DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        }
    }
};

}  // namespace

int fft_ct_per_cta(int n) { return per_cta(n); }

StageKernel ragged_fft_kernel(int stage, bool mixed, bool fx) {
    if (!mixed && fx && (stage == kRsFftYUvw || stage == kRsFftYInv || stage == kRsFftYFwd))
        return ragged_nl_kernel(stage, mixed);
    switch (stage) {
        case kRsFftYUvw:
            return mixed ? k_stage<RsFftY<+1, 0, float, double2>> : k_stage<RsFftY<+1, 0, double, double2>>;
        case kRsFftYInv:
            return mixed ? k_stage<RsFftY<+1, 3, float, float2>> : k_stage<RsFftY<+1, 3, double, double2>>;
        case kRsFftC2R: return k_stage<RsC2R>;
        case kRsFftR2C: return k_stage<RsR2C>;
        case kRsFftYFwd:
            return mixed ? k_stage<RsFftY<-1, 0, float, float2>> : k_stage<RsFftY<-1, 0, double, double2>>;
    }
    return nullptr;
}

namespace {

template <int SIGN, typename C, int N>
void launch_y(FieldsT<C> src, FieldsT<C> dst, const GridDev& g, int nplanes, int ncol, int nf, const C* tw,
              cudaStream_t s) {
    constexpr int CX = per_cta(N);
    const long long ncols = (long long)nplanes * ncol;
    dim3 grid((unsigned)((ncols + CX - 1) / CX), 1, nf);
    k_fft_y_ct<N, SIGN, C><<<grid, kThreads, 0, s>>>(src, dst, g, nplanes, ncol, tw);
}

template <int N>
void launch_c2r(Fields src, RFields dst, const GridDev& g, int nrows, int nf, const double2* tw_n,
                const double2* tw_nx, cudaStream_t s) {
    constexpr int RX = per_cta(N);
    dim3 grid((nrows + RX - 1) / RX, nf);
    k_c2r_x_ct<N><<<grid, kThreads, 0, s>>>(src, dst, g, nrows, tw_n, tw_nx);
}

template <int N>
void launch_r2c(RFields src, Fields dst, const GridDev& g, int nrows, int nf, const double2* tw_n,
                const double2* tw_nx, cudaStream_t s) {
    constexpr int RX = per_cta(N);
    dim3 grid((nrows + RX - 1) / RX, nf);
    k_r2c_x_ct<N><<<grid, kThreads, 0, s>>>(src, dst, g, nrows, tw_n, tw_nx);
}

template <int SIGN, int N>
void launch_y_fx(Fields src, Fields dst, const GridDev& g, int nplanes, int ncol, int nf, const fx2* tw,
                 cudaStream_t s) {
    constexpr int CX = per_cta(N);
    const long long ncols = (long long)nplanes * ncol;
    dim3 grid((unsigned)((ncols + CX - 1) / CX), 1, nf);
    k_fft_y_fx<N, SIGN><<<grid, kThreads, 0, s>>>(src, dst, g, nplanes, ncol, tw);
}

template <int N>
void launch_c2r_fx(Fields src, RFields dst, RFields dst2, const GridDev& g, int nrows, int nf, const fx2* tw_n,
                   const fx2* tw_nx, cudaStream_t s) {
    constexpr int RX = per_cta(N);
    dim3 grid((nrows + RX - 1) / RX, nf);
    k_c2r_x_fx<N><<<grid, kThreads, 0, s>>>(src, dst, dst2, g, nrows, tw_n, tw_nx);
}

template <int N>
void launch_r2c_fx(RFields src, Fields dst, const GridDev& g, int nrows, int nf, const fx2* tw_n, const fx2* tw_nx,
                   bool host_src, cudaStream_t s) {
    constexpr int RX = per_cta(N);
    dim3 grid((nrows + RX - 1) / RX, nf);
    k_r2c_x_fx<N><<<grid, kThreads, 0, s>>>(src, dst, g, nrows, tw_n, tw_nx, host_src ? 0 : 1);
}

}  // namespace


bool fft_ct_supported(int ny, int nxh) {
    bool y = false, x = false;
#define Y_CASE(n) y = y || ny == n;
#define X_CASE(n) x = x || nxh == n;
    DNS3D_CT_Y_LENGTHS(Y_CASE)
    DNS3D_CT_X_LENGTHS(X_CASE)
#undef Y_CASE
#undef X_CASE
    return y && x;
}

template <int SIGN, typename C>
cudaError_t fft_ct_y(FieldsT<C> src, FieldsT<C> dst, const GridDev& g, int nplanes, int ncol, int nf, const C* tw,
                     cudaStream_t s) {
    if (ncol < 1 || ncol > g.nxhp) return cudaErrorInvalidValue;
    switch (g.ny) {
#define Y_CASE(n) \
    case n: launch_y<SIGN, C, n>(src, dst, g, nplanes, ncol, nf, tw, s); break;
        DNS3D_CT_Y_LENGTHS(Y_CASE)
#undef Y_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t fft_ct_c2r_x(Fields src, RFields dst, const GridDev& g, int nrows, int nf, const double2* tw_n,
                         const double2* tw_nx, cudaStream_t s) {
    switch (g.nxh) {
#define X_CASE(n) \
    case n: launch_c2r<n>(src, dst, g, nrows, nf, tw_n, tw_nx, s); break;
        DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t fft_ct_r2c_x(RFields src, Fields dst, const GridDev& g, int nrows, int nf, const double2* tw_n,
                         const double2* tw_nx, cudaStream_t s) {
    switch (g.nxh) {
#define X_CASE(n) \
    case n: launch_r2c<n>(src, dst, g, nrows, nf, tw_n, tw_nx, s); break;
        DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <int SIGN>
cudaError_t fft_fx_y(Fields src, Fields dst, const GridDev& g, int nplanes, int ncol, int nf, const longlong2* tw,
                     cudaStream_t s) {
    if (ncol < 1 || ncol > g.nxhp) return cudaErrorInvalidValue;
    switch (g.ny) {
#define Y_CASE(n) \
    case n: launch_y_fx<SIGN, n>(src, dst, g, nplanes, ncol, nf, tw, s); break;
        DNS3D_CT_Y_LENGTHS(Y_CASE)
#undef Y_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t fft_fx_c2r_x(Fields src, RFields dst, RFields dst2, const GridDev& g, int nrows, int nf,
                         const longlong2* tw_n, const longlong2* tw_nx, cudaStream_t s) {
    switch (g.nxh) {
#define X_CASE(n) \
    case n: launch_c2r_fx<n>(src, dst, dst2, g, nrows, nf, tw_n, tw_nx, s); break;
        DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t fft_fx_r2c_x(RFields src, Fields dst, const GridDev& g, int nrows, int nf, const longlong2* tw_n,
                         const longlong2* tw_nx, bool host_src, cudaStream_t s) {
    switch (g.nxh) {
#define X_CASE(n) \
    case n: launch_r2c_fx<n>(src, dst, g, nrows, nf, tw_n, tw_nx, host_src, s); break;
        DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template cudaError_t fft_fx_y<-1>(Fields, Fields, const GridDev&, int, int, int, const longlong2*, cudaStream_t);
template cudaError_t fft_fx_y<+1>(Fields, Fields, const GridDev&, int, int, int, const longlong2*, cudaStream_t);

template cudaError_t fft_ct_y<-1, double2>(Fields, Fields, const GridDev&, int, int, int, const double2*,
                                         cudaStream_t);
template cudaError_t fft_ct_y<+1, double2>(Fields, Fields, const GridDev&, int, int, int, const double2*,
                                         cudaStream_t);
template cudaError_t fft_ct_y<-1, float2>(FFields, FFields, const GridDev&, int, int, int, const float2*,
                                         cudaStream_t);
template cudaError_t fft_ct_y<+1, float2>(FFields, FFields, const GridDev&, int, int, int, const float2*,
                                         cudaStream_t);

}  // namespace dns3d
