// The transforms of the nonlinear term u x omega (compute_source_terms_3d,
// DNS_pressure_BC_3D.f90:1032-1098), from the spectra of u, v, w, ox, oy, oz to
// the source spectra: inverse y pass, then ONE x kernel that takes the rows of
// all six fields to physical space, forms the products there and takes the
// three results back (c2r, u x omega, r2c), then the forward y pass.  The
// physical fields never leave the SM.
//
// FP64 runs work in 64-bit block fixed point throughout (fft_dev.cuh) and pass
// the integers themselves between the passes, with one power of two per y
// column (inverse) or per x row (forward): the conversions between FP64 and
// the integers, about a third of the instructions of an FP64-in, FP64-out
// pass, are left only at the outer ends.  Each point's products are formed in
// integers in place of FP64 arithmetic: each of the two is rounded at 2^-60 of
// the product of its row maxima, the one of the smaller scale once more where
// they are aligned, and the forward transform takes their difference rounded
// to B = 51 to 53 bits of the row's largest (fx_bits).  Accuracy is relative to
// the row: a point whose product is far below the row's largest keeps fewer bits
// than in FP64 arithmetic, as it does in the transforms on both sides of it.
// Source terms against extended precision, 40 random fields on ten grids from
// 32 x 16 to 512 x 128 points per plane, white and smooth: rms error 9.2e-16 of the rms
// value in the geometric mean (separate kernels with FP64 products: 9.8e-16),
// not larger on any.  The mixed form runs the same kernel in FP32.
//
// The x kernel: one warp per field, the warp's 32 lanes hold 32 / (N/8)
// transforms of length N = nx/2 with 8 elements each, so every pass of the
// transform is synchronised by the warp alone; two CTA barriers (before and
// after the products).  At 128x128x65 the FP64 chain c2r, products, r2c took
// 100 + 18 + 43 us (six fields in, three out) and 78 us as one kernel, the
// FP32 one 17.6 + 9.1 + 13.4 us and 18 us.
#include "fft_dev.cuh"
#include "ragged.cuh"

namespace dns3d {

namespace {

// ------------------------------------------------------------------ keys and scales
// A fixed-point value X with exponent e stands for X 2^e.  The key of a
// complex value orders by the bit length of its larger component: 0 for zero,
// else bits + e + kKeyOff with |re|, |im| <= 2^bits.  Exponents from kNanExp on
// mark a transform whose FP64 input held a non-finite value: its outputs are
// non-finite throughout.
constexpr int kKeyOff = 1 << 16;
constexpr int kNanExp = 1 << 20;

__device__ __forceinline__ unsigned fx_key(fx2 x, int e) {
    const unsigned long long v =
        (unsigned long long)((x.x ^ (x.x >> 63)) | (x.y ^ (x.y >> 63)));
    return v ? (unsigned)(64 - __clzll((long long)v) + e + kKeyOff) : 0u;
}

// ------------------------------------------------------------------ y passes
// Columns per CTA and padded transform stride (16-byte slots: one padding slot
// after every 8, so that the passes' stores at stride 8 fall in distinct banks).
template <int N> __host__ __device__ constexpr int yfx_ld() { return N + N / 8 + 1 - ((N + N / 8) & 1); }
template <int N, int CX = per_cta(N)> __host__ __device__ constexpr int yfx_elems() { return CX * yfx_ld<N>(); }
// Columns per CTA where per_cta(N) of them leave SMs without a CTA: a quarter,
// or half, as long as rows split evenly over the threads and a row of the tile
// is 128 bytes.
__host__ __device__ constexpr int per_cta_small(int n) {
    for (int c = per_cta(n) / 4; c < per_cta(n); c *= 2)
        if (c >= 8 && n % (kThreads / c) == 0) return c;
    return per_cta(n);
}

// CTAs per SM the register limit leaves room for: at 4 (64 registers) the long
// passes hide their loads better (512x384x129: the three passes 1914 -> 1820 us,
// 96x192x81 126 -> 120), the short ones lose more to the tighter limit
// (64x48x40 33.5 -> 38).  Lengths 256 and 512 spill 44 to 84 bytes at 64
// registers and are still not slower (three passes, us, 3 and 4 CTAs: 64x256x65
// 89.9 and 89.9, 128x256x65 149.5 and 145.5, 64x512x33 98.4 and 99.0, 128x512x65
// 286.5 and 283.3).
__host__ __device__ constexpr int y_min_ctas(int n) { return n > 128 ? 4 : 3; }

// Inverse y pass, FP64 spectra to integers: dst[f] holds X, ecol[column] its
// exponent (column = plane * nxhp + kx).
template <int N, int CX = per_cta(N)>
__device__ __forceinline__ void y_inv_body(const double2* __restrict__ s, fx2* __restrict__ d, int* __restrict__ ecol,
                                           const GridDev& g, int nplanes, const fx2* __restrict__ tw, int bx,
                                           fx2* buf, unsigned* emax) {
    constexpr int LD = yfx_ld<N>(), B = fx_bits(N, 0);
    const long long ncols = (long long)nplanes * g.nxhp;
    const int c = threadIdx.x % CX, y0 = threadIdx.x / CX;
    const long long vc = (long long)bx * CX + c;
    const bool live = vc < ncols;
    size_t base = 0;
    if (live) {
        const int p = (int)(vc / g.nxhp);
        base = (size_t)p * g.nm + (int)(vc - (long long)p * g.nxhp);
    }
    constexpr int RPI = kThreads / CX, ITERS = N / RPI;
    static_assert(N % RPI == 0, "rows split evenly over the threads");
    if (threadIdx.x < CX) emax[threadIdx.x] = 1u;
    double2 v[ITERS];
    unsigned e = 1u;
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        v[it] = live ? s[base + (size_t)(y0 + it * RPI) * g.nxhp] : make_double2(0.0, 0.0);
        e = max(e, fx_expo(v[it]));
    }
    __syncthreads();
    fx_key_max(emax, c, e);
    __syncthreads();
    const int em = (int)emax[c];
    const int rsb = 53 - B + em;
#pragma unroll
    for (int it = 0; it < ITERS; ++it)
        buf[c * LD + swp<3>(y0 + it * RPI)] = mk<fx2>(fx_from(v[it].x, rsb), fx_from(v[it].y, rsb));
    __syncthreads();
    ct_fft_pad<N, 1, +1, CX, LD, 3>(buf, tw);
    if (live) {
        const bool bad = em == 0x7FF;
        if (y0 == 0) ecol[vc] = bad ? kNanExp : em - 1022 - B;
#pragma unroll
        for (int it = 0; it < ITERS; ++it) {
            const fx2 z = buf[c * LD + swp<3>(y0 + it * RPI)];
            d[base + (size_t)(y0 + it * RPI) * g.nxhp] = bad ? mk<fx2>(1, 1) : z;  // nonzero: its key carries the mark
        }
    }
}

// Forward y pass in place, integers (row exponents erow[plane * ny + y]) to
// FP64 spectra, columns kx < ncol, times nl.m 2^(nl.e) = 1/(nx ny)^2 (the two
// factors of a product of inverse transforms).
template <int N, int CX = per_cta(N)>
__device__ __forceinline__ void y_fwd_body(fx2* __restrict__ sd, const int* __restrict__ erow, const GridDev& g,
                                           int nplanes, int ncol, const NlScale& nl, const fx2* __restrict__ tw,
                                           int bx, fx2* buf, unsigned* emax) {
    constexpr int LD = yfx_ld<N>(), B = fx_bits(N, 0);
    const long long ncols = (long long)nplanes * ncol;
    const int c = threadIdx.x % CX, y0 = threadIdx.x / CX;
    const long long vc = (long long)bx * CX + c;
    const bool live = vc < ncols;
    size_t base = 0;
    const int* er = erow;
    if (live) {
        const int p = (int)(vc / ncol);
        base = (size_t)p * g.nm + (int)(vc - (long long)p * ncol);
        er = erow + (size_t)p * N;
    }
    constexpr int RPI = kThreads / CX, ITERS = N / RPI;
    if (threadIdx.x < CX) emax[threadIdx.x] = 0u;
    fx2 v[ITERS];
    int ev[ITERS];
    unsigned key = 0u;
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        v[it] = live ? sd[base + (size_t)(y0 + it * RPI) * g.nxhp] : mk<fx2>(0, 0);
        ev[it] = live ? __ldg(&er[y0 + it * RPI]) : 0;
    }
#pragma unroll
    for (int it = 0; it < ITERS; ++it) key = max(key, fx_key(v[it], ev[it]));
    __syncthreads();
    fx_key_max(emax, c, key);
    __syncthreads();
    const unsigned km = emax[c];
    const int E = (int)km - kKeyOff;
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int sh = E - B - ev[it];
        buf[c * LD + swp<3>(y0 + it * RPI)] = mk<fx2>(fx_rshift(v[it].x, sh), fx_rshift(v[it].y, sh));
    }
    __syncthreads();
    ct_fft_pad<N, 1, -1, CX, LD, 3>(buf, tw);
    if (live) {
        double2* d = reinterpret_cast<double2*>(sd);
        const FxLimbs m = fx_packed(nl.m);
        const int e2 = E - B + nl.e;
#pragma unroll
        for (int it = 0; it < ITERS; ++it) {
            fx2 z = buf[c * LD + swp<3>(y0 + it * RPI)];
            if (!nl.pow2) z = mk<fx2>(fx_mulq(z.x, m), fx_mulq(z.y, m));
            d[base + (size_t)(y0 + it * RPI) * g.nxhp] =
                km >= (unsigned)kNanExp ? make_double2(fx_nan(), fx_nan()) : make_double2(fx_to(z.x, e2), fx_to(z.y, e2));
        }
    }
}

template <int N, int CX>
__global__ void __launch_bounds__(kThreads, y_min_ctas(N)) k_nl_y_inv(Fields src, Fields dst, int* ecol, GridDev g, int nplanes,
                                                          const fx2* __restrict__ tw) {
    __shared__ fx2 buf[yfx_elems<N, CX>()];
    __shared__ unsigned emax[CX];
    y_inv_body<N, CX>(field_ptr(src, blockIdx.z), reinterpret_cast<fx2*>(field_ptr(dst, blockIdx.z)),
                  ecol + (size_t)blockIdx.z * nplanes * g.nxhp, g, nplanes, tw, blockIdx.x, buf, emax);
}

template <int N, int CX>
__global__ void __launch_bounds__(kThreads, y_min_ctas(N)) k_nl_y_fwd(Fields srcdst, const int* erow, GridDev g, int nplanes,
                                                          int ncol, NlScale nl, const fx2* __restrict__ tw) {
    __shared__ fx2 buf[yfx_elems<N, CX>()];
    __shared__ unsigned emax[CX];
    y_fwd_body<N, CX>(reinterpret_cast<fx2*>(field_ptr(srcdst, blockIdx.z)), erow + (size_t)blockIdx.z * nplanes * N, g,
                  nplanes, ncol, nl, tw, blockIdx.x, buf, emax);
}

// ------------------------------------------------------------------ the x kernel
constexpr int kXThreads = 192;  // one warp per field

// Lanes per transform, transforms (rows) per warp and the padded row stride.
template <int N> __host__ __device__ constexpr int x_lanes() { return N / 8; }
template <int N> __host__ __device__ constexpr int x_rows() { return 32 / x_lanes<N>(); }
template <int N, int PAD> __host__ __device__ constexpr int x_ld() { return N + (N >> PAD); }
template <int N, int PAD> __host__ __device__ constexpr int x_elems() { return 6 * x_rows<N>() * x_ld<N, PAD>(); }

struct NoHook {
    template <typename C> __device__ __forceinline__ void operator()(C*, int) const {}
};

// One Stockham pass of the warp's rows, in place: `pre` on the inputs of each
// butterfly, `post` on the outputs before they are written.  The last pass
// writes each butterfly's outputs where its inputs were, so a lane finishes
// one butterfly before the next (radix 3, whose N/3 butterflies do not divide
// over N/8 lanes, holds 3 values at a time instead of 9); the others hold a
// lane's outputs until every input is read.
template <int N, int R, int NS, int SIGN, int PAD, typename C, typename Pre, typename Post>
__device__ __forceinline__ void warp_pass(C* buf, const C* __restrict__ tw, const Pre& pre, const Post& post) {
    constexpr int L = x_lanes<N>(), NB = N / R, PER = (NB + L - 1) / L, TSTEP = N / (NS * R);
    constexpr bool kLast = NS * R == N;
    static_assert(kLast || NB % L == 0, "only the last pass may leave lanes without a butterfly");
    const int lane = threadIdx.x & 31, c = lane / L, j0 = lane - c * L;
    const bool on = (32 % L == 0) || c < x_rows<N>();
    C* row = buf + (on ? c : 0) * x_ld<N, PAD>();  // lanes without a row compute one and drop it
    auto load = [&](C* v, int j) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = row[swp<PAD>(j + r * NB)];
        pre(v, R);
        if constexpr (NS > 1) {
            const int k = j % NS;
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = tw_mul<SIGN>(v[r], __ldg(&tw[r * k * TSTEP]));
        }
        dft<R, SIGN>(v);
    };
    if constexpr (kLast) {
        if (on) {
#pragma unroll(R == 3 ? 1 : PER)
            for (int p = 0; p < PER; ++p) {
                const int j = j0 + p * L;
                if (NB % L == 0 || j < NB) {
                    C v[R];
                    load(v, j);
                    post(v, R);
#pragma unroll
                    for (int q = 0; q < R; ++q) row[swp<PAD>(j + q * NB)] = v[q];
                }
            }
        }
    } else {
        C v[PER][R];
#pragma unroll
        for (int p = 0; p < PER; ++p) load(v[p], j0 + p * L);
        __syncwarp();
        if (on) {
#pragma unroll
            for (int p = 0; p < PER; ++p) {
                const int j = j0 + p * L;
                const int o = (j / NS) * NS * R + j % NS;
#pragma unroll
                for (int q = 0; q < R; ++q) row[swp<PAD>(o + q * NS)] = v[p][q];
            }
        }
    }
    __syncwarp();
}

// All passes: `pre` in the first, `post` in the last.
template <int N, int NS, int SIGN, int PAD, typename C, typename Pre, typename Post>
__device__ __forceinline__ void warp_fft(C* buf, const C* __restrict__ tw, const Pre& pre, const Post& post) {
    constexpr int R = next_radix(N / NS);
    if constexpr (NS * R == N) {
        warp_pass<N, R, NS, SIGN, PAD>(buf, tw, pre, post);
    } else {
        warp_pass<N, R, NS, SIGN, PAD>(buf, tw, pre, NoHook{});
        warp_fft<N, NS * R, SIGN, PAD>(buf, tw, NoHook{}, post);
    }
}

// The OR of v over the L lanes of this lane's transform.
template <int L> __device__ __forceinline__ unsigned row_or(unsigned v) {
    if constexpr ((L & (L - 1)) == 0) {
#pragma unroll
        for (int o = 1; o < L; o <<= 1) v |= __shfl_xor_sync(0xFFFFFFFFu, v, o);
        return v;
    } else {
        const int c = (int)(threadIdx.x & 31) / L;
        return __reduce_or_sync(c < 32 / L ? ((1u << L) - 1u) << (c * L) : 0xFFFFFFFFu << (32 / L * L), v);
    }
}

// Last pass: the OR of the outputs' high magnitude words.
struct RowBits {
    unsigned* bits;
    __device__ __forceinline__ void operator()(const fx2* v, int n) const {
#pragma unroll
        for (int r = 0; r < n; ++r)
            *bits |= (unsigned)((v[r].x ^ (v[r].x >> 63)) >> 32) | (unsigned)((v[r].y ^ (v[r].y >> 63)) >> 32);
    }
};

// First pass: a shift of the inputs (0: none).
struct ShiftIn {
    int sh;
    __device__ __forceinline__ void operator()(fx2* v, int n) const {
        if (sh) {
#pragma unroll
            for (int r = 0; r < n; ++r) v[r] = mk<fx2>(fx_rshift(v[r].x, sh), fx_rshift(v[r].y, sh));
        }
    }
};

// keys[r] = max(keys[r], key) over the warp's lanes (r uniform when the items
// of one iteration belong to one row)
template <int ITEMS> __device__ __forceinline__ void row_key_max(unsigned* keys, int r, unsigned key) {
    if constexpr (ITEMS % 32 == 0) {
        key = __reduce_max_sync(0xFFFFFFFFu, key);
        if ((threadIdx.x & 31) == 0) atomicMax(&keys[r], key);
    } else {
        fx_key_max(keys, r, key);
    }
}

struct XShared {
    int e[6 * 16];         // exponents of the physical rows [field][row], and the left
    int s[6 * 16];         // shift that gives their largest component 62 bits
    unsigned key[6 * 16];  // row maxima: inputs, then products [field][row]
    int bad[3 * 16];       // products: some input row held a non-finite value
};

// Rows row0 .. row0 + x_rows(N) - 1 of the six fields: src[f] integer rows of
// nx/2 + 1 values with column exponents ecol[f * ecs + plane * (N+1) + kx];
// dst[f] the three products' integer spectra, columns kx < ncol, with row
// exponents erow[f * nrows + row].  The packing of a real row of 2N points into
// N complex ones pairs k with N - k: with S = X[k] + conj X[N-k],
// D = X[k] - conj X[N-k], P = e^{2 pi i k / nx} D it is Z[k] = S + i P,
// Z[N-k] = conj(S) + i conj(P): one complex product per pair; likewise back.
template <int N>
__device__ __forceinline__ void x_body_fx(const Fields& src, const int* __restrict__ ecol, size_t ecs,
                                          const Fields& dst, int* __restrict__ erow, const GridDev& g, int nrows,
                                          int ncol, const fx2* __restrict__ tw_n, const fx2* __restrict__ tw_nx,
                                          int bx, fx2* buf, XShared& sh) {
    constexpr int TW = x_rows<N>(), LD = x_ld<N, 3>(), B = fx_bits(N, 2), H = N / 2;
    constexpr int NP = TW * H, ITS = (NP + 31) / 32, L = x_lanes<N>();
    const int f = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = bx * TW;
    fx2* bf = buf + f * TW * LD;
    unsigned* key = sh.key + f * 16;
    if (lane < 16) key[lane] = 0u;
    __syncwarp();
    {
        // the rows' inputs as they are into the slots of Z (k and N - k of a pair;
        // Im of kx = 0 and kx = nx/2 is ignored, so slot 0 holds (X[0], X[N])),
        // and the largest key of each row
        const fx2* __restrict__ s = reinterpret_cast<const fx2*>(field_ptr(src, f));
        const int* __restrict__ ec = ecol + (size_t)f * ecs;
        fx2 a[ITS], b[ITS];
        int ea[ITS], eb[ITS];
#pragma unroll
        for (int it = 0; it < ITS; ++it) {
            const int t = lane + 32 * it;
            const int r = t / H, k = t - r * H, row = row0 + r;
            a[it] = b[it] = mk<fx2>(0, 0);
            ea[it] = eb[it] = 0;
            if ((NP % 32 == 0 || t < NP) && row < nrows) {
                const fx2* p = s + (size_t)row * (N + 1);
                const int* q = ec + (size_t)(row / g.ny) * (N + 1);
                a[it] = p[k];
                b[it] = p[N - k];
                ea[it] = __ldg(&q[k]);
                eb[it] = __ldg(&q[N - k]);
                if (k == 0) a[it].y = b[it].y = 0;
            }
        }
        if (lane < TW) {  // k = N/2
            fx2 mid = mk<fx2>(0, 0);
            if (row0 + lane < nrows) {
                mid = s[(size_t)(row0 + lane) * (N + 1) + H];
                atomicMax(&key[lane], fx_key(mid, __ldg(&ec[(size_t)((row0 + lane) / g.ny) * (N + 1) + H])));
            }
            bf[lane * LD + swp<3>(H)] = mid;
        }
#pragma unroll
        for (int it = 0; it < ITS; ++it) {
            const int t = lane + 32 * it;
            const int r = min(t / H, TW - 1), k = t % H;
            row_key_max<H>(key, r, max(fx_key(a[it], ea[it]), fx_key(b[it], eb[it])));
            if (NP % 32 == 0 || t < NP) {
                bf[r * LD + swp<3>(k)] = k ? a[it] : mk<fx2>(a[it].x, b[it].x);
                if (k) bf[r * LD + swp<3>(N - k)] = b[it];
            }
        }
        __syncwarp();
        // scaled to B bits and packed, pair by pair in place (not unrolled: the
        // kernel's code must stay small for the instruction caches)
#pragma unroll 1
        for (int t = lane; t < NP; t += 32) {
            const int r = t / H, k = t - r * H, row = min(row0 + r, nrows - 1);
            const int* q = ec + (size_t)(row / g.ny) * (N + 1);
            const int base = (int)key[r] - kKeyOff - B;
            const int sa = base - __ldg(&q[k]), sb = base - __ldg(&q[N - k]);
            fx2* za = bf + r * LD + swp<3>(k);
            fx2* zb = bf + r * LD + swp<3>(k ? N - k : H);
            fx2 x = *za, y = *zb;
            if (k == 0) {
                const int sm = base - __ldg(&q[H]);  // Z[N/2] = 2 conj X[N/2]
                *zb = mk<fx2>(2 * fx_rshift(y.x, sm), -2 * fx_rshift(y.y, sm));
                y = mk<fx2>(x.y, 0);
                x.y = 0;
            }
            x = mk<fx2>(fx_rshift(x.x, sa), fx_rshift(x.y, sa));
            y = mk<fx2>(fx_rshift(y.x, sb), fx_rshift(y.y, sb));
            const fx2 sm = mk<fx2>(x.x + y.x, x.y - y.y), df = mk<fx2>(x.x - y.x, x.y + y.y);
            const fx2 p = tw_mul<+1>(df, __ldg(&tw_nx[k]));
            *za = mk<fx2>(sm.x - p.y, sm.y + p.x);
            if (k) *zb = mk<fx2>(sm.x + p.y, p.x - sm.y);
        }
        __syncwarp();
    }
    // Inverse transform, products, forward transform: both transforms run the
    // one copy of the inverse passes' code, the forward one on values with re
    // and im exchanged (F(z) = swap I(swap z)).
#pragma unroll 1
    for (int fwd = 0;; ++fwd) {
        const int c = lane / L, cc = min(c, TW - 1);
        unsigned bits = 0u;
        warp_fft<N, 1, +1, 3>(bf, tw_n, ShiftIn{fwd ? (int)key[cc] - B : 0}, RowBits{&bits});
        if (fwd) break;
        bits = row_or<L>(bits);
        if (lane == c * L && c < TW) {
            // below 2^32 only rows that are all but zero (a transform's largest
            // output is at least its largest input, 2^(B-1) or zero): 32 bits bound them
            const int s = 62 - (bits ? 64 - __clz(bits) : 32);
            const unsigned km = key[c];
            sh.s[f * 16 + c] = s;
            sh.e[f * 16 + c] = km >= (unsigned)kNanExp ? kNanExp : (int)km - kKeyOff - B - s;
        }
        __syncwarp();
        if (lane < 16) key[lane] = 0u;
        __syncthreads();
        // u x omega (3D:1085-1095), one point per item, in place over u, v, w with
        // the points of a slot exchanged
        long long* pt = reinterpret_cast<long long*>(buf);
#pragma unroll 1
        for (int t0 = f * 32; t0 < 2 * TW * N; t0 += kXThreads) {
            const int t = t0 + lane;
            const bool on = (TW * N) % 16 == 0 || t < 2 * TW * N;
            const int r = on ? t / (2 * N) : TW - 1;
            const int o = 2 * (r * LD + swp<3>((t >> 1) - r * N)), half = t & 1;
            FxLimbs x[6];
            int e[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                x[i] = fx_split(on ? pt[2 * i * TW * LD + o + half] << sh.s[i * 16 + r] : 0);
                e[i] = sh.e[i * 16 + r];
            }
            __syncwarp();  // the pair of points of a slot is read before either is written
#pragma unroll
            for (int q = 0; q < 3; ++q) {  // component q: (q+1) (3 + q+2) - (q+2) (3 + q+1)
                const int q1 = (q + 1) % 3, q2 = (q + 2) % 3;
                const int p1 = e[q1] + e[3 + q2], p2 = e[q2] + e[3 + q1], es = max(p1, p2);
                const long long v = fx_rshift(fx_prod(x[q1], x[3 + q2]), es - p1) -
                                    fx_rshift(fx_prod(x[q2], x[3 + q1]), es - p2);
                if (on) pt[2 * q * TW * LD + o + 1 - half] = v;
                const unsigned long long mag = (unsigned long long)(v ^ (v >> 63));
                row_key_max<2 * N>(sh.key + q * 16, r, mag ? 64u - (unsigned)__clzll((long long)mag) : 0u);
            }
        }
        __syncthreads();
        if (f >= 3) return;
    }
    if (lane < TW) {
        int m = sh.e[lane];
        for (int i = 1; i < 6; ++i) m = max(m, sh.e[i * 16 + lane]);
        sh.bad[f * 16 + lane] = m >= kNanExp;
        if (row0 + lane < nrows) {
            const int q1 = (f + 1) % 3, q2 = (f + 2) % 3;
            const int es = max(sh.e[q1 * 16 + lane] + sh.e[(3 + q2) * 16 + lane],
                               sh.e[q2 * 16 + lane] + sh.e[(3 + q1) * 16 + lane]);
            // the products' 2^64, the shift to B bits, the 1/2 of the unpacking
            erow[(size_t)f * nrows + row0 + lane] = m >= kNanExp ? kNanExp : es + 64 + (int)key[lane] - B - 1;
        }
    }
    __syncwarp();
    // 2 X[k] = E + P, 2 X[N-k] = conj(E) - conj(P) with E = Z[k] + conj Z[N-k],
    // P = e^{-2 pi i k / nx} (-i) (Z[k] - conj Z[N-k]); 2 X[N/2] = 2 conj Z[N/2]
    fx2* __restrict__ d = reinterpret_cast<fx2*>(field_ptr(dst, f));
#pragma unroll 1
    for (int t = lane; t < NP; t += 32) {
        const int r = t / H, k = t - r * H, row = row0 + r;
        if (row >= nrows) break;  // rows ascend with t
        const fx2 a = bf[r * LD + swp<3>(k)], b = bf[r * LD + swp<3>(k ? N - k : 0)];  // re, im exchanged
        const fx2 e = mk<fx2>(a.y + b.y, a.x - b.x), o = mk<fx2>(a.x + b.x, b.y - a.y);
        const fx2 p = tw_mul<-1>(o, __ldg(&tw_nx[k]));
        const bool bad = sh.bad[f * 16 + r] != 0;  // nonzero values: their keys carry the mark
        fx2* out = d + (size_t)row * (N + 1);
        if (k < ncol) out[k] = bad ? mk<fx2>(1, 1) : mk<fx2>(e.x + p.x, e.y + p.y);
        if (N - k < ncol) out[N - k] = bad ? mk<fx2>(1, 1) : mk<fx2>(e.x - p.x, p.y - e.y);
        if (k == 0 && H < ncol) {
            const fx2 z = bf[r * LD + swp<3>(H)];
            out[H] = bad ? mk<fx2>(1, 1) : mk<fx2>(2 * z.y, -2 * z.x);
        }
    }
}

template <int N>
__global__ void __launch_bounds__(kXThreads, 4) k_nl_x(Fields src, const int* ecol, size_t ecs, Fields dst, int* erow,
                                                       GridDev g, int nrows, int ncol, const fx2* __restrict__ tw_n,
                                                       const fx2* __restrict__ tw_nx) {
    __shared__ fx2 buf[x_elems<N, 3>()];
    __shared__ XShared sh;
    x_body_fx<N>(src, ecol, ecs, dst, erow, g, nrows, ncol, tw_n, tw_nx, blockIdx.x, buf, sh);
}

// The same in FP32 (the mixed form), the products in FP32 arithmetic.
template <int N>
__device__ __forceinline__ void x_body_32(const FFields& src, const FFields& dst, const GridDev& g, int nrows,
                                          int ncol, const float2* __restrict__ tw_n,
                                          const float2* __restrict__ tw_nx, int bx, float2* buf) {
    using C = float2;
    constexpr int TW = x_rows<N>(), LD = x_ld<N, 4>(), H = N / 2, NP = TW * H, ITS = (NP + 31) / 32;
    const int f = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = bx * TW;
    C* bf = buf + f * TW * LD;
    {
        const C* __restrict__ s = field_ptr(src, f);
        C a[ITS], b[ITS];
#pragma unroll
        for (int it = 0; it < ITS; ++it) {
            const int t = lane + 32 * it;
            const int r = t / H, k = t - r * H, row = row0 + r;
            a[it] = b[it] = mk<C>(0, 0);
            if ((NP % 32 == 0 || t < NP) && row < nrows) {
                const C* p = s + (size_t)row * (N + 1);
                a[it] = p[k];
                b[it] = p[N - k];
                if (k == 0) a[it].y = b[it].y = 0;
            }
        }
        C mid = mk<C>(0, 0);
        if (lane < TW && row0 + lane < nrows) mid = s[(size_t)(row0 + lane) * (N + 1) + H];
#pragma unroll
        for (int it = 0; it < ITS; ++it) {
            const int t = lane + 32 * it;
            const int r = t / H, k = t - r * H;
            if (NP % 32 == 0 || t < NP) {
                const C sm = mk<C>(a[it].x + b[it].x, a[it].y - b[it].y);
                const C df = mk<C>(a[it].x - b[it].x, a[it].y + b[it].y);
                C w = __ldg(&tw_nx[k]);
                w.y = -w.y;
                const C p = cmul(w, df);
                bf[r * LD + swp<4>(k)] = mk<C>(sm.x - p.y, sm.y + p.x);
                if (k) bf[r * LD + swp<4>(N - k)] = mk<C>(sm.x + p.y, p.x - sm.y);
            }
        }
        if (lane < TW) bf[lane * LD + swp<4>(H)] = mk<C>(2.0f * mid.x, -2.0f * mid.y);
        __syncwarp();
    }
    warp_fft<N, 1, +1, 4>(bf, tw_n, NoHook{}, NoHook{});
    __syncthreads();
    const float sc = (float)g.inv_nxny;
    for (int t = threadIdx.x; t < TW * N; t += kXThreads) {
        const int r = t / N, o = r * LD + swp<4>(t - r * N);
        C w[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const C z = buf[i * TW * LD + o];
            w[i] = mk<C>(z.x * sc, z.y * sc);
        }
        buf[o] = mk<C>(w[1].x * w[5].x - w[2].x * w[4].x, w[1].y * w[5].y - w[2].y * w[4].y);
        buf[TW * LD + o] = mk<C>(w[2].x * w[3].x - w[0].x * w[5].x, w[2].y * w[3].y - w[0].y * w[5].y);
        buf[2 * TW * LD + o] = mk<C>(w[0].x * w[4].x - w[1].x * w[3].x, w[0].y * w[4].y - w[1].y * w[3].y);
    }
    __syncthreads();
    if (f >= 3) return;
    warp_fft<N, 1, -1, 4>(bf, tw_n, NoHook{}, NoHook{});
    C* __restrict__ d = field_ptr(dst, f);
#pragma unroll
    for (int it = 0; it < ITS; ++it) {
        const int t = lane + 32 * it;
        const int r = t / H, k = t - r * H, row = row0 + r;
        if ((NP % 32 == 0 || t < NP) && row < nrows) {
            const C za = bf[r * LD + swp<4>(k)], zb = bf[r * LD + swp<4>(k ? N - k : 0)];
            const C e = mk<C>(0.5f * (za.x + zb.x), 0.5f * (za.y - zb.y));
            const C o = mk<C>(0.5f * (za.y + zb.y), -0.5f * (za.x - zb.x));
            const C p = cmul(__ldg(&tw_nx[k]), o);
            C* out = d + (size_t)row * (N + 1);
            if (k < ncol) out[k] = mk<C>(e.x + p.x, e.y + p.y);
            if (N - k < ncol) out[N - k] = mk<C>(e.x - p.x, p.y - e.y);
        }
    }
    if (H < ncol && lane < TW && row0 + lane < nrows) {
        const C z = bf[lane * LD + swp<4>(H)];
        d[(size_t)(row0 + lane) * (N + 1) + H] = mk<C>(z.x, -z.y);
    }
}

template <int N>
__global__ void __launch_bounds__(kXThreads, N > 128 ? 5 : 6) k_nl_x32(FFields src, FFields dst, GridDev g, int nrows, int ncol,
                                                         const float2* __restrict__ tw_n,
                                                         const float2* __restrict__ tw_nx) {
    __shared__ float2 buf[x_elems<N, 4>()];
    x_body_32<N>(src, dst, g, nrows, ncol, tw_n, tw_nx, blockIdx.x, buf);
}

// ------------------------------------------------------------------ ragged stages
// The same bodies over many runs in one launch (k_stage, ragged.cuh).
__host__ __device__ constexpr int yfx_elems_max() {
    int m = 0;
#define ELEMS_MAX(n) m = yfx_elems<n>() > m ? yfx_elems<n>() : m;
    DNS3D_CT_Y_LENGTHS(ELEMS_MAX)
#undef ELEMS_MAX
    return m;
}
template <int PAD> __host__ __device__ constexpr int x_elems_max() {
    int m = 0;
#define ELEMS_MAX(n) m = x_elems<n, PAD>() > m ? x_elems<n, PAD>() : m;
    DNS3D_CT_X_LENGTHS(ELEMS_MAX)
#undef ELEMS_MAX
    return m;
}

// Fields of a descriptor pointer list.
template <typename P, int K>
__device__ __forceinline__ FieldsT<P> list_fields(void* const* p) {
    FieldsT<P> r;
#pragma unroll
    for (int i = 0; i < kMaxFields; ++i) r.p[i] = i < K ? static_cast<P*>(p[i < K ? i : 0]) : nullptr;
    return r;
}

// F0 = 0: u, v, w; 3: the vorticity
template <int F0>
struct RsNlYInv {
    static constexpr int kMinCtas = 3;
    static __device__ __forceinline__ void run(const RunDesc& d, int b) {
        __shared__ fx2 buf[yfx_elems_max()];
        __shared__ unsigned emax[64];
        const int gx = d.gx[kRsFftYInv], f3 = b / gx, f = F0 + f3, bx = b - f3 * gx;
        const double2* s = static_cast<const double2*>(d.spec[f]);
        fx2* o = static_cast<fx2*>(d.tmp[f]);
        int* ec = d.ecol + (size_t)f * d.g.nz * d.g.nxhp;
        const fx2* tw = static_cast<const fx2*>(d.tw_ny);
        switch (d.g.ny) {
#define Y_CASE(n) \
    case n: y_inv_body<n>(s, o, ec, d.g, d.g.nz, tw, bx, buf, emax); break;
            DNS3D_CT_Y_LENGTHS(Y_CASE)
#undef Y_CASE
        }
    }
};

struct RsNlYFwd {
    static constexpr int kMinCtas = 3;
    static __device__ __forceinline__ void run(const RunDesc& d, int b) {
        __shared__ fx2 buf[yfx_elems_max()];
        __shared__ unsigned emax[64];
        const int gx = d.gx[kRsFftYFwd], f = b / gx, bx = b - f * gx;
        fx2* o = static_cast<fx2*>(d.src[f]);
        const int* er = d.erow + (size_t)f * d.g.nz * d.g.ny;
        const fx2* tw = static_cast<const fx2*>(d.tw_ny);
        switch (d.g.ny) {
#define Y_CASE(n) \
    case n: y_fwd_body<n>(o, er, d.g, d.g.nz, d.ncol, d.nl, tw, bx, buf, emax); break;
            DNS3D_CT_Y_LENGTHS(Y_CASE)
#undef Y_CASE
        }
    }
};

struct RsNlX {
    static constexpr int kMinCtas = 3;
    static __device__ __forceinline__ void run(const RunDesc& d, int b) {
        __shared__ fx2 buf[x_elems_max<3>()];
        __shared__ XShared sh;
        const fx2* twn = static_cast<const fx2*>(d.tw_nx2);
        const fx2* twx = static_cast<const fx2*>(d.tw_nx);
        const Fields src = list_fields<double2, 6>(d.tmp), dst = list_fields<double2, 3>(d.src);
        switch (d.g.nxh) {
#define X_CASE(n)                                                                                                   \
    case n:                                                                                                         \
        x_body_fx<n>(src, d.ecol, (size_t)d.g.nz * d.g.nxhp, dst, d.erow, d.g, d.g.nz * d.g.ny, d.ncol, twn, twx, b, \
                     buf, sh);                                                                                      \
        break;
            DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        }
    }
};

struct RsNlX32 {
    static constexpr int kMinCtas = 4;
    static __device__ __forceinline__ void run(const RunDesc& d, int b) {
        __shared__ float2 buf[x_elems_max<4>()];
        const float2* twn = static_cast<const float2*>(d.tw_nx2);
        const float2* twx = static_cast<const float2*>(d.tw_nx);
        const FFields src = list_fields<float2, 6>(d.tmp), dst = list_fields<float2, 3>(d.src);
        switch (d.g.nxh) {
#define X_CASE(n) \
    case n: x_body_32<n>(src, dst, d.g, d.g.nz * d.g.ny, d.ncol, twn, twx, b, buf); break;
            DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        }
    }
};

}  // namespace

StageKernel ragged_nl_kernel(int stage, bool mixed) {
    switch (stage) {
        case kRsFftYUvw: return k_stage<RsNlYInv<0>>;
        case kRsFftYInv: return k_stage<RsNlYInv<3>>;
        case kRsFftX: return mixed ? k_stage<RsNlX32> : k_stage<RsNlX>;
        case kRsFftYFwd: return k_stage<RsNlYFwd>;
    }
    return nullptr;
}

int nl_x_threads() { return kXThreads; }

int nl_x_rows(int nxh) {
    switch (nxh) {
#define X_CASE(n) \
    case n: return x_rows<n>();
        DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
    }
    return 1;
}

// Columns per CTA of a y pass over nf fields of ncols columns of length n.  Below
// a CTA per SM the pass is as long as one CTA's chain (load, scale, transform,
// store of 8 or 6 values per thread), so tiles of a quarter of the columns end
// sooner.  us per step with full tiles and with this rule: 32x32x17 55.3 and
// 49.1, 32x32x33 64 and 57, 64x48x40 112 and 108; with more tiles than SMs
// there is nothing to gain.
static int y_columns(int n, long long ncols, int nf) {
    const int c = per_cta(n);
    return (ncols + c - 1) / c * nf < 152 ? per_cta_small(n) : c;
}

cudaError_t nl_y_inverse(const FftCtx& ctx, const GridDev& g, Fields spec, int nf, int slot0, cudaStream_t s) {
    if (!ctx.fx || slot0 < 0 || slot0 + nf > 6) return cudaErrorInvalidValue;
    Fields tmp{};
    for (int f = 0; f < nf; ++f) tmp.p[f] = ctx.tmp + (size_t)(slot0 + f) * g.nm * g.nz;
    const long long ncols = (long long)g.nz * g.nxhp;
    int* ecol = ctx.ecol + (size_t)slot0 * ncols;
    switch (g.ny) {
#define Y_CASE(n)                                                                          \
    case n: {                                                                              \
        const int cx = y_columns(n, ncols, nf);                                            \
        auto k = cx == per_cta(n) ? k_nl_y_inv<n, per_cta(n)> : k_nl_y_inv<n, per_cta_small(n)>; \
        k<<<dim3((unsigned)((ncols + cx - 1) / cx), 1, nf), kThreads, 0, s>>>(spec, tmp, ecol, g, g.nz, ctx.twq_ny); \
        break;                                                                             \
    }
        DNS3D_CT_Y_LENGTHS(Y_CASE)
#undef Y_CASE
        default: return cudaErrorInvalidValue;
    }
    const cudaError_t e = cudaGetLastError();
    if (!e && ctx.hook) ctx.hook(ctx.hook_ctx, "fft_y_inverse");
    return e;
}

cudaError_t nl_products(const FftCtx& ctx, const GridDev& g, Fields src, int ncol, cudaStream_t s) {
    if (!ctx.fx) return cudaErrorInvalidValue;
    Fields tmp{};
    for (int f = 0; f < 6; ++f) tmp.p[f] = ctx.tmp + (size_t)f * g.nm * g.nz;
    const int nrows = g.nz * g.ny;
    const size_t ncols = (size_t)g.nz * g.nxhp;
    if (ncol <= 0 || ncol > g.nxhp) ncol = g.nxhp;
    switch (g.nxh) {
#define X_CASE(n)                                                                                             \
    case n:                                                                                                   \
        k_nl_x<n><<<(nrows + x_rows<n>() - 1) / x_rows<n>(), kXThreads, 0, s>>>(tmp, ctx.ecol, ncols, src, ctx.erow, \
                                                                               g, nrows, ncol, ctx.twq_nx2, ctx.twq_nx); \
        break;
        DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        default: return cudaErrorInvalidValue;
    }
    cudaError_t e = cudaGetLastError();
    if (e) return e;
    if (ctx.hook) ctx.hook(ctx.hook_ctx, "fft_x_products");
    switch (g.ny) {
#define Y_CASE(n)                                                                                              \
    case n: {                                                                                                  \
        const long long nc = (long long)g.nz * ncol;                                                           \
        const int cx = y_columns(n, nc, 3);                                                                    \
        auto k = cx == per_cta(n) ? k_nl_y_fwd<n, per_cta(n)> : k_nl_y_fwd<n, per_cta_small(n)>;                     \
        k<<<dim3((unsigned)((nc + cx - 1) / cx), 1, 3), kThreads, 0, s>>>(src, ctx.erow, g, g.nz, ncol, ctx.nl,    \
                                                                        ctx.twq_ny);                             \
        break;                                                                                                 \
    }
        DNS3D_CT_Y_LENGTHS(Y_CASE)
#undef Y_CASE
        default: return cudaErrorInvalidValue;
    }
    e = cudaGetLastError();
    if (!e && ctx.hook) ctx.hook(ctx.hook_ctx, "fft_y_forward");
    return e;
}

cudaError_t nl_transforms32(const FftCtx& ctx, const GridDev& g, FFields spec, FFields src, int ncol,
                            cudaStream_t s) {
    if (!ctx.use_ct || !ctx.tmp32) return cudaErrorInvalidValue;
    FFields tmp{};
    for (int f = 0; f < 6; ++f) tmp.p[f] = ctx.tmp32 + (size_t)f * g.nm * g.nz;
    const int nrows = g.nz * g.ny;
    if (ncol <= 0 || ncol > g.nxhp) ncol = g.nxhp;
    cudaError_t e = fft_ct_y<+1, float2>(spec, tmp, g, g.nz, g.nxhp, 6, ctx.tw32_ny, s);
    if (e) return e;
    if (ctx.hook) ctx.hook(ctx.hook_ctx, "fft32_y_inverse");
    switch (g.nxh) {
#define X_CASE(n)                                                                                              \
    case n:                                                                                                    \
        k_nl_x32<n><<<(nrows + x_rows<n>() - 1) / x_rows<n>(), kXThreads, 0, s>>>(tmp, src, g, nrows, ncol,     \
                                                                                 ctx.tw32_nx2, ctx.tw32_nx);   \
        break;
        DNS3D_CT_X_LENGTHS(X_CASE)
#undef X_CASE
        default: return cudaErrorInvalidValue;
    }
    e = cudaGetLastError();
    if (e) return e;
    if (ctx.hook) ctx.hook(ctx.hook_ctx, "fft32_x_products");
    e = fft_ct_y<-1, float2>(src, src, g, g.nz, ncol, 3, ctx.tw32_ny, s);
    if (!e && ctx.hook) ctx.hook(ctx.hook_ctx, "fft32_y_forward");
    return e;
}

}  // namespace dns3d
