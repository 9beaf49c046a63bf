// aw_gridfft.cuh — grid solves as three kernels (included by aw_spectral.cu inside
// its anonymous namespace): the unfused solves on the caller's arrays and the
// adjoints' transposed solves.
//
//   k_rows_fwd   rows of real planes -> complex along x
//   k_cols       complex along y, the solve's multiplier in k-space, and back
//   k_rows_inv   complex -> real along x, into planes
//
// One library transform per caller array and direction took 20 launches a solve; on
// grids of this path (up to 1024 on a side, a few MB) the latency of dependent launches
// is the time, not the bytes or the arithmetic. Here a row or column lives in shared
// memory from its load to its last use (the unfused Darwin step at 256 x 256: 604 ->
// 477 us). The fused steps, whose planes are contiguous and batched, keep the library
// transforms: the gain there is 1 to 4%, and the FP32 rounding of E decides in which
// step a particle crosses a cell edge, which a gradient shows.
//
// Two rows share one complex transform (z = a + i b, a and b of one field, so their
// magnitudes are alike). Between the kernels a field is stored transposed, [k][j], so
// that the columns are contiguous and a block of PR row pairs reads and writes 16 PR
// bytes at a time. The transforms are Stockham passes of radix 8, 4, 2, 3, 5, 7 between
// two shared buffers, padded by one element in 16 so that a pass's strided writes spread
// over the banks. The passes of radix 3, 5 and 7 compute in double: all in single, the
// error of some sizes was above the library transforms' (720 x 96 by a tenth).

constexpr int kFftMax = 1024;          // longest row or column
struct FftPlan {
    int n, np;
    int r[12];
    int odd;                           // some radix is odd
    float rnb[12], rl[12];             // 1 / (n / r), 1 / (product of the radices before)
};
__device__ __forceinline__ int fpad(int i) { return i + (i >> 4); }
// Arithmetic of the passes: single precision for the radices 8, 4, 2, double for 3, 5, 7.
template <int R> struct PassOf { using T = float; using T2 = float2; };
template <> struct PassOf<3> { using T = double; using T2 = double2; };
template <> struct PassOf<5> : PassOf<3> {};
template <> struct PassOf<7> : PassOf<3> {};
__device__ __forceinline__ float2 mk(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 mk(double x, double y) { return make_double2(x, y); }
template <class T2> __device__ __forceinline__ T2 cmul(T2 a, T2 b) {
    return mk(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
template <class T2> __device__ __forceinline__ T2 cadd(T2 a, T2 b) { return mk(a.x + b.x, a.y + b.y); }
template <class T2> __device__ __forceinline__ T2 csub(T2 a, T2 b) { return mk(a.x - b.x, a.y - b.y); }
// a * (SIGN i)
template <int SIGN, class T2> __device__ __forceinline__ T2 cimul(T2 a) {
    return SIGN < 0 ? mk(a.y, -a.x) : mk(-a.y, a.x);
}

// In-register transforms of R values, kernel exp(SIGN 2 pi i p q / R).
template <int R, int SIGN> struct Dft;
template <int SIGN> struct Dft<2, SIGN> {
    static __device__ __forceinline__ void run(float2 (&v)[2]) {
        const float2 a = v[0];
        v[0] = cadd(a, v[1]); v[1] = csub(a, v[1]);
    }
};
template <int SIGN> struct Dft<4, SIGN> {
    static __device__ __forceinline__ void run(float2 (&v)[4]) {
        const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = cimul<SIGN>(csub(v[1], v[3]));
        v[0] = cadd(a, c); v[1] = cadd(b, d); v[2] = csub(a, c); v[3] = csub(b, d);
    }
};
template <int SIGN> struct Dft<8, SIGN> {
    static __device__ __forceinline__ void run(float2 (&v)[8]) {
        float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        Dft<4, SIGN>::run(e);
        Dft<4, SIGN>::run(o);
        constexpr float h = 0.70710678118654752440f;
        const float2 i1 = cimul<SIGN>(o[1]), i3 = cimul<SIGN>(o[3]);
        o[1] = mk(h * (o[1].x + i1.x), h * (o[1].y + i1.y));
        o[2] = cimul<SIGN>(o[2]);
        o[3] = mk(h * (i3.x - o[3].x), h * (i3.y - o[3].y));
#pragma unroll
        for (int k = 0; k < 4; ++k) { v[k] = cadd(e[k], o[k]); v[k + 4] = csub(e[k], o[k]); }
    }
};
// Odd R: with s_p = v_p + v_(R-p), d_p = v_p - v_(R-p),
// V_q = v_0 + sum_p cos(2 pi p q / R) s_p + SIGN i sum_p sin(2 pi p q / R) d_p.
template <int R> struct OddTab;
template <> struct OddTab<3> {
    static __device__ __forceinline__ double c(int) { return -0.5; }
    static __device__ __forceinline__ double s(int m) { return m == 1 ? 0.86602540378443864676 : -0.86602540378443864676; }
};
template <> struct OddTab<5> {
    static __device__ __forceinline__ double c(int m) { return (m == 1 || m == 4) ? 0.30901699437494742410 : -0.80901699437494742410; }
    static __device__ __forceinline__ double s(int m) {
        return m == 1 ? 0.95105651629515357212 : m == 2 ? 0.58778525229247312917
             : m == 3 ? -0.58778525229247312917 : -0.95105651629515357212;
    }
};
template <> struct OddTab<7> {
    static __device__ __forceinline__ double c(int m) {
        return (m == 1 || m == 6) ? 0.62348980185873353053 : (m == 2 || m == 5) ? -0.22252093395631440429
                                                                                 : -0.90096886790241912624;
    }
    static __device__ __forceinline__ double s(int m) {
        return m == 1 ? 0.78183148246802980871 : m == 2 ? 0.97492791218182360702 : m == 3 ? 0.43388373911755812048
             : m == 4 ? -0.43388373911755812048 : m == 5 ? -0.97492791218182360702 : -0.78183148246802980871;
    }
};
template <int R, int SIGN> struct Dft {
    static __device__ __forceinline__ void run(double2 (&v)[R]) {
        constexpr int H = R / 2;
        double2 s[H], d[H], V[R];
        double2 t = v[0];
#pragma unroll
        for (int p = 0; p < H; ++p) {
            s[p] = cadd(v[p + 1], v[R - 1 - p]);
            d[p] = csub(v[p + 1], v[R - 1 - p]);
            t = cadd(t, s[p]);
        }
        V[0] = t;
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            double2 a = v[0], b = make_double2(0.0, 0.0);
#pragma unroll
            for (int p = 0; p < H; ++p) {
                const int m = ((p + 1) * q) % R;
                const double c = OddTab<R>::c(m), w = OddTab<R>::s(m);
                a.x = fma(c, s[p].x, a.x); a.y = fma(c, s[p].y, a.y);
                b.x = fma(w, d[p].x, b.x); b.y = fma(w, d[p].y, b.y);
            }
            const double2 ib = cimul<SIGN>(b);
            V[q] = cadd(a, ib);
            V[R - q] = csub(a, ib);
        }
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = V[q];
    }
};

// One Stockham pass of radix R over `batch` sequences (stride rs), l the product
// of the radices before: element i + q n/R -> (i - i mod l) R + i mod l + q l.
template <int R, int SIGN>
__device__ __forceinline__ void fft_pass(const float2* __restrict__ in, float2* __restrict__ out, int batch, int rs,
                                         int n, int l, float rnb, float rl, const typename PassOf<R>::T2* __restrict__ tw) {
    using T = typename PassOf<R>::T;
    using T2 = typename PassOf<R>::T2;
    const int nb = n / R, step = nb / l;            // twiddle of (q, k): tw[q k n / (l R)]
    for (int t = threadIdx.x; t < batch * nb; t += blockDim.x) {
        const int b = row_of(t, rnb), i = t - b * nb;
        const int k = i - row_of(i, rl) * l;
        T2 v[R];
        const float2* x = in + b * rs;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const float2 e = x[fpad(i + q * nb)];
            v[q] = mk(static_cast<T>(e.x), static_cast<T>(e.y));
        }
        if (l > 1) {
#pragma unroll
            for (int q = 1; q < R; ++q) {
                T2 w = tw[q * k * step];
                if (SIGN > 0) w.y = -w.y;
                v[q] = cmul(v[q], w);
            }
        }
        Dft<R, SIGN>::run(v);
        float2* y = out + b * rs;
        const int o = (i - k) * R + k;
#pragma unroll
        for (int q = 0; q < R; ++q) y[fpad(o + q * l)] = make_float2(static_cast<float>(v[q].x), static_cast<float>(v[q].y));
    }
}
// A length's twiddles: rounded to single precision, and in double for the odd radices
// (where the length has one).
struct Twiddles {
    const float2* f;
    const double2* d;
};
// The whole transform; the sequences are in `a` (written by this block, not yet
// synced) and come back in the buffer returned (synced).
template <int SIGN>
__device__ __forceinline__ float2* fft_run(float2* a, float2* b, int batch, int rs, const FftPlan& p,
                                           const Twiddles& tw) {
    int l = 1;
    __syncthreads();
    for (int s = 0; s < p.np; ++s) {
        const int r = p.r[s];
        const float rnb = p.rnb[s], rl = p.rl[s];
        if (r == 8) fft_pass<8, SIGN>(a, b, batch, rs, p.n, l, rnb, rl, tw.f);
        else if (r == 4) fft_pass<4, SIGN>(a, b, batch, rs, p.n, l, rnb, rl, tw.f);
        else if (r == 2) fft_pass<2, SIGN>(a, b, batch, rs, p.n, l, rnb, rl, tw.f);
        else if (r == 3) fft_pass<3, SIGN>(a, b, batch, rs, p.n, l, rnb, rl, tw.d);
        else if (r == 5) fft_pass<5, SIGN>(a, b, batch, rs, p.n, l, rnb, rl, tw.d);
        else fft_pass<7, SIGN>(a, b, batch, rs, p.n, l, rnb, rl, tw.d);
        __syncthreads();
        l *= r;
        float2* t = a; a = b; b = t;
    }
    return a;
}
// The twiddles into shared memory from the table of n doubles (published by fft_run's
// first barrier); `rest` is what follows them.
__device__ __forceinline__ Twiddles load_twiddles(double2* __restrict__ sm, const double2* __restrict__ tw, const FftPlan& p,
                                                  float2*& rest) {
    double2* const d = sm;
    float2* const f = reinterpret_cast<float2*>(sm + (p.odd ? p.n : 0));
    for (int t = threadIdx.x; t < p.n; t += kThreads) {
        const double2 w = __ldg(tw + t);
        if (p.odd) d[t] = w;
        f[t] = make_float2(static_cast<float>(w.x), static_cast<float>(w.y));
    }
    rest = f + ((p.n + 1) & ~1);
    return {f, d};
}
// Stride of a sequence of n elements in shared memory: padded, and congruent to 4
// modulo 16 elements so that neighbouring sequences start on different banks.
__host__ __device__ inline int fft_stride(int n) {
    const int p = n + (n >> 4) + 1;
    return p + ((4 - p) & 15);
}

// What every kernel of a solve knows of the grid.
struct GridFftArgs {
    FftPlan px, py;
    const double2 *twx, *twy;
    int nx, ny, nkx, ncell, nk;
    int pr;                            // row pairs per block
    int rsx, rsy;                      // sequence strides
};

// ---- rows, forward ----------------------------------------------------------------
struct RowsFwd {
    GridFftArgs g;
    const float* src[8];               // real planes [ny][nx]
    float2* out;                       // [field][nkx][ny]
};
// A value from the middle of a plane: the median of 32 of its cells (the same in every
// warp). The rows are transformed with it taken off, which changes the k = 0 mode alone,
// and that no solve uses. A mean would put its roundoff into the kx = 0 column: with
// rho's, E_y's error was up to ten times E_x's. (The median and not the mean of the
// cells: a few large ones don't move it.)
__device__ __forceinline__ float plane_middle(const float* __restrict__ src, int ncell) {
    const unsigned lane = threadIdx.x & 31;
    const float v = __ldg(src + (lane + 1u) * 0x9E3779B1u % static_cast<unsigned>(ncell));
    int below = 0;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        const float o = __shfl_sync(0xffffffffu, v, k);
        below += (o < v || (o == v && k < static_cast<int>(lane))) ? 1 : 0;
    }
    const unsigned who = __ballot_sync(0xffffffffu, below == 16);
    return who ? __shfl_sync(0xffffffffu, v, __ffs(static_cast<int>(who)) - 1) : 0.0f;
}
__global__ void __launch_bounds__(kThreads) k_rows_fwd(RowsFwd A) {
    extern __shared__ __align__(16) double2 fsm[];
    const GridFftArgs& g = A.g;
    const int f = blockIdx.y, p0 = blockIdx.x * g.pr;
    float2* b0;
    const Twiddles tw = load_twiddles(fsm, g.twx, g.px, b0);
    float2* const b1 = b0 + g.pr * g.rsx;
    const float rnx = 1.0f / static_cast<float>(g.nx);
    const float* __restrict__ src = A.src[f];
    const float mid = plane_middle(src, g.ncell);
#pragma unroll 4
    for (int t = threadIdx.x; t < g.pr * g.nx; t += kThreads) {
        const int pr = row_of(t, rnx), x = t - pr * g.nx;
        const int ja = 2 * (p0 + pr);
        const float a = ja < g.ny ? __ldg(src + ja * g.nx + x) - mid : 0.f;
        const float b = ja + 1 < g.ny ? __ldg(src + (ja + 1) * g.nx + x) - mid : 0.f;
        b0[pr * g.rsx + fpad(x)] = make_float2(a, b);
    }
    const float2* z = fft_run<-1>(b0, b1, g.pr, g.rsx, g.px, tw);
    // row a: (Z_k + conj Z_-k) / 2, row b: (Z_k - conj Z_-k) / (2 i)
    float2* const out = A.out + static_cast<size_t>(f) * g.nk;
    const float rpr = 1.0f / static_cast<float>(g.pr);
    for (int t = threadIdx.x; t < g.pr * g.nkx; t += kThreads) {
        const int k = row_of(t, rpr), pr = t - k * g.pr;
        const int ja = 2 * (p0 + pr);
        if (ja >= g.ny) continue;
        const float2* s = z + pr * g.rsx;
        const float2 zk = s[fpad(k)], zm = s[fpad(k == 0 ? 0 : g.nx - k)];
        const float2 a = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        const float2 b = make_float2(0.5f * (zk.y + zm.y), 0.5f * (zm.x - zk.x));
        float2* o = out + static_cast<size_t>(k) * g.ny + ja;
        if ((g.ny & 1) == 0) *reinterpret_cast<float4*>(o) = make_float4(a.x, a.y, b.x, b.y);
        else { o[0] = a; if (ja + 1 < g.ny) o[1] = b; }
    }
}

// ---- columns -----------------------------------------------------------------------
// Op: NI planes in, NO planes out (at most NI or NO held at once), one mode at a time.
template <class Op>
struct ColsArgs {
    GridFftArgs g;
    const float2* in[Op::NI];          // [nkx][ny] each
    float2* out;                       // [NO][nkx][ny]
    int cols;                          // columns per block
    Op op;
};
template <class Op>
__global__ void __launch_bounds__(kThreads) k_cols(ColsArgs<Op> A) {
    constexpr int NI = Op::NI, NO = Op::NO, NB = NI > NO ? NI : NO;
    extern __shared__ __align__(16) double2 fsm[];
    const GridFftArgs& g = A.g;
    const int k0 = blockIdx.x * A.cols, C = min(A.cols, g.nkx - k0);
    float2* b0;
    const Twiddles tw = load_twiddles(fsm, g.twy, g.py, b0);
    float2* const b1 = b0 + NB * A.cols * g.rsy;
    const float rny = 1.0f / static_cast<float>(g.ny);
    const int m = C * g.ny;
#pragma unroll
    for (int f = 0; f < NI; ++f)
        for (int t = threadIdx.x; t < m; t += kThreads) {
            const int c = row_of(t, rny), j = t - c * g.ny;
            b0[(f * C + c) * g.rsy + fpad(j)] = __ldg(A.in[f] + static_cast<size_t>(k0) * g.ny + t);
        }
    float2* z = fft_run<-1>(b0, b1, NI * C, g.rsy, g.py, tw);
    for (int t = threadIdx.x; t < m; t += kThreads) {
        const int c = row_of(t, rny), j = t - c * g.ny;
        float2 in[NI], out[NO];
#pragma unroll
        for (int f = 0; f < NI; ++f) in[f] = z[(f * C + c) * g.rsy + fpad(j)];
        A.op(k0 + c, j, in, out);
#pragma unroll
        for (int f = 0; f < NO; ++f) z[(f * C + c) * g.rsy + fpad(j)] = out[f];
    }
    float2* const other = z == b0 ? b1 : b0;
    const float2* y = fft_run<1>(z, other, NO * C, g.rsy, g.py, tw);
#pragma unroll
    for (int f = 0; f < NO; ++f)
        for (int t = threadIdx.x; t < m; t += kThreads) {
            const int c = row_of(t, rny), j = t - c * g.ny;
            A.out[static_cast<size_t>(f) * g.nk + static_cast<size_t>(k0) * g.ny + t] = y[(f * C + c) * g.rsy + fpad(j)];
        }
}

// ---- rows, inverse ------------------------------------------------------------------
struct RowsInv {
    GridFftArgs g;
    const float2* in;                  // [NF][nkx][ny]
    float* out[8];                     // real planes [ny][nx]
};
// One field per blockIdx.y.
__global__ void __launch_bounds__(kThreads) k_rows_inv(RowsInv A) {
    extern __shared__ __align__(16) double2 fsm[];
    const GridFftArgs& g = A.g;
    const int p0 = blockIdx.x * g.pr;
    float2* b0;
    const Twiddles tw = load_twiddles(fsm, g.twx, g.px, b0);
    float2* const b1 = b0 + g.pr * g.rsx;
    const float rpr = 1.0f / static_cast<float>(g.pr);
    const int f = blockIdx.y;
    for (int t = threadIdx.x; t < g.pr * g.nkx; t += kThreads) {
        const int k = row_of(t, rpr), pr = t - k * g.pr;
        const int ja = 2 * (p0 + pr);
        float2 a = make_float2(0.f, 0.f), b = a;
        if (ja < g.ny) {
            const float2* o = A.in + static_cast<size_t>(f) * g.nk + static_cast<size_t>(k) * g.ny + ja;
            if ((g.ny & 1) == 0) {
                const float4 q = __ldg(reinterpret_cast<const float4*>(o));
                a = make_float2(q.x, q.y); b = make_float2(q.z, q.w);
            } else {
                a = __ldg(o);
                if (ja + 1 < g.ny) b = __ldg(o + 1);
            }
        }
        // Z = A + i B with A, B Hermitian: the k = 0 and Nyquist modes of a real row are real
        float2* s = b0 + pr * g.rsx;
        if (k == 0 || 2 * k == g.nx) {
            s[fpad(k)] = make_float2(a.x, b.x);
        } else {
            s[fpad(k)] = make_float2(a.x - b.y, a.y + b.x);
            s[fpad(g.nx - k)] = make_float2(a.x + b.y, b.x - a.y);
        }
    }
    const float2* z = fft_run<1>(b0, b1, g.pr, g.rsx, g.px, tw);
    const float rnx = 1.0f / static_cast<float>(g.nx);
    float* __restrict__ out = A.out[f];
    for (int t = threadIdx.x; t < g.pr * g.nx; t += kThreads) {
        const int pr = row_of(t, rnx), x = t - pr * g.nx;
        const int ja = 2 * (p0 + pr);
        if (ja >= g.ny) continue;
        const float2 v = z[pr * g.rsx + fpad(x)];
        out[ja * g.nx + x] = v.x;
        if (ja + 1 < g.ny) out[(ja + 1) * g.nx + x] = v.y;
    }
}

// ---- the solves' multipliers -----------------------------------------------------------
struct OpEs {
    static constexpr int NI = 1, NO = 2;
    SpecGeo g; double eps0;
    __device__ void operator()(int i, int j, const float2 (&in)[1], float2 (&out)[2]) const {
        es_k(in[0], i, j, g, eps0, out[0], out[1]);
    }
};
struct OpElb {
    static constexpr int NI = 4, NO = 5;
    SpecGeo g; double eps0, c;
    __device__ void operator()(int i, int j, const float2 (&in)[4], float2 (&out)[5]) const { elb_k(i, j, g, eps0, c, in, out); }
};
struct OpEt {
    static constexpr int NI = 7, NO = 3;      // dcu x y z, amu 0..3
    SpecGeo g; double eps0, c, n0;
    __device__ void operator()(int i, int j, const float2 (&in)[7], float2 (&out)[3]) const { et_k(i, j, g, eps0, c, n0, in, out); }
};
// The adjoints' transposes: the conjugate multipliers.
struct OpEsT {       // lrho_k = sum_d conj(K_d) lE_d,k, K_d = -i k_d / (eps0 k^2)
    static constexpr int NI = 2, NO = 1;
    SpecGeo g; double eps0;
    __device__ void operator()(int i, int j, const float2 (&in)[2], float2 (&out)[1]) const { es_T_k(i, j, g, eps0, in, out[0]); }
};
struct OpEtT {
    static constexpr int NI = 3, NO = 7;
    SpecGeo g; double eps0, c, n0;
    __device__ void operator()(int i, int j, const float2 (&in)[3], float2 (&out)[7]) const { et_T_k(i, j, g, eps0, c, n0, in, out); }
};
struct OpElbT {
    static constexpr int NI = 5, NO = 4;
    SpecGeo g; double eps0, c;
    __device__ void operator()(int i, int j, const float2 (&in)[5], float2 (&out)[4]) const { elb_T_k(i, j, g, eps0, c, in, out); }
};
