// Inverse-noise tiles as right-angle convolutions: an overlap-save tile whose
// transform needs no real-FFT untangle.
//
// Reference: algebra/src/toeplitz/toeplitz.c:731-865 (stmm_core overlap-save
// tiles), 569-616 (scmm_direct: forward FFT, spectrum product, inverse FFT),
// 441-470 (circ_init_fftw: the embedding of the band).
//
// A tile of N = 2M real samples x_n is folded into M complex points z_j = x_j +
// i x_(j+M), the polynomial x(u) modulo u^M - i.  With X_k the value of x at u =
// exp(-2 pi i (k + a)/M), a = -1/4 (where u^M = i), the product with the band's
// kernel is X_k H_k with H_k = T_0 + 2 sum_i T_i cos(2 pi i (4k - 1)/(4M)), real
// because the band is symmetric, and the inverse transform is y_j + i y_(j+M), the
// skew-circular convolution of length N (Nussbaumer, Fast Fourier Transform and
// Convolution Algorithms, 1982).  Its wrapped ends fall into the tile's halo and
// are dropped like those of a circular one.  Against the usual packing of even and
// odd samples this costs a constant factor on the inputs of the first and the
// outputs of the last butterfly, and saves the pass that combines the bins k and
// M - k: every bin stands alone, so a row of a four-step split is transformed,
// multiplied and transformed back without seeing another row, and the product sits
// in registers between the last forward and the first inverse butterfly.
//
// M = M1 L points.  Columns (M1 > 1): the M1-point transforms over j1 of j = L j1 +
// j2 in registers, one thread a column, times W_M^(j2 (k1 + a)), to a scratch of
// M1 rows.  Rows: one CTA of L/16 threads a row of L = R 256 points, passes of
// radix R, 16 and 16 with two exchanges through shared memory, the product, and
// the same back.  M1 = 1: the row kernel loads the samples and stores the outputs
// itself, and no scratch is used.  The inverse passes run the forward code on
// values with real and imaginary parts exchanged, conj(DFT(conj v)) =
// swap(DFT(swap v)), a renaming of registers.
//
// FP32: two tiles run as the two lanes of the paired FP32 instructions (same
// twiddles, their own spectra); a shared-memory or scratch entry is 16 bytes, (x_0,
// x_1, y_0, y_1).  FP64: one tile, an entry is (x, y), 16 bytes too.
//
// Measured against the best of the even/odd-packed plans on a B200 (64 x 2^20 samples,
// half bandwidth 2^14): FP32 0.93 -> 0.71 ms (60 instead of ~250 thread instructions a
// complex point in the row kernel), error against 64 bits 5.9e-7 -> 2.6e-7; FP64 1.62 ->
// 1.46 ms, 1.1e-15 -> 8.7e-16.  A spectrum from the transform itself takes microseconds
// where the direct cosine sums took 3.7 ms (half bandwidth 2^13, 2^17 samples).
#include <algorithm>
#include <vector>

#include "lanes.cuh"
#include "mdp_internal.cuh"

namespace {

template <typename T> struct LaneOf;
template <> struct LaneOf<float> {
    using Tag = float;
    using V2 = float2;
    static constexpr int N = 2;
};
template <> struct LaneOf<double> {
    using Tag = mono64;
    using V2 = double2;
    static constexpr int N = 1;
};

template <typename G> struct alignas(16) REnt {  // one complex value per lane
    Pr<G> x, y;
};

// where the samples of one lane's tile lie
template <typename T> struct Lane {
    const T *in;   // the block's first sample
    T       *out;
    int      o;    // window start relative to the block
    int      len;  // block length (0: no tile on this lane)
    int      e;    // outputs of the tile inside the block
    T        mu;
};

// The Toeplitz row as the samples of a window (the skew-circular embedding of the
// band: T_n at n, -T_i at 2M - i), for the spectra
struct RowSrc {
    const double *T;
    int           lambda;
    int           M2;  // 2M
};

enum { RT_TILE, RT_SPEC };

template <typename T>
struct RArgs {
    using V2 = typename LaneOf<T>::V2;
    const T       *vin;
    T             *vout;
    const int64_t *tile_start;  // first output row of each tile
    const int32_t *tile_block;
    const int64_t *blk_start;
    const int32_t *blk_len;
    const int32_t *blk_spec;
    const T       *H;       // [n_spec][M1][16][L/16]: spectrum / M in the order of the row kernel's registers
    const V2      *tw1;     // [R][256]: W_L^(q (k + a)) when M1 = 1, W_L^(q k) otherwise
    const V2      *tw2;     // [16][16]: W_256^(c k)
    const V2      *wa, *wb; // M1 > 1: W_M^(j2 (k1 + a)) = wa[k1][j2 >> 6] wb[k1][j2 & 63]
    const double  *means;   // [ncols][nb]
    REnt<typename LaneOf<T>::Tag> *Y;  // scratch: [item of this launch][M1][L]
    int64_t        n_tiles, units;     // tiles; units of LaneOf::N tiles of a column of the batch
    int64_t        item0;              // first item (column, unit) of this launch
    int64_t        col_stride;
    const int     *active;  // [ncols] or nullptr
    int            lambda, nb, E, log_m1;
    // spectra (RT_SPEC, FP64): rows of the band and where the values go
    const double  *Trows;   // [n_spec][lambda]
    float         *H32;
    double        *H64;
};

template <typename T>
__device__ __forceinline__ bool lanes_of(const RArgs<T> &a, int64_t item, Lane<T> (&ln)[LaneOf<T>::N],
                                         int (&spec)[LaneOf<T>::N]) {
    const uint32_t col = item < a.units ? 0u : (uint32_t) item / (uint32_t) a.units;
    const int64_t  unit = item - col * a.units;
    if (a.active && !a.active[col]) return false;
#pragma unroll
    for (int l = 0; l < LaneOf<T>::N; l++) {
        const int64_t tile = unit * LaneOf<T>::N + l;
        if (tile >= a.n_tiles) {
            ln[l] = Lane<T>{a.vin, a.vout, 0, 0, 0, (T) 0};
            spec[l] = spec[0];
            continue;
        }
        const int     blk = a.tile_block[tile];
        const int64_t bs = a.blk_start[blk] + col * a.col_stride;
        const int     t0 = (int) (a.tile_start[tile] - a.blk_start[blk]);
        ln[l].in = a.vin + bs;
        ln[l].out = a.vout + bs;
        ln[l].o = t0 - (a.lambda - 1);
        ln[l].len = a.blk_len[blk];
        ln[l].e = min(a.E, ln[l].len - t0);
        ln[l].mu = a.means ? (T) a.means[col * a.nb + blk] : (T) 0;
        spec[l] = a.blk_spec[blk];
    }
    return true;
}

// sample n of the window, less the block mean; zero outside the block
template <typename T>
__device__ __forceinline__ T sample(const Lane<T> &ln, int n) {
    const int i = ln.o + n;
    return (unsigned) i < (unsigned) ln.len ? __ldg(ln.in + i) - ln.mu : (T) 0;
}
__device__ __forceinline__ Pr<float> samples(const Lane<float> (&ln)[2], int n) { return pmk(sample(ln[0], n), sample(ln[1], n)); }
__device__ __forceinline__ Pr<mono64> samples(const Lane<double> (&ln)[1], int n) { return Pr<mono64>{sample(ln[0], n)}; }
__device__ __forceinline__ Pr<mono64> samples(const RowSrc &r, int n) {
    return Pr<mono64>{n < r.lambda ? __ldg(r.T + n) : (r.M2 - n < r.lambda ? -__ldg(r.T + (r.M2 - n)) : 0.0)};
}

template <typename T>
__device__ __forceinline__ void put(const Lane<T> &ln, int halo, int n, T v) {
    if ((unsigned) (n - halo) < (unsigned) ln.e) ln.out[ln.o + n] = v;
}
__device__ __forceinline__ void put_all(const Lane<float> (&ln)[2], int halo, int n, Pr<float> v) {
    put(ln[0], halo, n, plo(v));
    put(ln[1], halo, n, phi(v));
}
__device__ __forceinline__ void put_all(const Lane<double> (&ln)[1], int halo, int n, Pr<mono64> v) { put(ln[0], halo, n, v.v); }

// v * w, the same w on every lane
__device__ __forceinline__ CP<float> tmul(CP<float> v, float2 w) {
    const Pr<float> wx = pdup(w.x), wy = pdup(w.y), ny = pdup(-w.y);
    return {pfma(v.y, ny, pmul(v.x, wx)), pfma(v.y, wx, pmul(v.x, wy))};
}
__device__ __forceinline__ CP<mono64> tmul(CP<mono64> v, double2 w) {
    return {Pr<mono64>{fma(-v.y.v, w.y, v.x.v * w.x)}, Pr<mono64>{fma(v.y.v, w.x, v.x.v * w.y)}};
}
__device__ __forceinline__ float2 wmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 wmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }

// cos and sin of 2 pi m / 64, m < 16: exp(-2 pi i a m / R) = exp(2 pi i (16 m / R) / 64)
__host__ __device__ constexpr double c64(int m) {
    return m == 0 ? 1.0 : m == 1 ? 0.99518472667219688624 : m == 2 ? 0.98078528040323044913
         : m == 3 ? 0.95694033573220886494 : m == 4 ? 0.92387953251128675613 : m == 5 ? 0.88192126434835502971
         : m == 6 ? 0.83146961230254523708 : m == 7 ? 0.77301045336273696081 : m == 8 ? 0.70710678118654752440
         : m == 9 ? 0.63439328416364549822 : m == 10 ? 0.55557023301960222474 : m == 11 ? 0.47139673682599764856
         : m == 12 ? 0.38268343236508977173 : m == 13 ? 0.29028467725446236764 : m == 14 ? 0.19509032201612826785
         : m == 15 ? 0.09801714032956060199 : 0.0;
}
__host__ __device__ constexpr double s64(int m) { return m == 0 ? 0.0 : c64(16 - m); }

// v[m] *= exp(2 pi i m / (4 R)): the quarter-bin shift a of the frequencies on an R-point butterfly
template <typename G, int R, int M>
__device__ __forceinline__ void quarter_shift(CP<G> (&v)[R]) {
    if constexpr (M < R) {
        constexpr int m = M * 16 / R;
        v[M] = cpmul(v[M], CP<G>{pcst<G>(c64(m)), pcst<G>(s64(m))});
        quarter_shift<G, R, M + 1>(v);
    }
}
template <typename G, int R>
__device__ __forceinline__ void quarter_shift(CP<G> (&v)[R]) { quarter_shift<G, R, 1>(v); }

__host__ __device__ constexpr int rt_pos(int p) { return p + (p >> 4); }  // padded: every pass spreads over all banks
__host__ __device__ constexpr int rt_entries(int L) { return L + L / 16; }

template <typename G> __device__ __forceinline__ CP<G> get(const REnt<G> *p) {
    const REnt<G> e = *p;
    return {e.x, e.y};
}
template <typename G> __device__ __forceinline__ CP<G> swapped(CP<G> v) { return {v.y, v.x}; }

// ------------------------------------------------------------------ rows
// Row of L = R 256 points, L/16 threads, 16 points a thread in every pass.
//   pass 1  n = 256 a + q over a (R points; 16/R columns q a thread), times tw1
//   pass 2  q = 16 b + c over b, thread (k_a, c), times tw2
//   pass 3  over c, thread (k_a, k_b): bins k_a + R (k_b + 16 k_c), k_c = register
// then the product and the same passes from the other end.  Bound: the FP and
// shared-memory pipes (4 exchanges of 32 bytes an entry).
template <typename T, int R, bool ONE, int SRC>
__global__ void __launch_bounds__(16 * R, R == 16 ? 2 : 32 / R) rt_rows_kernel(RArgs<T> a) {
    using G = typename LaneOf<T>::Tag;
    constexpr int LN = LaneOf<T>::N, L = 256 * R, NT = 16 * R, S = 16 / R;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    REnt<G> *s = reinterpret_cast<REnt<G> *>(smem_raw);
    const int     t = threadIdx.x;
    const int     log_m1 = ONE ? 0 : a.log_m1;
    const int64_t li = blockIdx.x >> log_m1;  // item of this launch
    const int     k1 = (int) blockIdx.x & ((1 << log_m1) - 1);
    const int     M = L << log_m1;
    Lane<T>       ln[LN];
    int           spec[LN];
    RowSrc        rs{};
    if constexpr (SRC == RT_SPEC) {
        rs = RowSrc{a.Trows + (a.item0 + li) * a.lambda, a.lambda, 2 * M};
    } else {
        if (!lanes_of(a, a.item0 + li, ln, spec)) return;
    }
    REnt<G> *Y = ONE ? nullptr : a.Y + (int64_t) blockIdx.x * L;

    CP<G> u[16];
    // pass 1
#pragma unroll
    for (int j = 0; j < S; j++) {
        const int q = t + NT * j;
        CP<G>     v[R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int n = 256 * i + q;
            if constexpr (!ONE) v[i] = get(Y + n);
            else if constexpr (SRC == RT_SPEC) v[i] = CP<G>{samples(rs, n), samples(rs, n + M)};
            else v[i] = CP<G>{samples(ln, n), samples(ln, n + M)};
        }
        if constexpr (ONE) quarter_shift<G, R>(v);
        dif_reg<G, R>(v);
#pragma unroll
        for (int k = 0; k < R; k++) {
            CP<G> w = v[rev_bits_c(k, ilog2_c(R))];
            if (ONE || k > 0) w = tmul(w, __ldg(a.tw1 + k * 256 + q));
            s[rt_pos(k * 256 + q)] = REnt<G>{w.x, w.y};
        }
    }
    __syncthreads();
    // pass 2
    const int c = t & 15, kh = t >> 4;  // also pass 3: (k_a, k_b) = (kh, c)
#pragma unroll
    for (int i = 0; i < 16; i++) u[i] = get(s + rt_pos(kh * 256 + 16 * i + c));
    dif_reg<G, 16>(u);
#pragma unroll
    for (int k = 0; k < 16; k++) {
        CP<G> w = u[rev_bits_c(k, 4)];
        if (k > 0) w = tmul(w, __ldg(a.tw2 + k * 16 + c));
        s[rt_pos(kh * 256 + 16 * k + c)] = REnt<G>{w.x, w.y};
    }
    __syncthreads();
    // pass 3, the product, pass 3 back
#pragma unroll
    for (int i = 0; i < 16; i++) u[i] = get(s + rt_pos(kh * 256 + 16 * c + i));
    dif_reg<G, 16>(u);
    if constexpr (SRC == RT_SPEC) {
        const int64_t at = (((a.item0 + li) << log_m1) + k1) * L + t;
        const double  sc = 1.0 / (double) M;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const double h = u[rev_bits_c(k, 4)].x.v * sc;
            if (a.H32) a.H32[at + k * NT] = (float) h;
            else a.H64[at + k * NT] = h;
        }
        return;
    } else {
        CP<G>    z[16];
        const T *h0 = a.H + (((int64_t) spec[0] << log_m1) + k1) * L + t;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const CP<G> w = u[rev_bits_c(k, 4)];
            Pr<G>       h;
            if constexpr (LN == 2) {
                const T *h1 = a.H + (((int64_t) spec[LN - 1] << log_m1) + k1) * L + t;
                h = pmk(__ldg(h0 + k * NT), __ldg(h1 + k * NT));
            } else {
                h = Pr<G>{__ldg(h0 + k * NT)};
            }
            z[k] = CP<G>{pmul(w.y, h), pmul(w.x, h)};  // real and imaginary parts exchanged from here on
        }
        dif_reg<G, 16>(z);
#pragma unroll
        for (int i = 0; i < 16; i++) {
            CP<G> w = z[rev_bits_c(i, 4)];
            if (i > 0) w = tmul(w, __ldg(a.tw2 + i * 16 + c));  // W_256^(c k_b), symmetric
            s[rt_pos(kh * 256 + 16 * c + i)] = REnt<G>{w.x, w.y};
        }
        __syncthreads();
        // pass 2 back
#pragma unroll
        for (int k = 0; k < 16; k++) z[k] = get(s + rt_pos(kh * 256 + 16 * k + c));
        dif_reg<G, 16>(z);
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const CP<G> w = tmul(z[rev_bits_c(i, 4)], __ldg(a.tw1 + kh * 256 + 16 * i + c));
            s[rt_pos(kh * 256 + 16 * i + c)] = REnt<G>{w.x, w.y};
        }
        __syncthreads();
        // pass 1 back
#pragma unroll
        for (int j = 0; j < S; j++) {
            const int q = t + NT * j;
            CP<G>     v[R], y[R];
#pragma unroll
            for (int k = 0; k < R; k++) v[k] = get(s + rt_pos(k * 256 + q));
            dif_reg<G, R>(v);
#pragma unroll
            for (int i = 0; i < R; i++) y[i] = v[rev_bits_c(i, ilog2_c(R))];
            if constexpr (ONE) quarter_shift<G, R>(y);
#pragma unroll
            for (int i = 0; i < R; i++) {
                const int n = 256 * i + q;
                if constexpr (ONE) {
                    put_all(ln, a.lambda - 1, n, y[i].y);
                    put_all(ln, a.lambda - 1, n + M, y[i].x);
                } else {
                    Y[n] = REnt<G>{y[i].x, y[i].y};
                }
            }
        }
    }
}

// ------------------------------------------------------------------ columns
// M1-point transforms over j1 of the columns j2, one thread a column, 16 points a
// thread; L = 4096.  Bound: memory (samples in, scratch out, and back).
template <typename T, int M1, bool INV, int SRC>
__global__ void __launch_bounds__(256, 2) rt_cols_kernel(RArgs<T> a) {
    using G = typename LaneOf<T>::Tag;
    constexpr int LN = LaneOf<T>::N, L = 4096, M = M1 * L, S = 16 / M1;
    const int64_t li = blockIdx.x / (unsigned) M1;
    const int     j0 = (int) (blockIdx.x % M1) * (256 * S) + threadIdx.x;
    Lane<T>       ln[LN];
    int           spec[LN];
    RowSrc        rs{};
    if constexpr (SRC == RT_SPEC) {
        rs = RowSrc{a.Trows + (a.item0 + li) * a.lambda, a.lambda, 2 * M};
    } else {
        if (!lanes_of(a, a.item0 + li, ln, spec)) return;
    }
    REnt<G> *Y = a.Y + li * M;
    CP<G>    v[S][M1];
    if constexpr (!INV) {
#pragma unroll
        for (int j = 0; j < S; j++)
#pragma unroll
            for (int i = 0; i < M1; i++) {
                const int n = L * i + j0 + 256 * j;
                if constexpr (SRC == RT_SPEC) v[j][i] = CP<G>{samples(rs, n), samples(rs, n + M)};
                else v[j][i] = CP<G>{samples(ln, n), samples(ln, n + M)};
            }
    } else {
#pragma unroll
        for (int j = 0; j < S; j++)
#pragma unroll
            for (int k = 0; k < M1; k++) v[j][k] = get(Y + k * L + j0 + 256 * j);
    }
#pragma unroll
    for (int j = 0; j < S; j++) {
        const int j2 = j0 + 256 * j;
        if constexpr (!INV) {
            quarter_shift<G, M1>(v[j]);
            dif_reg<G, M1>(v[j]);
#pragma unroll
            for (int k = 0; k < M1; k++) {
                const CP<G> w = tmul(v[j][rev_bits_c(k, ilog2_c(M1))],
                                     wmul(__ldg(a.wa + k * 64 + (j2 >> 6)), __ldg(a.wb + k * 64 + (j2 & 63))));
                Y[k * L + j2] = REnt<G>{w.x, w.y};
            }
        } else {  // real and imaginary parts exchanged
#pragma unroll
            for (int k = 0; k < M1; k++)
                v[j][k] = tmul(v[j][k], wmul(__ldg(a.wa + k * 64 + (j2 >> 6)), __ldg(a.wb + k * 64 + (j2 & 63))));
            dif_reg<G, M1>(v[j]);
            CP<G> y[M1];
#pragma unroll
            for (int i = 0; i < M1; i++) y[i] = v[j][rev_bits_c(i, ilog2_c(M1))];
            quarter_shift<G, M1>(y);
#pragma unroll
            for (int i = 0; i < M1; i++) {
                put_all(ln, a.lambda - 1, L * i + j2, y[i].y);
                put_all(ln, a.lambda - 1, L * i + j2 + M, y[i].x);
            }
        }
    }
}

// ------------------------------------------------------------------ host side
// items (tiles of FP64, pairs of tiles of FP32) whose columns, rows and columns back
// are launched together: their scratch stays in L2 between the three kernels
#ifndef RT_GROUP_BYTES
#define RT_GROUP_BYTES (int64_t(64) << 20)
#endif

template <typename T> size_t rows_smem(int L) { return 16 * (size_t) rt_entries(L); }

template <typename T, bool ONE, int SRC>
const void *rows_fn(int L) {
    if constexpr (ONE) {
        switch (L) {
            case 512: return (const void *) rt_rows_kernel<T, 2, true, SRC>;
            case 1024: return (const void *) rt_rows_kernel<T, 4, true, SRC>;
            case 2048: return (const void *) rt_rows_kernel<T, 8, true, SRC>;
        }
    }
    return L == 4096 ? (const void *) rt_rows_kernel<T, 16, ONE, SRC> : nullptr;
}
template <typename T, bool INV, int SRC>
const void *cols_fn(int m1) {
    switch (m1) {
        case 2: return (const void *) rt_cols_kernel<T, 2, INV, SRC>;
        case 4: return (const void *) rt_cols_kernel<T, 4, INV, SRC>;
        case 8: return (const void *) rt_cols_kernel<T, 8, INV, SRC>;
        case 16: return (const void *) rt_cols_kernel<T, 16, INV, SRC>;
    }
    return nullptr;
}

inline void set2(float2 &o, double x, double y) { o = make_float2((float) x, (float) y); }
inline void set2(double2 &o, double x, double y) { o = make_double2(x, y); }

// tables of the transform in the order tw1, tw2, wa, wb, one buffer
template <typename V2>
int build_tables(int m1, int L, DevBuf &buf, const V2 **tw1, const V2 **tw2, const V2 **wa, const V2 **wb) {
    const int       R = L / 256, M = m1 * L;
    std::vector<V2> t(L + 256 + (m1 > 1 ? 128 * m1 : 0));
    double          re, im;
    for (int k = 0; k < R; k++)
        for (int q = 0; q < 256; q++) {
            // W_L^(q (k - 1/4)) = W_4L^(q (4k - 1)), exponents modulo 4L
            const int64_t e = m1 == 1 ? (int64_t) q * (4 * k - 1) : (int64_t) 4 * q * k;
            mdp_host_cexp((long double) ((e + 4LL * L) % (4LL * L)), 4.0L * L, &re, &im);
            set2(t[k * 256 + q], re, im);
        }
    for (int k = 0; k < 16; k++)
        for (int c = 0; c < 16; c++) {
            mdp_host_cexp(k * c, 256, &re, &im);
            set2(t[L + 16 * k + c], re, im);
        }
    if (m1 > 1)
        for (int k = 0; k < m1; k++)
            for (int h = 0; h < 64; h++) {
                const int64_t den = 4LL * M, ea = 64LL * h * (4 * k - 1), eb = (int64_t) h * (4 * k - 1);
                mdp_host_cexp((long double) ((ea + den) % den), (long double) den, &re, &im);
                set2(t[L + 256 + 64 * k + h], re, im);
                mdp_host_cexp((long double) ((eb + den) % den), (long double) den, &re, &im);
                set2(t[L + 256 + 64 * m1 + 64 * k + h], re, im);
            }
    MDP_TRY(buf.alloc(sizeof(V2) * t.size()));
    MDP_CUDA(cudaMemcpy(buf.p, t.data(), sizeof(V2) * t.size(), cudaMemcpyHostToDevice));
    *tw1 = buf.as<V2>();
    *tw2 = *tw1 + L;
    *wa = *tw2 + 256;
    *wb = *wa + 64 * m1;
    return MDP_OK;
}

template <typename T>
int64_t group_items(int64_t M) { return std::max<int64_t>(1, RT_GROUP_BYTES / (16 * M)); }

}  // namespace

bool rtile_shape(int log_m1, int log_m2) {
    return log_m1 == 0 ? log_m2 >= 9 && log_m2 <= 12 : log_m1 >= 1 && log_m1 <= 4 && log_m2 == 12;
}

// Tables, scratch and spectra of a plan of M = 2^log_m1 x 2^log_m2 points (log_m2 = 12 when log_m1 > 0).  The
// spectra are the transform's own values of the embedded band, in FP64, rounded to T.
template <typename T>
int rtile_build(mdp_context *ctx, mdp_noise *N, mdp_tile_plan &P, bool spectra) {
    using V2 = typename LaneOf<T>::V2;
    const int m1 = 1 << P.log_m1, L = 1 << P.log_m2, M = m1 * L;
    if (!rtile_shape(P.log_m1, P.log_m2)) return MDP_EUNSUPPORTED;
    const V2 *p[4];
    MDP_TRY(build_tables<V2>(m1, L, P.ltw, &p[0], &p[1], &p[2], &p[3]));
    const int64_t units = (P.n_tiles + LaneOf<T>::N - 1) / LaneOf<T>::N;
    if (m1 > 1) {
        // FP32 plans also run column batches of up to 8 columns
        const int64_t items = std::min(group_items<T>(M), std::max<int64_t>(1, units * (sizeof(T) == 4 ? 8 : 1)));
        MDP_TRY(P.scratch.alloc(16 * (size_t) items * M));
    }
    const size_t nh = (size_t) std::max(N->n_spec, 1) * M;
    MDP_TRY(P.spectra.alloc(sizeof(T) * nh));
    const void *fr = m1 == 1 ? rows_fn<T, true, RT_TILE>(L) : rows_fn<T, false, RT_TILE>(L);
    MDP_CUDA(cudaFuncSetAttribute(fr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) rows_smem<T>(L)));
    if (!spectra) {
        MDP_CUDA(cudaMemset(P.spectra.p, 0, sizeof(T) * nh));
        return MDP_OK;
    }
    RArgs<double> a{};
    DevBuf        tab, rows, Y;
    MDP_TRY(build_tables<double2>(m1, L, tab, &a.tw1, &a.tw2, &a.wa, &a.wb));
    MDP_TRY(rows.alloc(sizeof(double) * N->h_Tuniq.size()));
    MDP_CUDA(cudaMemcpyAsync(rows.p, N->h_Tuniq.data(), sizeof(double) * N->h_Tuniq.size(), cudaMemcpyHostToDevice,
                             ctx->stream));
    const int64_t per = m1 > 1 ? std::min<int64_t>(N->n_spec, group_items<double>(M)) : N->n_spec;
    if (m1 > 1) MDP_TRY(Y.alloc(16 * (size_t) per * M));
    a.Trows = rows.as<double>();
    a.lambda = N->lambda;
    a.log_m1 = P.log_m1;
    a.Y = Y.as<REnt<mono64>>();
    if (sizeof(T) == 4) a.H32 = P.spectra.as<float>();
    else a.H64 = P.spectra.as<double>();
    const void *fs = m1 == 1 ? rows_fn<double, true, RT_SPEC>(L) : rows_fn<double, false, RT_SPEC>(L);
    MDP_CUDA(cudaFuncSetAttribute(fs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) rows_smem<double>(L)));
    for (int64_t i = 0; i < N->n_spec; i += per) {
        const int64_t n = std::min<int64_t>(per, N->n_spec - i);
        a.item0 = i;
        void *args[] = {&a};
        if (m1 > 1) {
            MDP_CUDA(cudaLaunchKernel(cols_fn<double, false, RT_SPEC>(m1), dim3((unsigned) (n * m1)), dim3(256), args, 0,
                                      ctx->stream));
            MDP_CHECK_LAUNCH(ctx);
        }
        MDP_CUDA(cudaLaunchKernel(fs, dim3((unsigned) (n * m1)), dim3(L / 16), args, rows_smem<double>(L), ctx->stream));
        MDP_CHECK_LAUNCH(ctx);
    }
    MDP_CUDA(cudaStreamSynchronize(ctx->stream));  // the temporaries are released on return
    return MDP_OK;
}

template <typename T>
int rtile_launch(mdp_context *ctx, const mdp_noise *N, const mdp_tile_plan &P, const T *d_in, T *d_out,
                 const double *d_means, int ncols, int64_t col_stride, const int *d_active) {
    using V2 = typename LaneOf<T>::V2;
    const int m1 = 1 << P.log_m1, L = 1 << P.log_m2, M = m1 * L;
    RArgs<T>  a{};
    a.vin = d_in;
    a.vout = d_out;
    a.tile_start = P.tile_start.as<int64_t>();
    a.tile_block = P.tile_block.as<int32_t>();
    a.blk_start = N->blk_start.as<int64_t>();
    a.blk_len = N->blk_len.as<int32_t>();
    a.blk_spec = N->blk_spec.as<int32_t>();
    a.H = P.spectra.as<T>();
    a.tw1 = P.ltw.as<V2>();
    a.tw2 = a.tw1 + L;
    a.wa = a.tw2 + 256;
    a.wb = a.wa + 64 * m1;
    a.means = d_means;
    a.Y = P.scratch.as<REnt<typename LaneOf<T>::Tag>>();
    a.n_tiles = P.n_tiles;
    a.units = (P.n_tiles + LaneOf<T>::N - 1) / LaneOf<T>::N;
    a.col_stride = col_stride;
    a.active = d_active;
    a.lambda = N->lambda;
    a.nb = N->nb;
    a.E = P.fft_n - 2 * (N->lambda - 1);
    a.log_m1 = P.log_m1;
    const int64_t items = a.units * ncols;
    if (items << P.log_m1 > 0x7fffffffLL) return MDP_EUNSUPPORTED;
    const int64_t per = m1 > 1 ? (int64_t) (P.scratch.bytes / (16 * (size_t) M)) : (int64_t) 0x7fffffff;
    const void   *fr = m1 == 1 ? rows_fn<T, true, RT_TILE>(L) : rows_fn<T, false, RT_TILE>(L);
    for (int64_t i = 0; i < items; i += per) {
        const int64_t n = std::min(per, items - i);
        a.item0 = i;
        void      *args[] = {&a};
        const dim3 grid((unsigned) (n * m1));
        if (m1 > 1) {
            MDP_CUDA(cudaLaunchKernel(cols_fn<T, false, RT_TILE>(m1), grid, dim3(256), args, 0, ctx->stream));
            MDP_CHECK_LAUNCH(ctx);
        }
        MDP_CUDA(cudaLaunchKernel(fr, grid, dim3(L / 16), args, rows_smem<T>(L), ctx->stream));
        MDP_CHECK_LAUNCH(ctx);
        if (m1 > 1) {
            MDP_CUDA(cudaLaunchKernel(cols_fn<T, true, RT_TILE>(m1), grid, dim3(256), args, 0, ctx->stream));
            MDP_CHECK_LAUNCH(ctx);
        }
    }
    return MDP_OK;
}

template int rtile_build<float>(mdp_context *, mdp_noise *, mdp_tile_plan &, bool);
template int rtile_build<double>(mdp_context *, mdp_noise *, mdp_tile_plan &, bool);
template int rtile_launch<float>(mdp_context *, const mdp_noise *, const mdp_tile_plan &, const float *, float *,
                                 const double *, int, int64_t, const int *);
template int rtile_launch<double>(mdp_context *, const mdp_noise *, const mdp_tile_plan &, const double *, double *,
                                  const double *, int, int64_t, const int *);
