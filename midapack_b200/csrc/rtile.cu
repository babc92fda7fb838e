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
// One tile a CTA (FP32: 16 points take 32 of 80 registers, three CTAs of 256 threads an SM;
// FP64: 64 of 128, two).  FP32 complex sums are one paired FP32 instruction (add/sub
// .f32x2) on (x, y).  Two FP32 tiles on the lanes of paired instructions took fewer
// instructions and half the resident warps: 0.71 against 0.70 ms below, 131 against 94 us for
// 8 x 2^20 samples at half bandwidth 2^13.
//
// Measured against the best of the even/odd-packed plans on a B200 (64 x 2^20 samples,
// half bandwidth 2^14): FP32 0.93 -> 0.58 ms, error against 64 bits 5.9e-7 -> 2.7e-7; FP64
// 1.62 -> 1.19 ms, 1.1e-15 -> 8.3e-16.  The row kernel takes half of it: L1 74 % busy in
// FP32, waiting for its loads in FP64; the columns wait for theirs.  A spectrum from the transform itself takes
// microseconds where the direct cosine sums took 3.7 ms (half bandwidth 2^13, 2^17 samples).
#include <algorithm>
#include <cmath>
#include <vector>

#include "lanes.cuh"
#include "mdp_internal.cuh"

namespace {

template <typename T> struct LaneOf;
template <> struct LaneOf<float> {
    using Tag = mono32;
    using V2 = float2;
};
template <> struct LaneOf<double> {
    using Tag = mono64;
    using V2 = double2;
};

template <typename G> struct alignas(2 * sizeof(Pr<G>)) REnt {  // a complex value in shared memory or scratch
    Pr<G> x, y;
};

// a tile's window: sample n is in[n] for lo <= n < lo + cnt and zero outside the block; output n is out[n]
template <typename T> struct Tile {
    const T *in;
    T       *out;
    int      lo, cnt;
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

template <typename T>
struct RArgs {
    using V2 = typename LaneOf<T>::V2;
    const T       *vin;
    T             *vout;
    const mdp_rtile *tiles;
    const T       *H;       // [n_spec][M1][L]: spectrum / M in the order of the row kernel's registers (see h_at)
    const V2      *tw1;     // [R][256]: W_L^(q (k + a)) when M1 = 1, W_L^(q k) otherwise (see tw_at)
    const V2      *tw1b;    // the same for the pass back: [R][16][16], q = 16 i + c
    const V2      *tw2;     // [16][16]: W_256^(c k)
    const V2      *wa, *wb; // M1 > 1: W_M^(j2 (k1 + a)) = wa[k1][j2 >> 6] wb[k1][j2 & 63]
    const double  *means;   // [ncols][nb]
    REnt<typename LaneOf<T>::Tag> *Y;  // scratch: [item of this launch][M1][L]
    int64_t        n_tiles;
    int64_t        item0;              // first item (column of the batch, tile) of this launch
    int64_t        col_stride;
    const int     *active;  // [ncols] or nullptr
    int            lambda, nb, log_m1;
    // spectra (RT_SPEC, FP64): rows of the band and where the values go
    const double  *Trows;   // [n_spec][lambda]
    float         *H32;
    double        *H64;
};

// the tile of an item; false when its column is not to be applied
template <typename T>
__device__ __forceinline__ bool tile_of(const RArgs<T> &a, int64_t item, Tile<T> &tl, int &spec) {
    const uint32_t col = item < a.n_tiles ? 0u : (uint32_t) item / (uint32_t) a.n_tiles;
    const int64_t  tile = item - col * a.n_tiles;
    chain_next();
    const int4 d0 = __ldg(reinterpret_cast<const int4 *>(a.tiles + tile)), d1 = __ldg(reinterpret_cast<const int4 *>(a.tiles + tile) + 1);
    const int64_t bs = (int64_t) (((uint64_t) (uint32_t) d0.y << 32) | (uint32_t) d0.x) + col * a.col_stride;
    tl.in = a.vin + bs;
    tl.out = a.vout + bs;
    tl.lo = d0.z;
    tl.cnt = d0.w;
    tl.e = d1.x;
    spec = d1.y;
    chain_wait();  // the records above are the plan's own; all else may come from the kernel before
    if (a.active && !a.active[col]) return false;
    tl.mu = a.means ? (T) a.means[col * a.nb + d1.z] : (T) 0;
    return true;
}

__device__ __forceinline__ float ld_sample(const float *p) {  // from the kernel before (as ld_after), read once
    float v;
    asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_sample(const double *p) {
    double v;
    asm volatile("ld.global.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
// sample n of the window, less the block mean; zero outside the block
template <typename T>
__device__ __forceinline__ T sample(const Tile<T> &tl, int n) {
    return (unsigned) (n - tl.lo) < (unsigned) tl.cnt ? ld_sample(tl.in + n) - tl.mu : (T) 0;
}
// the same of a window inside its block: point j0 + n, n known at compile time
template <typename T>
__device__ __forceinline__ T sample_in(const Tile<T> &tl, int j0, int n) {
    return ld_sample(tl.in + j0 + n) - tl.mu;
}
__device__ __forceinline__ double sample(const RowSrc &r, int n) {
    return n < r.lambda ? __ldg(r.T + n) : (r.M2 - n < r.lambda ? -__ldg(r.T + (r.M2 - n)) : 0.0);
}
template <typename T>
__device__ __forceinline__ void put(const Tile<T> &tl, int halo, int n, T v) {
    if ((unsigned) (n - halo) < (unsigned) tl.e) tl.out[n] = v;
}
template <typename T>
__device__ __forceinline__ CP<typename LaneOf<T>::Tag> point(T x, T y) {
    using G = typename LaneOf<T>::Tag;
    return CP<G>{Pr<G>{x}, Pr<G>{y}};
}

// v * w
template <typename G, typename V2>
__device__ __forceinline__ CP<G> tmul(CP<G> v, V2 w) {
    return {pfma(Pr<G>{-v.y.v}, Pr<G>{w.y}, pmul(v.x, Pr<G>{w.x})), pfma(v.y, Pr<G>{w.x}, pmul(v.x, Pr<G>{w.y}))};
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
// from L2, where the kernel before wrote it
__device__ __forceinline__ CP<mono32> get_l2(const REnt<mono32> *p) {
    float2 v;
    asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return {Pr<mono32>{v.x}, Pr<mono32>{v.y}};
}
__device__ __forceinline__ CP<mono64> get_l2(const REnt<mono64> *p) {
    double2 v;
    asm volatile("ld.global.cg.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return {Pr<mono64>{v.x}, Pr<mono64>{v.y}};
}

// CTAs of 256 threads an SM that transform rows: three FP32 ones (80 registers a thread: 16 points
// take 32, the 16-byte loads of twiddles and spectrum in flight the rest), two FP64 ones.  Columns: four.
// 64 x 2^20 samples, half bandwidth 2^14: 4-byte spectrum and 8-byte twiddle loads 623 us at four CTAs
// (64 registers), 641 at three; 16-byte loads 632 at four, 588 at three; with four for the columns 583.
// FP64 spectrum loads of 16 bytes: 1224 -> 1190 us.
template <typename T> constexpr int rt_ctas() { return sizeof(T) == 4 ? 3 : 2; }
template <typename T> constexpr int rt_col_ctas() { return sizeof(T) == 4 ? 4 : 2; }

// ------------------------------------------------------------------ rows
// Row of L = R 256 points, L/16 threads, 16 points a thread in every pass.
//   pass 1  n = 256 a + q over a (R points; 16/R columns q a thread), times tw1
//   pass 2  q = 16 b + c over b, thread (k_a, c), times tw2
//   pass 3  over c, thread (k_a, k_b): bins k_a + R (k_b + 16 k_c), k_c = register
// then the product and the same passes from the other end.  Bound: FP32 shared memory
// and issue (four exchanges of a write and a read of each 8-byte point: L1 74 % busy, 48 % of
// the issue slots), FP64 (16-byte points: 62 %, 25 %) the latency of its loads at 16 warps an SM.

// Tables are read 16 bytes at a time: FP32 twiddles of two consecutive k lie side by side ([k/2][n][2]
// instead of [k][n]), a thread's spectrum values four (FP32) or two (FP64) together.
template <typename V2> __host__ __device__ constexpr int tw_at(int k, int q, int n) {
    return sizeof(V2) == 8 ? ((k >> 1) * n + q) * 2 + (k & 1) : k * n + q;
}
__device__ __forceinline__ void tw_load(const float2 *t, int k, int q, int n, float2 (&w)[2]) {  // k even
    const float4 v = __ldg(reinterpret_cast<const float4 *>(t) + ((k >> 1) * n + q));
    w[0] = make_float2(v.x, v.y);
    w[1] = make_float2(v.z, v.w);
}
__device__ __forceinline__ void tw_load(const double2 *t, int k, int q, int n, double2 (&w)[1]) { w[0] = __ldg(t + k * n + q); }
// the registers of a butterfly times their twiddles; FIRST: register 0 has one too
template <bool FIRST, typename G, int R, typename V2, typename Put>
__device__ __forceinline__ void twiddled(const CP<G> (&v)[R], const V2 *t, int q, int n, Put put) {
    constexpr int W = 16 / (int) sizeof(V2);
#pragma unroll
    for (int k = 0; k < R; k += W) {
        V2 w[W];
        tw_load(t, k, q, n, w);
#pragma unroll
        for (int i = 0; i < W; i++) {
            CP<G> e = v[rev_bits_c(k + i, ilog2_c(R))];
            if (FIRST || k + i > 0) e = tmul(e, w[i]);
            put(k + i, REnt<G>{e.x, e.y});
        }
    }
}
// register k of thread t, nt threads
template <typename T> __host__ __device__ constexpr int h_at(int k, int t, int nt) {
    constexpr int W = 16 / (int) sizeof(T);
    return ((k / W) * nt + t) * W + k % W;
}
__device__ __forceinline__ float4 ld_stream4(const float *p) {  // constant, read once: not kept in L1
    float4 v;
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ double2 ld_stream4(const double *p) {
    double2 v;
    asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

// passes 1 to 3 of a row: in(n) gives point n; u[rev(k)] = bin of register k.  ONE: quarter shift
template <typename T, int R, bool ONE, typename In>
__device__ __forceinline__ void row_forward(REnt<typename LaneOf<T>::Tag> *s, const typename LaneOf<T>::V2 *tw1,
                                            const typename LaneOf<T>::V2 *tw2, In in,
                                            CP<typename LaneOf<T>::Tag> (&u)[16]) {
    using G = typename LaneOf<T>::Tag;
    using V2 = typename LaneOf<T>::V2;
    constexpr int NT = 16 * R, S = 16 / R;
    const int     t = threadIdx.x, c = t & 15, kh = t >> 4;
#pragma unroll
    for (int j = 0; j < S; j++) {
        const int q = t + NT * j;
        CP<G>     v[R];
#pragma unroll
        for (int i = 0; i < R; i++) v[i] = in(256 * i + q);
        if constexpr (ONE) quarter_shift<G, R>(v);
        dif_reg<G, R>(v);
        twiddled<ONE>(v, tw1, q, 256, [&](int k, REnt<G> e) { s[rt_pos(k * 256 + q)] = e; });
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; i++) u[i] = get(s + rt_pos(kh * 256 + 16 * i + c));
    dif_reg<G, 16>(u);
    twiddled<false>(u, tw2, c, 16, [&](int k, REnt<G> e) { s[rt_pos(kh * 256 + 16 * k + c)] = e; });
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; i++) u[i] = get(s + rt_pos(kh * 256 + 16 * c + i));  // (k_a, k_b) = (kh, c)
    dif_reg<G, 16>(u);
}

// the passes back from z[k] (register k, parts exchanged); out(n, v) takes point n
template <typename T, int R, bool ONE, typename Out>
__device__ __forceinline__ void row_back(REnt<typename LaneOf<T>::Tag> *s, const typename LaneOf<T>::V2 *tw1b,
                                         const typename LaneOf<T>::V2 *tw2, CP<typename LaneOf<T>::Tag> (&z)[16],
                                         Out out) {
    using G = typename LaneOf<T>::Tag;
    using V2 = typename LaneOf<T>::V2;
    constexpr int NT = 16 * R, S = 16 / R;
    const int     t = threadIdx.x, c = t & 15, kh = t >> 4;
    dif_reg<G, 16>(z);
    twiddled<false>(z, tw2, c, 16, [&](int i, REnt<G> e) { s[rt_pos(kh * 256 + 16 * c + i)] = e; });  // W_256^(c k_b)
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; k++) z[k] = get(s + rt_pos(kh * 256 + 16 * k + c));
    dif_reg<G, 16>(z);
    twiddled<true>(z, tw1b + kh * 256, c, 16, [&](int i, REnt<G> e) { s[rt_pos(kh * 256 + 16 * i + c)] = e; });
    __syncthreads();
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
        for (int i = 0; i < R; i++) out(256 * i + q, y[i]);
    }
}

// z[k] = u[rev(k)] H, real and imaginary parts exchanged; h: the thread's values (nt threads)
template <typename T, typename G>
__device__ __forceinline__ void row_product(const CP<G> (&u)[16], const T *h, int nt, CP<G> (&z)[16]) {
    constexpr int W = 16 / (int) sizeof(T);
#pragma unroll
    for (int k = 0; k < 16; k += W) {
        const auto v = ld_stream4(h + (k / W) * nt * W);
        T          hk[W];
        hk[0] = v.x;
        hk[1] = v.y;
        if constexpr (W == 4) {
            hk[2] = v.z;
            hk[3] = v.w;
        }
#pragma unroll
        for (int i = 0; i < W; i++) {
            const CP<G> w = u[rev_bits_c(k + i, 4)];
            z[k + i] = CP<G>{pmul(w.y, Pr<G>{hk[i]}), pmul(w.x, Pr<G>{hk[i]})};
        }
    }
}

// tiles of one row (M = L): samples in, outputs out
template <typename T, int R>
__global__ void __launch_bounds__(16 * R, rt_ctas<T>() * 16 / R) rt_one_kernel(RArgs<T> a) {
    using G = typename LaneOf<T>::Tag;
    constexpr int M = 256 * R, NT = 16 * R;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    REnt<G> *s = reinterpret_cast<REnt<G> *>(smem_raw);
    Tile<T>  tl;
    int      spec;
    if (!tile_of(a, a.item0 + blockIdx.x, tl, spec)) return;
    CP<G>     u[16], z[16];
    const int halo = a.lambda - 1;
    row_forward<T, R, true>(s, a.tw1, a.tw2, [&](int n) { return point(sample(tl, n), sample(tl, n + M)); }, u);
    row_product(u, a.H + (int64_t) spec * M + threadIdx.x * (16 / sizeof(T)), NT, z);
    row_back<T, R, true>(s, a.tw1b, a.tw2, z, [&](int n, CP<G> y) {
        put(tl, halo, n, y.y.v);
        put(tl, halo, n + M, y.x.v);
    });
}

// the spectra / M of rows of the band (FP64): one-row tiles (ONE) or the rows after the columns
template <int R, bool ONE>
__global__ void __launch_bounds__(16 * R, R == 16 ? 2 : 32 / R) rt_spec_rows_kernel(RArgs<double> a) {
    constexpr int L = 256 * R, NT = 16 * R;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    REnt<mono64> *s = reinterpret_cast<REnt<mono64> *>(smem_raw);
    const int     M = L << a.log_m1;
    const RowSrc  rs{a.Trows + (a.item0 + blockIdx.x) * a.lambda, a.lambda, 2 * M};
    REnt<mono64> *Y = a.Y + (int64_t) blockIdx.x * L;
    CP<mono64>    u[16];
    row_forward<double, R, ONE>(s, a.tw1, a.tw2, [&](int n) {
        if constexpr (ONE) return point(sample(rs, n), sample(rs, n + M));
        else return get(Y + n);
    }, u);
    const int64_t at = ((a.item0 << a.log_m1) + blockIdx.x) * L;
    const double  sc = 1.0 / (double) M;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const double h = u[rev_bits_c(k, 4)].x.v * sc;
        if (a.H32) a.H32[at + h_at<float>(k, threadIdx.x, NT)] = (float) h;
        else a.H64[at + h_at<double>(k, threadIdx.x, NT)] = h;
    }
}

// ------------------------------------------------------------------ columns
// M1-point transforms over j1 of the columns j2, one thread a column, 16 points a
// thread: part p of M1 covers columns p (4096/M1) on; L = 4096.
template <typename T, int M1, typename In>
__device__ __forceinline__ void cols_forward(const RArgs<T> &a, int part, REnt<typename LaneOf<T>::Tag> *Y, In in) {
    using G = typename LaneOf<T>::Tag;
    constexpr int L = 4096, S = 16 / M1;
    const int     j0 = part * (256 * S) + (int) threadIdx.x;
    CP<G>         v[S][M1];
#pragma unroll
    for (int j = 0; j < S; j++)
#pragma unroll
        for (int i = 0; i < M1; i++) v[j][i] = in(j0, L * i + 256 * j);
#pragma unroll
    for (int j = 0; j < S; j++) {
        const int j2 = j0 + 256 * j;
        quarter_shift<G, M1>(v[j]);
        dif_reg<G, M1>(v[j]);
#pragma unroll
        for (int k = 0; k < M1; k++) {
            const CP<G> w = tmul(v[j][rev_bits_c(k, ilog2_c(M1))],
                                 wmul(__ldg(a.wa + k * 64 + (j2 >> 6)), __ldg(a.wb + k * 64 + (j2 & 63))));
            Y[k * L + j2] = REnt<G>{w.x, w.y};
        }
    }
}

// and back, from rows whose parts are exchanged
template <typename T, int M1>
__device__ __forceinline__ void cols_back(const RArgs<T> &a, int part, const REnt<typename LaneOf<T>::Tag> *Y,
                                          const Tile<T> &tl) {
    using G = typename LaneOf<T>::Tag;
    constexpr int L = 4096, M = M1 * L, S = 16 / M1;
    const int     j0 = part * (256 * S) + (int) threadIdx.x, halo = a.lambda - 1;
    CP<G>         v[S][M1];
#pragma unroll
    for (int j = 0; j < S; j++)
#pragma unroll
        for (int k = 0; k < M1; k++) v[j][k] = get_l2(Y + k * L + j0 + 256 * j);
#pragma unroll
    for (int j = 0; j < S; j++) {
        const int j2 = j0 + 256 * j;
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
            put(tl, halo, L * i + j2, y[i].y.v);
            put(tl, halo, L * i + j2 + M, y[i].x.v);
        }
    }
}

template <int M1>
__global__ void __launch_bounds__(256, 2) rt_spec_cols_kernel(RArgs<double> a) {
    constexpr int M = M1 * 4096;
    const int64_t li = blockIdx.x / (unsigned) M1;
    const RowSrc  rs{a.Trows + (a.item0 + li) * a.lambda, a.lambda, 2 * M};
    cols_forward<double, M1>(a, (int) (blockIdx.x % M1), a.Y + li * M,
                             [&](int j0, int n) { return point(sample(rs, j0 + n), sample(rs, j0 + n + M)); });
}

template <typename T, int M1>
__global__ void __launch_bounds__(256, rt_col_ctas<T>()) rt_cols_kernel(RArgs<T> a) {
    constexpr int M = M1 * 4096;
    const int     li = blockIdx.x / (unsigned) M1, part = blockIdx.x % (unsigned) M1;
    Tile<T>       tl;
    int           spec;
    if (!tile_of(a, a.item0 + li, tl, spec)) return;
    auto *Y = a.Y + (int64_t) li * M;
    if (tl.cnt == 2 * M)
        cols_forward<T, M1>(a, part, Y, [&](int j0, int n) { return point(sample_in(tl, j0, n), sample_in(tl, j0, n + M)); });
    else
        cols_forward<T, M1>(a, part, Y, [&](int j0, int n) { return point(sample(tl, j0 + n), sample(tl, j0 + n + M)); });
}
template <typename T, int M1>
__global__ void __launch_bounds__(256, rt_col_ctas<T>()) rt_cols_back_kernel(RArgs<T> a) {
    constexpr int M = M1 * 4096;
    const int     li = blockIdx.x / (unsigned) M1, part = blockIdx.x % (unsigned) M1;
    Tile<T>       tl;
    int           spec;
    if (!tile_of(a, a.item0 + li, tl, spec)) return;
    cols_back<T, M1>(a, part, a.Y + (int64_t) li * M, tl);
}
template <typename T>
__global__ void __launch_bounds__(256, rt_ctas<T>()) rt_rows_kernel(RArgs<T> a) {
    using G = typename LaneOf<T>::Tag;
    constexpr int L = 4096;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    REnt<G>  *s = reinterpret_cast<REnt<G> *>(smem_raw);
    const int li = blockIdx.x >> a.log_m1, part = blockIdx.x & ((1 << a.log_m1) - 1);
    Tile<T>   tl;
    int       spec;
    if (!tile_of(a, a.item0 + li, tl, spec)) return;
    REnt<G> *row = a.Y + (int64_t) blockIdx.x * L;
    CP<G>    u[16], z[16];
    row_forward<T, 16, false>(s, a.tw1, a.tw2, [&](int n) { return get_l2(row + n); }, u);
    row_product(u, a.H + (((int64_t) spec << a.log_m1) + part) * L + threadIdx.x * (16 / sizeof(T)), 256, z);
    row_back<T, 16, false>(s, a.tw1b, a.tw2, z, [&](int n, CP<G> y) { row[n] = REnt<G>{y.x, y.y}; });
}

// ------------------------------------------------------------------ host side
template <typename T> size_t rows_smem(int L) { return 2 * sizeof(T) * (size_t) rt_entries(L); }
// Items whose columns, rows and columns back are launched together, so that their scratch
// is read from L2 (126 MB) by the next kernel; what is written goes out to DRAM all the same (2^25
// samples, half bandwidth 2^14, FP32: 158 MB read and 373 written, samples and outputs 134 each).  Groups alternate between the context's
// stream and its side stream with a scratch half each: the last CTAs of one group's kernel
// and the next launch share the device with the other group's.  64 x 2^20 samples, half
// bandwidth 2^14, one stream and 64 MB -> two and 64 MB each: FP32 0.70 -> 0.645 ms, FP64 1.34
// -> 1.20 ms (halves of 24, 32, 48 MB: 0.68, 0.66, 0.64 and 1.24, 1.21, 1.24 ms); work that fits
// one half is cut in two from 2 x 16 MB on (8 x 2^20, 2^13, FP32: 99 -> 96 us), and less is one group (2^20
// samples, half bandwidth 2^13, FP64: 41.0 us in two groups, 34.4 in one; FP32, 18 MB in all: 42.3 and 37.6 us).
constexpr int64_t RT_HALF_BYTES = int64_t(64) << 20, RT_MIN_BYTES = int64_t(16) << 20;
struct Groups {
    int64_t n, per;  // how many, items in each but the last
};
constexpr int64_t half_items(int64_t item_bytes) { return std::max<int64_t>(1, RT_HALF_BYTES / item_bytes); }
// of `items` items with scratch for `cap` of them: all at once, in two halves, or (cap < items) in
// groups of half the scratch; n = 1 is one group on the context's stream
Groups groups_of(int64_t items, int64_t item_bytes, int64_t cap) {
    const int64_t half = std::min(half_items(item_bytes), items <= cap ? items : std::max<int64_t>(1, cap / 2));
    int64_t       n = (items + half - 1) / half;
    if (n == 1 && items > 1 && items * item_bytes >= 2 * RT_MIN_BYTES) n = 2;
    const int64_t per = (items + n - 1) / n;
    return Groups{(items + per - 1) / per, per};
}

template <typename T>
const void *one_fn(int L) {
    switch (L) {
        case 512: return (const void *) rt_one_kernel<T, 2>;
        case 1024: return (const void *) rt_one_kernel<T, 4>;
        case 2048: return (const void *) rt_one_kernel<T, 8>;
        case 4096: return (const void *) rt_one_kernel<T, 16>;
    }
    return nullptr;
}
template <typename T, bool BACK>
const void *cols_fn(int log_m1) {
    switch (log_m1) {
        case 1: return BACK ? (const void *) rt_cols_back_kernel<T, 2> : (const void *) rt_cols_kernel<T, 2>;
        case 2: return BACK ? (const void *) rt_cols_back_kernel<T, 4> : (const void *) rt_cols_kernel<T, 4>;
        case 3: return BACK ? (const void *) rt_cols_back_kernel<T, 8> : (const void *) rt_cols_kernel<T, 8>;
        case 4: return BACK ? (const void *) rt_cols_back_kernel<T, 16> : (const void *) rt_cols_kernel<T, 16>;
    }
    return nullptr;
}
const void *spec_rows_fn(int m1, int L) {
    if (m1 > 1) return (const void *) rt_spec_rows_kernel<16, false>;
    switch (L) {
        case 512: return (const void *) rt_spec_rows_kernel<2, true>;
        case 1024: return (const void *) rt_spec_rows_kernel<4, true>;
        case 2048: return (const void *) rt_spec_rows_kernel<8, true>;
        case 4096: return (const void *) rt_spec_rows_kernel<16, true>;
    }
    return nullptr;
}
const void *spec_cols_fn(int m1) {
    switch (m1) {
        case 2: return (const void *) rt_spec_cols_kernel<2>;
        case 4: return (const void *) rt_spec_cols_kernel<4>;
        case 8: return (const void *) rt_spec_cols_kernel<8>;
        case 16: return (const void *) rt_spec_cols_kernel<16>;
    }
    return nullptr;
}

inline void set2(float2 &o, double x, double y) { o = make_float2((float) x, (float) y); }
inline void set2(double2 &o, double x, double y) { o = make_double2(x, y); }

// tables of the transform in the order tw1, tw1b, tw2, wa, wb, one buffer
template <typename V2>
int build_tables(int m1, int L, DevBuf &buf, const V2 **tw1, const V2 **tw1b, const V2 **tw2, const V2 **wa,
                 const V2 **wb) {
    const int       R = L / 256, M = m1 * L;
    const int       B = sizeof(V2) == 8 ? L : 0;  // where tw1b starts: FP64 has one layout for both
    std::vector<V2> t(B + L + 256 + (m1 > 1 ? 128 * m1 : 0));
    double          re, im;
    for (int k = 0; k < R; k++)
        for (int q = 0; q < 256; q++) {
            // W_L^(q (k - 1/4)) = W_4L^(q (4k - 1)), exponents modulo 4L
            const int64_t e = m1 == 1 ? (int64_t) q * (4 * k - 1) : (int64_t) 4 * q * k;
            mdp_host_cexp((long double) ((e + 4LL * L) % (4LL * L)), 4.0L * L, &re, &im);
            set2(t[tw_at<V2>(k, q, 256)], re, im);
            set2(t[B + k * 256 + tw_at<V2>(q >> 4, q & 15, 16)], re, im);
        }
    for (int k = 0; k < 16; k++)
        for (int c = 0; c < 16; c++) {
            mdp_host_cexp(k * c, 256, &re, &im);
            set2(t[B + L + tw_at<V2>(k, c, 16)], re, im);
        }
    if (m1 > 1)
        for (int k = 0; k < m1; k++)
            for (int h = 0; h < 64; h++) {
                const int64_t den = 4LL * M, ea = 64LL * h * (4 * k - 1), eb = (int64_t) h * (4 * k - 1);
                mdp_host_cexp((long double) ((ea + den) % den), (long double) den, &re, &im);
                set2(t[B + L + 256 + 64 * k + h], re, im);
                mdp_host_cexp((long double) ((eb + den) % den), (long double) den, &re, &im);
                set2(t[B + L + 256 + 64 * m1 + 64 * k + h], re, im);
            }
    MDP_TRY(buf.alloc(sizeof(V2) * t.size()));
    MDP_CUDA(cudaMemcpy(buf.p, t.data(), sizeof(V2) * t.size(), cudaMemcpyHostToDevice));
    *tw1 = buf.as<V2>();
    *tw1b = *tw1 + B;
    *tw2 = *tw1b + L;
    *wa = *tw2 + 256;
    *wb = *wa + 64 * m1;
    return MDP_OK;
}

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
    // where each tile's window lies, in one 32-byte record (a chain of loads through the tile, its
    // block and the block's place would be on every CTA's path)
    {
        std::vector<mdp_rtile> tiles;
        const int64_t          E = P.fft_n - 2LL * (N->lambda - 1);
        for (int b = 0; b < N->nb; b++)
            for (int64_t o = 0; o < N->h_n[b]; o += E) {
                const int64_t w = o - (N->lambda - 1), lo = std::max<int64_t>(-w, 0);
                tiles.push_back(mdp_rtile{N->h_idv[b] + w, (int32_t) lo,
                                          (int32_t) (std::min<int64_t>(N->h_n[b] - w, P.fft_n) - lo),
                                          (int32_t) std::min<int64_t>(E, N->h_n[b] - o), N->h_spec.empty() ? 0 : N->h_spec[b],
                                          b, 0});
            }
        MDP_TRY(P.tile_start.alloc(sizeof(mdp_rtile) * std::max<size_t>(tiles.size(), 1)));
        if (!tiles.empty())
            MDP_CUDA(cudaMemcpy(P.tile_start.p, tiles.data(), sizeof(mdp_rtile) * tiles.size(), cudaMemcpyHostToDevice));
    }
    const V2 *p[5];
    MDP_TRY(build_tables<V2>(m1, L, P.ltw, &p[0], &p[1], &p[2], &p[3], &p[4]));
    if (m1 > 1) {
        // FP32 plans also run column batches of up to 8 columns
        const int64_t item_bytes = 2 * (int64_t) sizeof(T) * M;
        const int64_t items = std::max<int64_t>(1, P.n_tiles * (sizeof(T) == 4 ? 8 : 1));
        P.scratch_items = std::max<int64_t>(2, std::min(items, 2 * half_items(item_bytes)));
        MDP_TRY(P.scratch.alloc((size_t) (P.scratch_items * item_bytes)));
        MDP_CUDA(cudaFuncSetAttribute((const void *) rt_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) rows_smem<T>(L)));
    } else {
        MDP_CUDA(cudaFuncSetAttribute(one_fn<T>(L), cudaFuncAttributeMaxDynamicSharedMemorySize, (int) rows_smem<T>(L)));
    }
    const size_t nh = (size_t) std::max(N->n_spec, 1) * M;
    MDP_TRY(P.spectra.alloc(sizeof(T) * nh));
    if (!spectra) {
        MDP_CUDA(cudaMemset(P.spectra.p, 0, sizeof(T) * nh));
        return MDP_OK;
    }
    RArgs<double> a{};
    DevBuf        tab, rows, Y;
    MDP_TRY(build_tables<double2>(m1, L, tab, &a.tw1, &a.tw1b, &a.tw2, &a.wa, &a.wb));
    MDP_TRY(rows.alloc(sizeof(double) * N->h_Tuniq.size()));
    MDP_CUDA(cudaMemcpyAsync(rows.p, N->h_Tuniq.data(), sizeof(double) * N->h_Tuniq.size(), cudaMemcpyHostToDevice,
                             ctx->stream));
    const int64_t per = m1 > 1 ? std::min<int64_t>(N->n_spec, 64) : N->n_spec;
    if (m1 > 1) MDP_TRY(Y.alloc(16 * (size_t) per * M));
    a.Trows = rows.as<double>();
    a.lambda = N->lambda;
    a.log_m1 = P.log_m1;
    a.Y = Y.as<REnt<mono64>>();
    if (sizeof(T) == 4) a.H32 = P.spectra.as<float>();
    else a.H64 = P.spectra.as<double>();
    const void *fs = spec_rows_fn(m1, L);
    MDP_CUDA(cudaFuncSetAttribute(fs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) rows_smem<double>(L)));
    for (int64_t i = 0; i < N->n_spec; i += per) {
        const int64_t n = std::min<int64_t>(per, N->n_spec - i);
        a.item0 = i;
        void *args[] = {&a};
        if (m1 > 1) {
            MDP_CUDA(cudaLaunchKernel(spec_cols_fn(m1), dim3((unsigned) (n * m1)), dim3(256), args, 0, ctx->stream));
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
    a.tiles = P.tile_start.as<mdp_rtile>();
    a.H = P.spectra.as<T>();
    a.tw1 = P.ltw.as<V2>();
    a.tw1b = a.tw1 + (sizeof(V2) == 8 ? L : 0);
    a.tw2 = a.tw1b + L;
    a.wa = a.tw2 + 256;
    a.wb = a.wa + 64 * m1;
    a.means = d_means;
    a.Y = P.scratch.as<REnt<typename LaneOf<T>::Tag>>();
    a.n_tiles = P.n_tiles;
    a.col_stride = col_stride;
    a.active = d_active;
    a.lambda = N->lambda;
    a.nb = N->nb;
    a.log_m1 = P.log_m1;
    const int64_t items = P.n_tiles * ncols;
    if (items << P.log_m1 > 0x7fffffffLL) return MDP_EUNSUPPORTED;
    void *args[] = {&a};
    // Chained to the kernel before, but for the first launches of two streams; FP64 groups on two
    // streams are not: a waiting CTA takes one of an SM's two places from the other stream's group
    // (64 x 2^20 samples, half bandwidth 2^14: 1.206 against 1.194 ms; FP32, of four places, 0.647 ->
    // 0.620 ms, and one group 140 -> 129 us for 24 ragged blocks).
    auto launch = [&](const void *fn, dim3 grid, int nt, size_t smem, cudaStream_t stream, bool chain) -> int {
        cudaLaunchAttribute attr;
        cudaLaunchConfig_t  cfg = chained_config(&attr, stream, grid, nt, smem);
        if (!chain) cfg.numAttrs = 0;
        MDP_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
        MDP_CHECK_LAUNCH(ctx);
        return MDP_OK;
    };
    if (m1 == 1) return launch(one_fn<T>(L), dim3((unsigned) items), L / 16, rows_smem<T>(L), ctx->stream, true);
    const Groups g = groups_of(items, 2 * (int64_t) sizeof(T) * M, P.scratch_items);
    cudaStream_t st[2] = {ctx->stream, ctx->stream};
    if (g.n > 1) {
        MDP_TRY(mdp_side_fork(ctx));
        st[1] = ctx->side;
    }
    auto      *Y = a.Y;
    const bool chain = sizeof(T) == 4 || g.n == 1;
    for (int64_t k = 0; k < g.n; k++) {
        const int64_t i = k * g.per;
        const dim3    grid((unsigned) (std::min(g.per, items - i) * m1));
        a.item0 = i;
        a.Y = Y + (k & 1) * g.per * M;
        MDP_TRY(launch(cols_fn<T, false>(P.log_m1), grid, 256, 0, st[k & 1], g.n == 1 || (chain && k > 1)));
        MDP_TRY(launch((const void *) rt_rows_kernel<T>, grid, 256, rows_smem<T>(L), st[k & 1], chain));
        MDP_TRY(launch(cols_fn<T, true>(P.log_m1), grid, 256, 0, st[k & 1], chain));
    }
    if (g.n > 1) MDP_TRY(mdp_side_join(ctx));
    return MDP_OK;
}

template int rtile_build<float>(mdp_context *, mdp_noise *, mdp_tile_plan &, bool);
template int rtile_build<double>(mdp_context *, mdp_noise *, mdp_tile_plan &, bool);
template int rtile_launch<float>(mdp_context *, const mdp_noise *, const mdp_tile_plan &, const float *, float *,
                                 const double *, int, int64_t, const int *);
template int rtile_launch<double>(mdp_context *, const mdp_noise *, const mdp_tile_plan &, const double *, double *,
                                  const double *, int, int64_t, const int *);
