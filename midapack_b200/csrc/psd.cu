// Periodograms of many stationary intervals at once: scipy.signal.welch(x, fs,
// window='hann', nperseg=n, detrend='linear') of one segment per block, the first
// step of MAPPRAISER's noise2invtt (mappraiser/python/TOAST_interface/utils.py:531).
//
// Per block of n samples: least-squares line removed, periodic Hann window,
// |X_k|^2 / (fs sum w^2), doubled except DC and Nyquist.  X is a transform of L = n1 x
// 4096 points as columns (n1 points over j1 of j = 4096 j1 + j2, times W_L^(j2 k1)) and
// rows; a block whose length is not a power of two goes through Bluestein's chirp
// convolution, of which only the bins k <= n/2 are wanted, so that L >= n + n/2 is
// enough (the wrapped part of the convolution lies beyond them).
//
// Blocks with the same L share the launches, whatever their lengths, in groups whose
// work arrays stay in L2: (1) columns of the samples (detrended, windowed and chirped on
// load) and of the group's chirp filters, (2) rows of the filters, (3) rows of the
// samples, times the filter's row, and back, (4) columns back, storing the densities.
// Every CTA transforms 4096 points by radix-16 passes in registers, 256 threads.
//
// Before, each run of equal lengths went through on its own: four passes for two filters
// (one of them the inverse transform's, unused), radix-2 stages with a barrier each, and
// the launches of a 2^19-point transform on 128 CTAs.  32 blocks of 100002 to 200003
// samples: 9.0 ms, 13-17 ms with the allocations between calls; now 0.72 ms, bound by the
// CTAs' load, exchange and store phases at two CTAs an SM.
#include <algorithm>
#include <cmath>
#include <vector>

#include "lanes.cuh"
#include "mdp_internal.cuh"

namespace {

using C1 = CP<mono64>;
constexpr int     kRow = 4096;
constexpr int     kT = 256;
constexpr int64_t kGroupBytes = int64_t(96) << 20;

struct PsdBlock {
    int64_t at;      // first sample
    int64_t out;     // first density
    int     n, filt; // samples; chirp filter of the group (-1: L = n, none)
    double  inv_stt, inv_stt_lo, scale;  // 1 / sum (t - (n-1)/2)^2 in two parts
};

struct PsdArgs {
    const double   *x;
    double         *psd;
    const PsdBlock *blk;    // [cnt]
    const int      *fn;     // [nfilt] lengths of the filters
    const double2  *tw1;    // [16][256] W_4096^(q k)
    const double2  *tw2;    // [16][16]  W_256^(c k)
    const double2  *tw4k;   // [4096]    W_4096^e
    const double4  *line;   // [cnt] least-squares line: mean and slope in two parts each
    double2        *buf;    // [cnt + nfilt][n1][4096]
    int             cnt, nfilt, n1;
};

__host__ __device__ constexpr int pp(int p) { return p + (p >> 4); }  // padded shared-memory position
constexpr int kSmem = 16 * (kRow + kRow / 16);

__device__ __forceinline__ C1 mk(double x, double y) { return {Pr<mono64>{x}, Pr<mono64>{y}}; }
__device__ __forceinline__ C1 ld(const double2 *p) {
    const double2 v = *p;
    return mk(v.x, v.y);
}
__device__ __forceinline__ double2 st(C1 v) { return make_double2(v.x.v, v.y.v); }
__device__ __forceinline__ C1 tw(C1 v, double2 w) {
    return {Pr<mono64>{fma(-v.y.v, w.y, v.x.v * w.x)}, Pr<mono64>{fma(v.y.v, w.x, v.x.v * w.y)}};
}
__device__ __forceinline__ C1 swp(C1 v) { return {v.y, v.x}; }
__device__ __forceinline__ double2 expi(double turns_pi, double sign) {
    double s, c;
    sincospi(turns_pi, &s, &c);
    return make_double2(c, sign * s);
}
// A length and its reciprocal: the angles pi a / n below are at most a quarter of a turn, so that the rounding
// of the reciprocal and of a product with it moves them by 2^-54 of a turn at most, and no quotient is formed.  (With
// a division each and a 64-bit modulo the columns of 12 blocks and their filters, L = 2^18, took 39 M warp
// instructions and 86 us, without 34 M and 74.)
struct Recip {
    double n, inv;
};
// exp(sign i pi m^2 / n): m^2 < 2^48 less the nearest multiple k of n/2, exactly (multiples of 1/2 below
// 2^53), so that the angle is at most an eighth of a turn and its rounding as much smaller; then k quarter turns.
// Amplitudes of 174763 white samples against extended precision: 3.87e-16 with angles of up to a turn, 3.52e-16
// with these and the window's within a quarter turn (100003 samples 3.26 and 2.82).
__device__ __forceinline__ double2 chirp1(int m, const Recip &n, double sign) {
    const double  mm = (double) m * (double) m, k = rint(mm * (2.0 * n.inv));
    const double2 w = expi(fma(-k, 0.5 * n.n, mm) * n.inv, 1.0);
    const int     q = (int) k;
    const double  c = q & 1 ? w.y : w.x, s = q & 1 ? w.x : w.y;
    return make_double2((q + 1) & 2 ? -c : c, sign * (q & 2 ? -s : s));
}

__global__ void psd_tables_kernel(double2 *tw1, double2 *tw2, double2 *tw4k) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;  // < 4096
    tw1[e] = expi((double) ((e >> 8) * (e & 255)) / 2048.0, -1.0);
    if (e < 256) tw2[e] = expi((double) ((e >> 4) * (e & 15)) / 128.0, -1.0);
    tw4k[e] = expi((double) e / 2048.0, -1.0);
}

// A number as the unevaluated sum of two doubles, for the least-squares line of a block: the same error in
// the line at every sample falls into the lowest bins, which hold most of 1/f data (12909 samples against extended
// precision, the line's part alone: plain sums, rounded mean and slope 3.4e-16 of a block's norm on average and up
// to 3.0e-15, in two parts 3e-17).  The roundings of single samples, and of the sums of a warp's few
// hundred, average out: those stay plain.
struct Two {
    double h, l;
};
__device__ __forceinline__ Two operator+(Two a, Two b) {  // two-sum: Knuth, The Art of Computer Programming, vol. 2
    const double s = a.h + b.h, t = s - a.h;
    return {s, (a.h - (s - t)) + (b.h - t) + (a.l + b.l)};
}
__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ Two warp_sum(Two v) {
    for (int o = 16; o > 0; o >>= 1)
        v = v + Two{__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)};
    return v;
}

// sums of x and (t - (n-1)/2) x over each block: partials, chunk by chunk
__global__ void __launch_bounds__(kT) psd_sums_kernel(PsdArgs a, Two *part) {
    const PsdBlock b = a.blk[blockIdx.y];
    const double  *x = a.x + b.at;
    const double   c = 0.5 * (double) (b.n - 1);
    double         s0 = 0.0, s1 = 0.0;
    for (int t = blockIdx.x * kT + threadIdx.x; t < b.n; t += gridDim.x * kT) {
        const double v = x[t];
        s0 += v;
        s1 += ((double) t - c) * v;
    }
    __shared__ double sh[2][kT / 32];
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = s0;
        sh[1][threadIdx.x >> 5] = s1;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        Two v{0.0, 0.0};
        for (int w = 0; w < kT / 32; w++) v = v + Two{sh[threadIdx.x][w], 0.0};
        part[((int64_t) blockIdx.y * 2 + threadIdx.x) * gridDim.x + blockIdx.x] = v;
    }
}
// mean and slope of each block, a warp a block
__global__ void __launch_bounds__(kT) psd_line_kernel(PsdArgs a, const Two *part, int chunks, double4 *line) {
    const int i = (blockIdx.x * kT + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= a.cnt) return;
    Two s[2];
    for (int q = 0; q < 2; q++) {
        s[q] = Two{0.0, 0.0};
        for (int c = lane; c < chunks; c += 32) s[q] = s[q] + part[((int64_t) i * 2 + q) * chunks + c];
        s[q] = warp_sum(s[q]);
    }
    if (lane != 0) return;
    const PsdBlock b = a.blk[i];
    const double   n = (double) b.n, m = s[0].h / n, k = s[1].h * b.inv_stt;
    line[i] = make_double4(m, (fma(-m, n, s[0].h) + s[0].l) / n, k,
                           fma(s[1].h, b.inv_stt, -k) + (s[1].h * b.inv_stt_lo + s[1].l * b.inv_stt));
}

// point j of a block's transform input: detrended, windowed, chirped sample; or of a filter
struct Load {
    const double *x;
    double4       line;
    double        c;
    Recip         rn;       // of n
    int           n, kind;  // 0: samples, 1: chirped samples, 2: filter
    int           L;
};
__device__ __forceinline__ C1 point(const Load &l, int j) {
    if (l.kind == 2) {
        // exp(i pi m^2 / n) for -n < m <= n/2, negative m at L + m
        const int m = j <= l.n / 2 ? j : (j > l.L - l.n ? l.L - j : -1);
        if (m < 0) return mk(0.0, 0.0);
        const double2 w = chirp1(m, l.rn, 1.0);
        return mk(w.x, w.y);
    }
    if (j >= l.n) return mk(0.0, 0.0);
    // (1 - cos(2 pi j / n)) / 2, the angle within a quarter turn of 0 or 1/2 (exact for a power of two)
    const int    h = 2 * min(j, l.n - j);
    const bool   far = 2 * h > l.n;
    const double w = fma(far ? 0.5 : -0.5, cospi((double) (far ? l.n - h : h) * l.rn.inv), 0.5);
    const double t = (double) j - l.c;
    const double v = (fma(-l.line.z, t, __ldg(l.x + j) - l.line.x) - fma(l.line.w, t, l.line.y)) * w;
    if (l.kind == 0) return mk(v, 0.0);
    const double2 ch = chirp1(j, l.rn, -1.0);
    return mk(v * ch.x, v * ch.y);
}

// density of bin k from the squared modulus of its transform value
__device__ __forceinline__ void store_psd(const PsdArgs &a, const PsdBlock &b, int64_t k, C1 v) {
    if (k > b.n / 2) return;
    double p = (v.x.v * v.x.v + v.y.v * v.y.v) * b.scale;
    if (k > 0 && !((b.n & 1) == 0 && k == b.n / 2)) p *= 2.0;
    a.psd[b.out + k] = p;
}

// n1 = 2^LOG1 point transforms of 4096/n1 adjacent columns, natural order in and out:
// passes of radix R = 2^((LOG1-1)%4+1), then 16 (LOG1 > 4), then 16 (LOG1 > 8).
// Forward: inputs from point(), outputs times W_L^(j2 k1) to buf.  Back (real and imaginary
// parts exchanged): inputs from buf times W_L^(j2 k1), densities out.
template <int LOG1, bool INV>
__global__ void __launch_bounds__(kT, 2) psd_cols_kernel(PsdArgs a) {
    constexpr int N1 = 1 << LOG1, LC = 12 - LOG1, C = 1 << LC;
    constexpr int NP = (LOG1 + 3) / 4, LR = LOG1 - 4 * (NP - 1), R = 1 << LR, S = 16 / R, REST = N1 / R;
    extern __shared__ __align__(16) double2 s[];
    const int t = threadIdx.x, item = blockIdx.y, c0 = (int) blockIdx.x << LC;
    double2  *Y = a.buf + (int64_t) item * N1 * kRow;
    Load      l{};
    if (!INV) {
        l.L = N1 * kRow;
        if (item < a.cnt) {
            const PsdBlock b = a.blk[item];
            l.x = a.x + b.at;
            l.n = b.n;
            l.kind = b.filt < 0 ? 0 : 1;
            l.line = a.line[item];
            l.c = 0.5 * (double) (b.n - 1);
        } else {
            l.n = a.fn[item - a.cnt];
            l.kind = 2;
        }
        l.rn = Recip{(double) l.n, 1.0 / (double) l.n};
    }
    auto twl = [&](int k1, int c) {  // W_L^(j2 k1), j2 = c0 + c, j2 k1 < L
        return expi((double) ((c0 + c) * k1) / (2048.0 * N1), -1.0);
    };
    auto load = [&](int i, int c) -> C1 {
        if constexpr (INV) return tw(ld(Y + (int64_t) i * kRow + c0 + c), twl(i, c));
        else return point(l, i * kRow + c0 + c);
    };
    auto store = [&](int k, int c, C1 v) {
        if constexpr (INV) store_psd(a, a.blk[item], (int64_t) k * kRow + c0 + c, v);
        else Y[(int64_t) k * kRow + c0 + c] = st(tw(v, twl(k, c)));
    };
    // pass 1: S sets of R points a thread, set (q, c)
#pragma unroll
    for (int j = 0; j < S; j++) {
        const int id = t + kT * j, c = id & (C - 1), q = id >> LC;
        C1        v[R];
#pragma unroll
        for (int i = 0; i < R; i++) v[i] = load(i * REST + q, c);
        dif_reg<mono64, R>(v);
#pragma unroll
        for (int k = 0; k < R; k++) {
            C1 w = v[rev_bits_c(k, LR)];
            if constexpr (NP == 1) {
                store(k, c, w);
            } else {
                if (k > 0) w = tw(w, __ldg(a.tw4k + ((q * k) << (12 - LOG1))));
                s[pp((k * REST + q) * C + c)] = st(w);
            }
        }
    }
    if constexpr (NP > 1) {
        const int c = t & (C - 1), h = t >> LC;
        C1        v[16];
        __syncthreads();
        if constexpr (NP == 3) {  // h = (k_a, c2)
            const int c2 = h & 15, ka = h >> 4;
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = ld(s + pp((ka * 256 + 16 * i + c2) * C + c));
            dif_reg<mono64, 16>(v);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                C1 w = v[rev_bits_c(k, 4)];
                if (k > 0) w = tw(w, __ldg(a.tw2 + k * 16 + c2));
                s[pp((ka * 256 + 16 * k + c2) * C + c)] = st(w);
            }
            __syncthreads();
        }
        // last pass: h = k_a (two passes) or (k_a, k_b)
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = ld(s + pp((h * 16 + i) * C + c));
        dif_reg<mono64, 16>(v);
        const int k0 = NP == 2 ? h : (h >> 4) + R * (h & 15);
#pragma unroll
        for (int k = 0; k < 16; k++) store(k0 + (N1 / 16) * k, c, v[rev_bits_c(k, 4)]);
    }
}

// 4096-point rows: FILT, a filter's row, left in the register order of the product;
// BLUE, a row of samples, times its filter's row, and back (parts exchanged); POW2, a
// row of samples, densities out.
enum { FILT, BLUE, POW2 };
template <int MODE>
__global__ void __launch_bounds__(kT, 2) psd_rows_kernel(PsdArgs a) {
    extern __shared__ __align__(16) double2 s[];
    const int      t = threadIdx.x, c = t & 15, h = t >> 4, k1 = blockIdx.x;
    const int      item = MODE == FILT ? a.cnt + blockIdx.y : blockIdx.y;
    const PsdBlock b = MODE == FILT ? PsdBlock{} : a.blk[item];
    double2       *Y = a.buf + ((int64_t) item * a.n1 + k1) * kRow;
    C1             u[16], z[16];
#pragma unroll
    for (int i = 0; i < 16; i++) u[i] = ld(Y + 256 * i + t);
    dif_reg<mono64, 16>(u);
#pragma unroll
    for (int k = 0; k < 16; k++) {
        C1 w = u[rev_bits_c(k, 4)];
        if (k > 0) w = tw(w, __ldg(a.tw1 + k * 256 + t));
        s[pp(k * 256 + t)] = st(w);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; i++) u[i] = ld(s + pp(h * 256 + 16 * i + c));
    dif_reg<mono64, 16>(u);
#pragma unroll
    for (int k = 0; k < 16; k++) {
        C1 w = u[rev_bits_c(k, 4)];
        if (k > 0) w = tw(w, __ldg(a.tw2 + k * 16 + c));
        s[pp(h * 256 + 16 * k + c)] = st(w);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; i++) u[i] = ld(s + pp(h * 256 + 16 * c + i));
    dif_reg<mono64, 16>(u);
    if constexpr (MODE == FILT) {
#pragma unroll
        for (int k = 0; k < 16; k++) Y[k * 256 + t] = st(u[rev_bits_c(k, 4)]);
    } else if constexpr (MODE == POW2) {  // bin k1 + n1 k2, k2 = h + 16 c + 256 k
#pragma unroll
        for (int k = 0; k < 16; k++)
            store_psd(a, b, k1 + (int64_t) a.n1 * (h + 16 * c + 256 * k), u[rev_bits_c(k, 4)]);
    } else {
        const double2 *F = a.buf + ((int64_t) (a.cnt + b.filt) * a.n1 + k1) * kRow;
#pragma unroll
        for (int k = 0; k < 16; k++) z[k] = swp(tw(u[rev_bits_c(k, 4)], __ldg(F + k * 256 + t)));
        dif_reg<mono64, 16>(z);
#pragma unroll
        for (int i = 0; i < 16; i++) {
            C1 w = z[rev_bits_c(i, 4)];
            if (i > 0) w = tw(w, __ldg(a.tw2 + i * 16 + c));
            s[pp(h * 256 + 16 * c + i)] = st(w);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; k++) z[k] = ld(s + pp(h * 256 + 16 * k + c));
        dif_reg<mono64, 16>(z);
#pragma unroll
        for (int i = 0; i < 16; i++) s[pp(h * 256 + 16 * i + c)] = st(tw(z[rev_bits_c(i, 4)], __ldg(a.tw1 + h * 256 + 16 * i + c)));
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; k++) z[k] = ld(s + pp(k * 256 + t));
        dif_reg<mono64, 16>(z);
#pragma unroll
        for (int i = 0; i < 16; i++) Y[256 * i + t] = st(z[rev_bits_c(i, 4)]);
    }
}

template <bool INV>
const void *cols_kernel(int log1) {
    switch (log1) {
        case 1: return (const void *) psd_cols_kernel<1, INV>;
        case 2: return (const void *) psd_cols_kernel<2, INV>;
        case 3: return (const void *) psd_cols_kernel<3, INV>;
        case 4: return (const void *) psd_cols_kernel<4, INV>;
        case 5: return (const void *) psd_cols_kernel<5, INV>;
        case 6: return (const void *) psd_cols_kernel<6, INV>;
        case 7: return (const void *) psd_cols_kernel<7, INV>;
        case 8: return (const void *) psd_cols_kernel<8, INV>;
        case 9: return (const void *) psd_cols_kernel<9, INV>;
        case 10: return (const void *) psd_cols_kernel<10, INV>;
        case 11: return (const void *) psd_cols_kernel<11, INV>;
        case 12: return (const void *) psd_cols_kernel<12, INV>;
    }
    return nullptr;
}

int launch(mdp_context *ctx, const void *fn, dim3 grid, size_t smem, const PsdArgs &a) {
    PsdArgs b = a;
    void   *args[] = {&b};
    if (smem) MDP_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    MDP_CUDA(cudaLaunchKernel(fn, grid, dim3(kT), args, smem, ctx->stream));
    MDP_CHECK_LAUNCH(ctx);
    return MDP_OK;
}

bool pow2(int64_t n) { return (n & (n - 1)) == 0; }

// log2 of the transform of a block here: n for a power of two, else at least n + n/2
int log_len(int64_t n) {
    const int64_t need = pow2(n) ? n : n + n / 2;
    int           l = 0;
    while ((int64_t(1) << l) < need) l++;
    return l;
}

}  // namespace

// Blocks of 8192 samples and more, and shorter ones whose chirp convolution takes 8192
// points: the transforms of one CTA below that stay with the single-pass kernels (noise.cu).
bool mdp_psd_takes(int64_t n) { return log_len(n) >= 13; }

// densities of the blocks idx (lengths n, first sample at, first density out)
int mdp_psd_blocks(mdp_context *ctx, const std::vector<int> &idx, const int32_t *n, const std::vector<int64_t> &at,
                   const std::vector<int64_t> &out, const double *d_x, double fsamp, double *d_psd) {
    std::vector<int> order(idx);
    std::stable_sort(order.begin(), order.end(), [&](int p, int q) {
        const int lp = log_len(n[p]), lq = log_len(n[q]);
        return lp != lq ? lp < lq : pow2(n[p]) != pow2(n[q]) ? pow2(n[p]) : n[p] < n[q];
    });
    // groups: one transform length, one kind, at most kGroupBytes of work arrays (or one block)
    struct Group {
        int first, cnt, ffirst, nf, ll, chunks;
    };
    std::vector<Group>    groups;
    std::vector<PsdBlock> blk;
    std::vector<int>      fn;
    size_t                work = 0, parts = 0;
    for (int b : order) {
        const int     ll = log_len(n[b]);
        const bool    p2 = pow2(n[b]);
        const int64_t L = int64_t(1) << ll;
        bool          joins = !groups.empty() && groups.back().ll == ll && (blk.back().filt < 0) == p2;
        if (joins) {
            const Group &g = groups.back();
            joins = g.cnt < 4096 && (int64_t) (g.cnt + g.nf + (p2 || fn.back() == n[b] ? 1 : 2)) * L * 16 <= kGroupBytes;
        }
        if (!joins) groups.push_back(Group{(int) blk.size(), 0, (int) fn.size(), 0, ll, 1});
        Group &g = groups.back();
        if (!p2 && (g.nf == 0 || fn.back() != n[b])) {
            fn.push_back(n[b]);
            g.nf++;
        }
        // constants of the block, each rounded once
        const long double dn = n[b], il = 1.0L / (long double) L, is = 12.0L / (dn * (dn * dn - 1.0L));
        blk.push_back(PsdBlock{at[b], out[b], n[b], p2 ? -1 : g.nf - 1, (double) is, (double) (is - (long double) (double) is),
                               (double) (8.0L * (p2 ? 1.0L : il * il) / (3.0L * (long double) fsamp * dn))});
        g.cnt++;
        g.chunks = std::max<int>(g.chunks, (int) std::min<int64_t>(((int64_t) n[b] + 4095) / 4096, 256));
        work = std::max(work, 16 * (size_t) (g.cnt + g.nf) * (size_t) L);
        parts = std::max(parts, 2 * (size_t) g.cnt * g.chunks);
    }
    // one buffer: tables, descriptors, the sums of a group and its work arrays
    auto   up = [](size_t b) { return (b + 255) & ~size_t(255); };
    size_t o_blk = up(16 * (2 * 4096 + 256)), o_fn = o_blk + up(sizeof(PsdBlock) * blk.size()), o_part = o_fn + up(4 * fn.size()),
           o_line = o_part + up(sizeof(Two) * parts), o_buf = o_line + up(sizeof(double4) * blk.size());
    MDP_TRY(ctx->scratch.alloc(o_buf + work));
    char    *base = ctx->scratch.as<char>();
    double2 *tab = (double2 *) base;
    Two     *part = (Two *) (base + o_part);
    double4 *line = (double4 *) (base + o_line);
    psd_tables_kernel<<<16, 256, 0, ctx->stream>>>(tab, tab + 8192, tab + 4096);
    MDP_CHECK_LAUNCH(ctx);
    MDP_CUDA(cudaMemcpyAsync(base + o_blk, blk.data(), sizeof(PsdBlock) * blk.size(), cudaMemcpyHostToDevice, ctx->stream));
    if (!fn.empty())
        MDP_CUDA(cudaMemcpyAsync(base + o_fn, fn.data(), 4 * fn.size(), cudaMemcpyHostToDevice, ctx->stream));
    for (const Group &g : groups) {
        PsdArgs a{};
        a.x = d_x;
        a.psd = d_psd;
        a.blk = (const PsdBlock *) (base + o_blk) + g.first;
        a.fn = (const int *) (base + o_fn) + g.ffirst;
        a.tw1 = tab;
        a.tw4k = tab + 4096;
        a.tw2 = tab + 8192;
        a.line = line;
        a.buf = (double2 *) (base + o_buf);
        a.cnt = g.cnt;
        a.nfilt = g.nf;
        a.n1 = 1 << (g.ll - 12);
        psd_sums_kernel<<<dim3(g.chunks, g.cnt), kT, 0, ctx->stream>>>(a, part);
        MDP_CHECK_LAUNCH(ctx);
        psd_line_kernel<<<(g.cnt * 32 + kT - 1) / kT, kT, 0, ctx->stream>>>(a, part, g.chunks, line);
        MDP_CHECK_LAUNCH(ctx);
        const size_t csm = g.ll - 12 > 4 ? kSmem : 0;
        MDP_TRY(launch(ctx, cols_kernel<false>(g.ll - 12), dim3(a.n1, g.cnt + g.nf), csm, a));
        if (g.nf == 0) {
            MDP_TRY(launch(ctx, (const void *) psd_rows_kernel<POW2>, dim3(a.n1, g.cnt), kSmem, a));
        } else {
            MDP_TRY(launch(ctx, (const void *) psd_rows_kernel<FILT>, dim3(a.n1, g.nf), kSmem, a));
            MDP_TRY(launch(ctx, (const void *) psd_rows_kernel<BLUE>, dim3(a.n1, g.cnt), kSmem, a));
            MDP_TRY(launch(ctx, cols_kernel<true>(g.ll - 12), dim3(a.n1, g.cnt), csm, a));
        }
    }
    return MDP_OK;
}
