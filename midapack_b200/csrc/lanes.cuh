// Complex arithmetic on register lanes, and the small in-register transforms
// built on it, shared by the inverse-noise tile kernels.
//
// Pr<T> is one real value on every lane of a register set: Pr<float> is two
// FP32 lanes in one 64-bit register pair (Blackwell's paired add/sub/mul/fma
// .f32x2, one instruction for both lanes, each rounded as the scalar one),
// Pr<double> two FP64 lanes, Pr<mono32> and Pr<mono64> a single lane.  CP<T> is a complex
// value per lane, real and imaginary parts in separate Pr.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

namespace {

// ------------------------------------------------------------------ lane pairs
template <typename T> struct Pr;
template <> struct Pr<float> {
    unsigned long long v;
};
template <> struct Pr<double> {
    double a, b;
};
struct mono64 {};
template <> struct Pr<mono64> {
    double v;
};
struct mono32 {};
template <> struct Pr<mono32> {
    float v;
};

__device__ __forceinline__ Pr<float> pmk(float a, float b) {
    Pr<float> r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float plo(Pr<float> p) {
    float a;
    asm("{.reg .f32 t; mov.b64 {%0, t}, %1;}" : "=f"(a) : "l"(p.v));
    return a;
}
__device__ __forceinline__ float phi(Pr<float> p) {
    float b;
    asm("{.reg .f32 t; mov.b64 {t, %0}, %1;}" : "=f"(b) : "l"(p.v));
    return b;
}
__device__ __forceinline__ Pr<float> padd(Pr<float> a, Pr<float> b) {
    Pr<float> r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Pr<float> psub(Pr<float> a, Pr<float> b) {
    Pr<float> r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Pr<float> pmul(Pr<float> a, Pr<float> b) {
    Pr<float> r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Pr<float> pfma(Pr<float> a, Pr<float> b, Pr<float> c) {  // a*b + c
    Pr<float> r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ Pr<float> pswap(Pr<float> p) { return pmk(phi(p), plo(p)); }

__device__ __forceinline__ Pr<double> pmk(double a, double b) { return Pr<double>{a, b}; }
__device__ __forceinline__ double plo(Pr<double> p) { return p.a; }
__device__ __forceinline__ double phi(Pr<double> p) { return p.b; }
__device__ __forceinline__ Pr<double> padd(Pr<double> x, Pr<double> y) { return {x.a + y.a, x.b + y.b}; }
__device__ __forceinline__ Pr<double> psub(Pr<double> x, Pr<double> y) { return {x.a - y.a, x.b - y.b}; }
__device__ __forceinline__ Pr<double> pmul(Pr<double> x, Pr<double> y) { return {x.a * y.a, x.b * y.b}; }
__device__ __forceinline__ Pr<double> pfma(Pr<double> x, Pr<double> y, Pr<double> z) {
    return {fma(x.a, y.a, z.a), fma(x.b, y.b, z.b)};
}
__device__ __forceinline__ Pr<double> pswap(Pr<double> p) { return {p.b, p.a}; }

__device__ __forceinline__ Pr<mono64> padd(Pr<mono64> x, Pr<mono64> y) { return {x.v + y.v}; }
__device__ __forceinline__ Pr<mono64> psub(Pr<mono64> x, Pr<mono64> y) { return {x.v - y.v}; }
__device__ __forceinline__ Pr<mono64> pmul(Pr<mono64> x, Pr<mono64> y) { return {x.v * y.v}; }
__device__ __forceinline__ Pr<mono64> pfma(Pr<mono64> x, Pr<mono64> y, Pr<mono64> z) { return {fma(x.v, y.v, z.v)}; }

__device__ __forceinline__ Pr<mono32> padd(Pr<mono32> x, Pr<mono32> y) { return {x.v + y.v}; }
__device__ __forceinline__ Pr<mono32> psub(Pr<mono32> x, Pr<mono32> y) { return {x.v - y.v}; }
__device__ __forceinline__ Pr<mono32> pmul(Pr<mono32> x, Pr<mono32> y) { return {x.v * y.v}; }
__device__ __forceinline__ Pr<mono32> pfma(Pr<mono32> x, Pr<mono32> y, Pr<mono32> z) { return {fmaf(x.v, y.v, z.v)}; }

template <typename T> __device__ __forceinline__ Pr<T> pdup(T s) { return pmk(s, s); }
// a compile-time constant on both lanes: plain integer bits for FP32 (the
// compiler may rematerialise it at each use instead of keeping it live)
template <typename T> __device__ __forceinline__ Pr<T> pcst(double v);
template <> __device__ __forceinline__ Pr<float> pcst<float>(double v) {
    const unsigned long long u = __float_as_uint((float) v);
    return Pr<float>{(u << 32) | u};
}
template <> __device__ __forceinline__ Pr<double> pcst<double>(double v) { return Pr<double>{v, v}; }
template <> __device__ __forceinline__ Pr<mono64> pcst<mono64>(double v) { return Pr<mono64>{v}; }
template <> __device__ __forceinline__ Pr<mono32> pcst<mono32>(double v) { return Pr<mono32>{(float) v}; }

// complex values on both lanes: x = real parts (lane A, lane B), y = imaginary parts
template <typename T> struct CP {
    Pr<T> x, y;
};

template <typename T> __device__ __forceinline__ CP<T> cpadd(CP<T> a, CP<T> b) { return {padd(a.x, b.x), padd(a.y, b.y)}; }
template <typename T> __device__ __forceinline__ CP<T> cpsub(CP<T> a, CP<T> b) { return {psub(a.x, b.x), psub(a.y, b.y)}; }
// one FP32 lane: the two components in one paired instruction
template <> __device__ __forceinline__ CP<mono32> cpadd<mono32>(CP<mono32> a, CP<mono32> b) {
    const Pr<float> r = padd(pmk(a.x.v, a.y.v), pmk(b.x.v, b.y.v));
    return {Pr<mono32>{plo(r)}, Pr<mono32>{phi(r)}};
}
template <> __device__ __forceinline__ CP<mono32> cpsub<mono32>(CP<mono32> a, CP<mono32> b) {
    const Pr<float> r = psub(pmk(a.x.v, a.y.v), pmk(b.x.v, b.y.v));
    return {Pr<mono32>{plo(r)}, Pr<mono32>{phi(r)}};
}
// a * w
template <typename T> __device__ __forceinline__ CP<T> cpmul(CP<T> a, CP<T> w) {
    return {psub(pmul(a.x, w.x), pmul(a.y, w.y)), pfma(a.x, w.y, pmul(a.y, w.x))};
}
// a * conj(w)
template <typename T> __device__ __forceinline__ CP<T> cpmulc(CP<T> a, CP<T> w) {
    return {pfma(a.x, w.x, pmul(a.y, w.y)), psub(pmul(a.y, w.x), pmul(a.x, w.y))};
}

// ------------------------------------------------------------------ W_16^m, m < 8
// cos and -sin of 2 pi m / 16 (exact decimal expansions rounded by the compiler)
__host__ __device__ constexpr double w16c(int m) {
    return m == 0 ? 1.0 : m == 1 ? 0.92387953251128675613 : m == 2 ? 0.70710678118654752440
         : m == 3 ? 0.38268343236508977173 : m == 4 ? 0.0 : m == 5 ? -0.38268343236508977173
         : m == 6 ? -0.70710678118654752440 : -0.92387953251128675613;
}
__host__ __device__ constexpr double w16s(int m) {  // imaginary part of W_16^m = -sin(2 pi m / 16)
    return m == 0 ? 0.0 : m == 1 ? -0.38268343236508977173 : m == 2 ? -0.70710678118654752440
         : m == 3 ? -0.92387953251128675613 : m == 4 ? -1.0 : m == 5 ? -0.92387953251128675613
         : m == 6 ? -0.70710678118654752440 : -0.38268343236508977173;
}

// cos and -sin of 2 pi m / 32, m < 16
__host__ __device__ constexpr double w32c(int m) {
    return m == 0 ? 1.0 : m == 1 ? 0.98078528040323044913 : m == 2 ? 0.92387953251128675613
         : m == 3 ? 0.83146961230254523708 : m == 4 ? 0.70710678118654752440 : m == 5 ? 0.55557023301960222474
         : m == 6 ? 0.38268343236508977173 : m == 7 ? 0.19509032201612826785 : m == 8 ? 0.0
         : m == 9 ? -0.19509032201612826785 : m == 10 ? -0.38268343236508977173 : m == 11 ? -0.55557023301960222474
         : m == 12 ? -0.70710678118654752440 : m == 13 ? -0.83146961230254523708 : m == 14 ? -0.92387953251128675613
         : -0.98078528040323044913;
}
__host__ __device__ constexpr double w32s(int m) { return -w32c((m + 24) % 32 < 16 ? (m + 24) % 32 : 32 - (m + 24) % 32); }

// v sqrt(1/2), or minus it (NEG).  FP64: by the constant's two parts, because the rounded one is
// 7e-17 high and every point of a chain of transforms meets it several times, always the same way
// (periodograms of 1/f data 3.6-6.9e-16 off -> 1.5-4.9e-16; N^-1 8.7e-16 -> 8.3e-16, 1178 -> 1191 us)
template <typename T, bool NEG> __device__ __forceinline__ Pr<T> by_rsqrt2(Pr<T> v) {
    constexpr double s = NEG ? -1.0 : 1.0;
    if constexpr (std::is_same<T, mono64>::value)
        return Pr<T>{fma(v.v, s * 0.70710678118654752440, v.v * (s * -4.8336466567264567e-17))};
    else return pmul(v, pcst<T>(s * 0.70710678118654752440));
}
// d * W_16^m (CONJ: d * conj(W_16^m)), m known at compile time
template <typename T, int M, bool CONJ>
__device__ __forceinline__ CP<T> mulw16(CP<T> d) {
    if constexpr (M == 0) {
        return d;
    } else if constexpr (M == 4) {
        if constexpr (!CONJ) return {d.y, psub(pcst<T>(0.0), d.x)};  // * -i
        else return {psub(pcst<T>(0.0), d.y), d.x};                   // * i
    } else if constexpr (M == 2 || M == 6) {
        // W^2 = (1 - i) r, W^6 = (-1 - i) r; conjugates (1 + i) r, (-1 + i) r
        if constexpr (M == 2 && !CONJ) return {by_rsqrt2<T, false>(padd(d.x, d.y)), by_rsqrt2<T, false>(psub(d.y, d.x))};
        else if constexpr (M == 2 && CONJ) return {by_rsqrt2<T, false>(psub(d.x, d.y)), by_rsqrt2<T, false>(padd(d.x, d.y))};
        else if constexpr (M == 6 && !CONJ) return {by_rsqrt2<T, false>(psub(d.y, d.x)), by_rsqrt2<T, true>(padd(d.x, d.y))};
        else return {by_rsqrt2<T, true>(padd(d.x, d.y)), by_rsqrt2<T, false>(psub(d.x, d.y))};
    } else {
        const CP<T> w{pcst<T>(w16c(M)), pcst<T>(w16s(M))};
        return CONJ ? cpmulc(d, w) : cpmul(d, w);
    }
}

// In-register radix-2 decimation in frequency over R = 2^L points (natural in;
// v[i] = DFT_R(v)[rev_L(i)] out).  Stage j: span h = R/2^(j+1), the difference
// of (i, i + h) times W_{2h}^(i mod 2h) = W_16^((i mod 2h) * 8/h) (R <= 16).
template <typename T, int R, int H>
__device__ __forceinline__ void dif_stage(CP<T> (&v)[R]) {
#pragma unroll
    for (int i = 0; i < R; i++) {
        if ((i % (2 * H)) < H) {
            const CP<T> a = v[i], b = v[i + H];
            v[i] = cpadd(a, b);
            const CP<T> d = cpsub(a, b);
            constexpr int S = 8 / H;
            switch ((i % (2 * H)) * S) {
                case 0: v[i + H] = d; break;
                case 1: v[i + H] = mulw16<T, 1, false>(d); break;
                case 2: v[i + H] = mulw16<T, 2, false>(d); break;
                case 3: v[i + H] = mulw16<T, 3, false>(d); break;
                case 4: v[i + H] = CP<T>{psub(a.y, b.y), psub(b.x, a.x)}; break;  // -i d
                case 5: v[i + H] = mulw16<T, 5, false>(d); break;
                case 6: v[i + H] = mulw16<T, 6, false>(d); break;
                default: v[i + H] = mulw16<T, 7, false>(d); break;
            }
        }
    }
}
template <typename T, int R>
__device__ __forceinline__ void dif_reg(CP<T> (&v)[R]) {
    if constexpr (R >= 16) dif_stage<T, R, 8>(v);
    if constexpr (R >= 8) dif_stage<T, R, 4>(v);
    if constexpr (R >= 4) dif_stage<T, R, 2>(v);
    if constexpr (R >= 2) dif_stage<T, R, 1>(v);
}
// the mirror: decimation in time with conjugate twiddles, v[i] = X[rev_L(i)]
// in, the unnormalised inverse DFT in natural order out
template <typename T, int R, int H>
__device__ __forceinline__ void dit_stage(CP<T> (&v)[R]) {
#pragma unroll
    for (int i = 0; i < R; i++) {
        if ((i % (2 * H)) < H) {
            const CP<T> a = v[i];
            CP<T>       b;
            constexpr int S = 8 / H;
            switch ((i % (2 * H)) * S) {
                case 0: b = v[i + H]; break;
                case 1: b = mulw16<T, 1, true>(v[i + H]); break;
                case 2: b = mulw16<T, 2, true>(v[i + H]); break;
                case 3: b = mulw16<T, 3, true>(v[i + H]); break;
                case 4: b = mulw16<T, 4, true>(v[i + H]); break;
                case 5: b = mulw16<T, 5, true>(v[i + H]); break;
                case 6: b = mulw16<T, 6, true>(v[i + H]); break;
                default: b = mulw16<T, 7, true>(v[i + H]); break;
            }
            v[i] = cpadd(a, b);
            v[i + H] = cpsub(a, b);
        }
    }
}
template <typename T, int R>
__device__ __forceinline__ void dit_reg(CP<T> (&v)[R]) {
    if constexpr (R >= 2) dit_stage<T, R, 1>(v);
    if constexpr (R >= 4) dit_stage<T, R, 2>(v);
    if constexpr (R >= 8) dit_stage<T, R, 4>(v);
    if constexpr (R >= 16) dit_stage<T, R, 8>(v);
}

__host__ __device__ constexpr int rev_bits_c(int v, int bits) {
    int r = 0;
    for (int b = 0; b < bits; b++) r |= ((v >> b) & 1) << (bits - 1 - b);
    return r;
}
__host__ __device__ constexpr int ilog2_c(int v) { return v <= 1 ? 0 : 1 + ilog2_c(v >> 1); }

}  // namespace
